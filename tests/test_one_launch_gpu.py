"""VBD sub-steps of one scene in one cooperative launch, and the point lanes of the many-point
elements, at the sizes where their work changes shape: one block, several blocks with a partly
filled last item, colours of more items than blocks, a scene too large for one launch; each
against the FP64 oracle, with Chebyshev and damping, and against the same scene in a batch, which
takes the launch path."""
import numpy as np
import pytest

import oracle_lib as O
from scenes import check_parity, pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("element,cells", [
    (O.TETRA, (1, 1, 1)), (O.TETRA, (9, 3, 2)), (O.TETRA, (24, 9, 7)), (O.HEXA, (1, 1, 1)), (O.HEXA, (7, 5, 3)),
    (O.HEXA, (30, 11, 9)), (O.TETRA10, (1, 1, 1)), (O.TETRA10, (6, 3, 3)), (O.TETRA10, (26, 10, 9)),
    (O.TETRA10, (64, 17, 17)), (O.TETRA20, (1, 1, 1)), (O.TETRA20, (5, 4, 3)), (O.HEXA27, (1, 1, 1)), (O.HEXA27, (6, 4, 3))])
@pytest.mark.parametrize("rho,damping,precision", [(0.0, 0.0, 0), (0.9, 1e-4, 1)])
def test_sub_step_matches_the_oracle(ctx, element, cells, rho, damping, precision):
    import octopusengine_b200 as ob
    size = tuple(0.125 * c for c in cells)
    kw = dict(cells=cells, size=size, iterations=4, rho=rho, damping=damping, precision=precision)
    s, o32, o64, mesh = pair(ctx, element, **kw)
    twin = pair(ctx, element, **kw)[0]
    batch = ob.Batch(ctx, [twin])
    for _ in range(2):
        s.step(1 / 60, 2)
        batch.step(1 / 60, 2)
        o32.step(1 / 60, 2)
        o64.step(1 / 60, 2)
    check_parity(s.get_position(), o32, o64, mesh["X"], "e%d %s" % (element, cells))
    np.testing.assert_array_equal(twin.get_position(), s.get_position())
    np.testing.assert_array_equal(twin.get_velocity(), s.get_velocity())
    assert s.status() == 0
    batch.close()
