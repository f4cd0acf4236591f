"""Lanes per vertex chosen by the launch: copies of one scene in batches of growing size run the
same colours with fewer and fewer lanes per vertex (one owner per lane for a scene alone, the
element's least for a launch that fills the GPU), and each copy matches the FP64 oracle."""
import numpy as np
import pytest

import oracle_lib as O
from scenes import check_parity, pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 37, 150, 600])
@pytest.mark.parametrize("element", [O.TETRA, O.HEXA, O.TETRA10])
@pytest.mark.parametrize("precision", [0, 1])
def test_copies_in_one_launch_match_the_oracle(ctx, element, copies, precision):
    import octopusengine_b200 as ob
    s, o32, o64, mesh = pair(ctx, element, cells=(5, 3, 2), iterations=4, precision=precision)
    kw = dict(masses=mesh["m"], material=ob.STABLE_NEOHOOKE, young=1e5, poisson=0.45, fixed_ids=mesh["fixed"],
              iterations=4, gravity=(0.0, 0.0, -9.81), precision=precision)
    scenes = [s] + [ob.Scene(ctx, element, mesh["X"], mesh["T"], **kw) for _ in range(copies - 1)]
    batch = ob.Batch(ctx, scenes)
    batch.step(1 / 60, 2)
    o32.step(1 / 60, 2)
    o64.step(1 / 60, 2)
    first = s.get_position()
    check_parity(first, o32, o64, mesh["X"], "%d copies" % copies)
    for k in (copies // 2, copies - 1):
        np.testing.assert_array_equal(scenes[k].get_position(), first)   # the copies share every launch
    batch.close()
    for x in scenes:
        x.close()
