"""Fixed vertices cost no owner: once a sub-step has fixed them, the sweeps of scenes that are fixed but
for their tip take less than those of the same scenes free, by a part of the work; and such scenes
match the oracle, in both launch forms, while the fixation moves."""
import ctypes as C

import numpy as np
import pytest

import oracle_lib as O
from scenes import check_parity, pair

pytestmark = pytest.mark.gpu


def _sweep_ms(ctx, element, cells, copies, part):
    import octopusengine_b200 as ob
    from octopusengine_b200 import capi
    X, T = O.beam_mesh(element, cells, tuple(n / 16 for n in cells))
    fixed = np.nonzero(X[:, 0] < part * X[:, 0].max())[0].astype(np.int32)
    scenes = [ob.Scene(ctx, element, X, T, fixed_ids=fixed, iterations=2, young=1e6) for _ in range(copies)]
    batch = ob.Batch(ctx, scenes)
    batch.step(1 / 60, 1)
    ms, best = C.c_float(), 1e9
    for _ in range(5):
        capi.check(capi.lib().oct_batch_time_group(batch._h, 0, 20, 1 / 60, C.byref(ms)), "time", ctx.handle)
        best = min(best, ms.value / 20)
    batch.close()
    for s in scenes:
        s.close()
    return best


@pytest.mark.parametrize("element,cells,copies", [(O.TETRA, (64, 16, 16), 24), (O.HEXA, (64, 16, 16), 12),
                                                  (O.TETRA10, (32, 10, 10), 8), (O.TETRA20, (16, 8, 8), 6),
                                                  (O.HEXA27, (24, 10, 10), 6)])
def test_sweeps_skip_the_owners_of_fixed_vertices(ctx, element, cells, copies):
    # a sweep takes a fixed part and a part by vertex, which a batch of twice the copies tells apart;
    # of the latter, fixing all but a twentieth of the vertices must save a sixth at least.  Reading
    # every vertex's slot, mask and first entry remains: kernels that skip the owners save 0.19 (Q1)
    # to 0.52 (Q2) of it, kernels that evaluate them and drop the result 0.10 to 0.12.
    free, twice = [_sweep_ms(ctx, element, cells, n * copies, 0.02) for n in (1, 2)]
    held = _sweep_ms(ctx, element, cells, copies, 0.95)
    print("e%d free %.3f twice %.3f held %.3f ms: saved %.2f of the work" % (element, free, twice, held,
                                                                            (free - held) / (twice - free)))
    assert free - held > (twice - free) / 6, (free, twice, held)


@pytest.mark.parametrize("element,cells", [(O.TETRA, (8, 3, 3)), (O.HEXA, (8, 3, 3)), (O.TETRA10, (5, 3, 2)),
                                           (O.TETRA20, (4, 2, 2)), (O.HEXA27, (5, 3, 2))])
@pytest.mark.parametrize("rho", [0.0, 0.9])
def test_mostly_fixed_scenes_match_the_oracle(ctx, element, cells, rho):
    import octopusengine_b200 as ob
    size = tuple(0.125 * n for n in cells)
    X, _ = O.beam_mesh(element, cells, size)
    fixed = np.nonzero(X[:, 0] < 0.7 * size[0])[0].astype(np.int32)
    kw = dict(cells=cells, size=size, iterations=4, rho=rho, fixed=fixed)
    s, o32, o64, mesh = pair(ctx, element, **kw)
    twin = pair(ctx, element, **kw)[0]
    batch = ob.Batch(ctx, [twin])
    for k in range(3):
        for x in (s, twin, o32, o64):
            x.set_fixation(offset=(0.002 * k, 0.001 * k, 0.0))
        s.step(1 / 60, 2)
        batch.step(1 / 60, 2)
        o32.step(1 / 60, 2)
        o64.step(1 / 60, 2)
    check_parity(s.get_position(), o32, o64, mesh["X"], "e%d" % element)
    np.testing.assert_array_equal(twin.get_position(), s.get_position())
    batch.close()
