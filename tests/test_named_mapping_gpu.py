"""A lane mapping named in the description belongs to the scene: alone, and among so many copies that
the launches fill the GPU, it steps to the same bits.  (Under the default mapping a launch with few
vertices gives each more lanes, which changes the order of their sums.)"""
import numpy as np
import pytest

import oracle_lib as O
from scenes import check_parity, pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("element,lanes,copies", [(O.TETRA, 4, 600), (O.HEXA, 4, 600), (O.TETRA10, 1, 300),
                                                  (O.TETRA10, 4, 300), (O.TETRA20, -1, 120), (O.HEXA27, -1, 120)])
def test_the_same_bits_alone_and_in_a_full_launch(ctx, element, lanes, copies, precision):
    import octopusengine_b200 as ob
    kw = dict(cells=(5, 3, 2), iterations=4, precision=precision, tpv=lanes)
    alone, o32, o64, mesh = pair(ctx, element, **kw)
    assert alone.mapping() == lanes
    skw = dict(masses=mesh["m"], material=ob.STABLE_NEOHOOKE, young=1e5, poisson=0.45, fixed_ids=mesh["fixed"],
               iterations=4, gravity=(0.0, 0.0, -9.81), precision=precision, threads_per_vertex=lanes)
    scenes = [ob.Scene(ctx, element, mesh["X"], mesh["T"], **skw) for _ in range(copies)]
    batch = ob.Batch(ctx, scenes)
    for _ in range(2):
        alone.step(1 / 60, 2)
        batch.step(1 / 60, 2)
        o32.step(1 / 60, 2)
        o64.step(1 / 60, 2)
    check_parity(alone.get_position(), o32, o64, mesh["X"], "e%d" % element)
    for k in (0, copies - 1):
        np.testing.assert_array_equal(scenes[k].get_position(), alone.get_position())
        np.testing.assert_array_equal(scenes[k].get_velocity(), alone.get_velocity())
    batch.close()
    for s in scenes:
        s.close()
