"""Failures of the one-launch VBD sub-step, without faulting the GPU: a grid barrier that runs out
of looks is reported by the scene it belongs to and leaves the scene usable."""
import numpy as np
import pytest

import oracle_lib as O
from scenes import check_parity, pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("element", [O.TETRA, O.HEXA, O.TETRA10])
def test_a_barrier_time_out_belongs_to_its_scene(ctx, element):
    from octopusengine_b200 import capi
    kw = dict(cells=(12, 5, 4), size=(1.5, 0.625, 0.5), iterations=4)   # several blocks per colour
    s, o32, o64, mesh = pair(ctx, element, **kw)
    other = pair(ctx, element, **kw)[0]
    assert capi.lib().oct_scene_wait_probe(s.handle, 2000) == capi.ETIMEDOUT   # reads and clears the context's word
    assert other.status() == 0
    assert s.status() == capi.ETIMEDOUT
    assert s.status() == 0   # reported once
    for _ in range(2):       # both counters were cleared: the next steps are the scene's own
        s.step(1 / 60, 2)
        other.step(1 / 60, 2)
        o32.step(1 / 60, 2)
        o64.step(1 / 60, 2)
    check_parity(s.get_position(), o32, o64, mesh["X"], "e%d" % element)
    np.testing.assert_array_equal(s.get_position(), other.get_position())
    assert s.status() == 0
