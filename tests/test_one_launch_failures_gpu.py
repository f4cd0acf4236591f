"""Failures of the one-launch VBD sub-step, without faulting the GPU: a grid barrier that runs out
of looks is reported by the scene it belongs to and leaves the scene usable; a cooperative launch
that the driver refuses is replaced by the launches per colour, also in a captured frame."""
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


@pytest.mark.parametrize("capture", [False, True])
@pytest.mark.parametrize("element,cells", [(O.TETRA, (1, 1, 1)), (O.HEXA, (12, 5, 4)), (O.TETRA10, (6, 3, 3))])
def test_a_refused_launch_falls_back_to_launches_per_colour(ctx, element, cells, capture):
    from octopusengine_b200 import capi
    X, _ = O.beam_mesh(element, cells, tuple(0.125 * c for c in cells))
    v0 = np.random.default_rng(1).normal(0.0, 0.05, X.shape).astype(np.float32)   # a pending first velocity
    kw = dict(cells=cells, size=tuple(0.125 * c for c in cells), iterations=4, rho=0.9, v0=v0)
    s, twin = pair(ctx, element, **kw)[0], pair(ctx, element, **kw)[0]
    s.set_capture(capture)
    twin.set_capture(capture)
    twin.step(1 / 60, 2)
    assert capi.lib().oct_ctx_refuse_probe(ctx.handle, 0 if capture else 1) == 0
    s.step(1 / 60, 2)
    if capture:   # the first frame, with the pending velocity, is not captured
        assert capi.lib().oct_ctx_refuse_probe(ctx.handle, 1) == 0
    for _ in range(3):   # the frame that meets the refusal, and replays of it
        s.step(1 / 60, 2)
    assert capi.lib().oct_ctx_refuse_probe(ctx.handle, 0) == 0
    for _ in range(3):
        twin.step(1 / 60, 2)
    np.testing.assert_array_equal(s.get_position(), twin.get_position())
    np.testing.assert_array_equal(s.get_velocity(), twin.get_velocity())
    assert np.abs(s.get_velocity()).max() > 0


def test_a_sync_before_the_first_step_leaves_no_error(built):
    import octopusengine_b200 as ob
    c = ob.Context(0, 1 << 28)
    X, T = O.beam_mesh(O.TETRA, (2, 1, 1), (1.0, 0.5, 0.5))
    s = ob.Scene(c, O.TETRA, X, T, iterations=2)
    s.sync()
    s.step(1 / 60, 1)
    assert s.status() == 0
    c.close()
