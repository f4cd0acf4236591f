"""Two contexts, each stepped by its own thread, share the GPU: a scene's launches leave room on the
SMs for another's.  Medium scenes, whose one-launch sub-steps hold as many blocks as there are SMs
or close to it: if they took turns, two would take twice as long as one.  While another context's
launches hold the SMs, a scene takes the launch path, to the same bits."""
import threading
import time

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


def _frames(scenes, frames):
    def run(s):
        for _ in range(frames):
            s.step(1 / 60, 2)

    best = 1e9
    for _ in range(5):
        threads = [threading.Thread(target=run, args=(s,)) for s in scenes]
        t = time.perf_counter()
        for x in threads:
            x.start()
        for x in threads:
            x.join()
        best = min(best, time.perf_counter() - t)
    return best


@pytest.mark.parametrize("element,cells", [(O.TETRA, (64, 16, 16)), (O.HEXA, (64, 16, 16)), (O.TETRA10, (24, 7, 7))])
def test_two_contexts_overlap(built, element, cells):
    import octopusengine_b200 as ob
    X, T = O.beam_mesh(element, cells, tuple(n / 16 for n in cells))
    fixed = np.nonzero(X[:, 0] < 1e-3)[0].astype(np.int32)
    ctxs = [ob.Context(0, 1 << 30) for _ in range(2)]
    scenes = [ob.Scene(c, element, X, T, fixed_ids=fixed, iterations=10, young=1e6) for c in ctxs]
    for s in scenes:
        s.step(1 / 60, 2)
    one, two = _frames(scenes[:1], 40), _frames(scenes, 40)
    a, b = scenes[0], scenes[1]
    for _ in range(200):   # the first has stepped more frames: the second catches up
        b.step(1 / 60, 2)
    np.testing.assert_array_equal(a.get_position(), b.get_position())
    for c in ctxs:
        c.close()
    assert two < 1.5 * one, (one, two)


def test_a_context_gives_way_to_one_in_flight(built):
    import octopusengine_b200 as ob
    X, T = O.beam_mesh(O.TETRA10, (36, 9, 9), (2.25, 0.5625, 0.5625))   # two groups of threads on most SMs
    ctxs = [ob.Context(0, 1 << 30) for _ in range(2)]
    a, b = [ob.Scene(c, O.TETRA10, X, T, iterations=4, young=1e6) for c in ctxs]

    def launches(s):
        n = s.ctx.launch_count()
        s.step(1 / 60, 3)
        return s.ctx.launch_count() - n

    assert launches(a) == 3 and launches(b) == 3
    a.step(1 / 60, 3, sync=False)
    assert launches(b) > 3
    a.sync()
    assert launches(b) == 3
    a.step(1 / 60, 3, sync=False)
    a.get_position()   # waits for the frame, too
    assert launches(b) == 3
    a.step(1 / 60, 3)
    np.testing.assert_array_equal(a.get_position(), b.get_position())
    np.testing.assert_array_equal(a.get_velocity(), b.get_velocity())
    for c in ctxs:
        c.close()
