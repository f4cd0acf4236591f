"""Node state and error word between a context and host memory: a state that just fits the context's
pinned block and one that just does not, into pageable and pinned memory, in the context's first uses
(without the block) and after them, from one thread and from two at once; and contexts that wait at
the same time, each in its own thread, which must not slow one another down beyond taking turns."""
import ctypes as C
import threading
import time

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu

MOST = 262144 // 12   # nodes of the largest state in the pinned block


def _scene(ctx, cells):
    import octopusengine_b200 as ob
    X, T = O.beam_mesh(O.TETRA, cells, tuple(n / 16 for n in cells))
    return ob.Scene(ctx, O.TETRA, X, T, iterations=2, young=1e5), X


@pytest.mark.parametrize("cells,nodes", [((1, 1, 1), 8), ((4, 16, 256), MOST), ((1, 32, 330), MOST + 1),
                                         ((40, 40, 40), 41 ** 3)])
def test_state_round_trips(built, cells, nodes):
    import torch
    import octopusengine_b200 as ob
    from octopusengine_b200 import capi
    ctx = ob.Context(0, 4 << 30)
    scenes = [_scene(ctx, cells)[0] for _ in range(2)]
    X = _scene(ctx, cells)[1]
    assert len(X) == nodes
    pinned = torch.empty((nodes, 3), dtype=torch.float32, pin_memory=True).numpy()
    wrong = []

    def check(s, seed):
        v = np.random.default_rng(seed).normal(0.0, 1.0, X.shape).astype(np.float32)
        s.set_velocity(v)
        if not np.array_equal(s.get_velocity(), v) or not np.array_equal(s.get_position(), X):
            wrong.append(seed)
        s.sync()

    for k in range(3):     # without the block
        check(scenes[0], k)
    for k in range(40):    # makes it
        scenes[0].sync()
    for k in range(3, 6):
        check(scenes[0], k)
        capi.check(capi.lib().oct_scene_get_velocities(scenes[0].handle, capi.ptr(pinned, C.c_float)), "get", ctx.handle)
        np.testing.assert_array_equal(pinned, scenes[0].get_velocity())
    threads = [threading.Thread(target=lambda i=i: [check(scenes[i], 100 * i + k) for k in range(20)]) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    ctx.close()


def test_waiting_contexts_do_not_hold_each_other_up(built):
    import octopusengine_b200 as ob
    ctxs = [ob.Context(0, 1 << 28) for _ in range(8)]
    scenes = [_scene(c, (8, 2, 2))[0] for c in ctxs]

    def run(s):
        for _ in range(30):
            s.step(1 / 60, 2)
            s.get_position()

    def all_of(some):
        best = 1e9
        for _ in range(5):
            threads = [threading.Thread(target=run, args=(s,)) for s in some]
            t = time.perf_counter()
            for x in threads:
                x.start()
            for x in threads:
                x.join()
            best = min(best, time.perf_counter() - t)
        return best

    for s in scenes:
        run(s)
    one, eight = all_of(scenes[:1]), all_of(scenes)
    for c in ctxs:
        c.close()
    assert eight < 8 * one, (one, eight)
