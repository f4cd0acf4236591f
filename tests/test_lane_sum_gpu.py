"""The sum of a vertex's terms over its lanes in mixed precision: with one owner per lane and one
quadrature point per element, the force is the correctly rounded sum of the owners' terms, up to the
rounding of the compensations themselves (five additions of what five additions round off: 2^-43 of
the terms' magnitudes).  The terms come, bit for bit, from scenes of one element each."""
import ctypes as C
import math

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


def _force(ctx, X, T, p, lanes):
    import octopusengine_b200 as ob
    from octopusengine_b200 import capi
    s = ob.Scene(ctx, O.TETRA, X, T, material=ob.STABLE_NEOHOOKE, young=1e5, poisson=0.45, precision=ob.PREC_MIXED,
                 threads_per_vertex=lanes)
    s.set_position(p)
    f = np.zeros((len(X), 3), np.float32)
    # a time step of 1e6 s: the inertial part of the residual is far below the force's last bit
    capi.check(capi.lib().oct_scene_vertex_residuals(s.handle, 1e6, capi.ptr(f, C.c_float)), "residuals")
    s.close()
    return f


def test_owners_are_summed_without_loss(ctx):
    X, T = O.beam_mesh(O.TETRA, (3, 3, 3), (0.2, 0.3, 0.25))
    r = np.random.default_rng(3)
    # a stretch, under which the terms of an inner vertex cancel, and a small disturbance
    p = (X.astype(np.float64) @ (np.eye(3) + r.uniform(-0.1, 0.1, (3, 3))) + r.normal(0, 1e-6, X.shape)).astype(np.float32)
    terms = [[[] for _ in range(3)] for _ in X]
    for t in T:
        f = _force(ctx, X[t], np.arange(4, dtype=np.int32)[None], p[t], 32)
        for k in range(4):
            for d in range(3):
                terms[t[k]][d].append(float(f[k, d]))
    assert max(len(v[0]) for v in terms) > 16
    got = _force(ctx, X, T, p, 32)
    for v in range(len(X)):
        for d in range(3):
            exact = math.fsum(terms[v][d])
            bound = 2.0 ** -24 * abs(exact) + 2.0 ** -43 * math.fsum(map(abs, terms[v][d]))
            assert abs(float(got[v, d]) - exact) <= bound, (v, d, float(got[v, d]), exact)
