"""How much the FP32 elastic force adds to the rounding that it cannot avoid.  Near the rest shape the
entries of F are stored next to one, so F's own rounding (computed here: F rounded to 32 bits, all
else in 64) sets a floor under the force error.  lambda (det F - 1) carries it: three roundings of
diagonal entries, and one more of the cofactor entry that det F multiplies, if no later step rounds
next to one: sqrt(4 / 3) = 1.16 of the floor, and a few percent for the terms in mu (a ninth of
lambda here).  Two roundings more in det F would give sqrt(6 / 3) = 1.41."""
import ctypes as C

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu

CELLS = {O.TETRA: (8, 4, 4), O.HEXA: (8, 4, 4), O.TETRA10: (6, 4, 4), O.TETRA20: (5, 4, 3), O.HEXA27: (6, 4, 4)}
EDGE, YOUNG, POISSON = 0.0625, 1e5, 0.45


def _force(element, X, T, u, rounded):
    import octopusengine_b200 as ob
    _, w, dN = ob.shape_table(element)
    x = X.astype(np.float64)[T]
    J = np.einsum("eni,qnk->eqik", x, dN)
    inv, V = np.linalg.inv(J), np.abs(np.linalg.det(J)) * w
    F = np.eye(3) + np.einsum("eni,qnk->eqik", u.astype(np.float64)[T], dN) @ inv
    if rounded:
        F = F.astype(np.float32).astype(np.float64)
    lam = np.float64(np.float32(YOUNG * POISSON / ((1 + POISSON) * (1 - 2 * POISSON))))
    mu = np.float64(np.float32(YOUNG / (2 * (1 + POISSON))))
    a, b, c = F[..., 0], F[..., 1], F[..., 2]
    K = np.stack([np.cross(b, c), np.cross(c, a), np.cross(a, b)], -1)
    det = (a * K[..., 0]).sum(-1)[..., None, None]
    P = mu * F + (lam * (det - 1) - mu) * K
    g = np.einsum("qnk,eqkb->eqnb", dN, inv)
    f = np.zeros_like(X, np.float64)
    np.add.at(f, T.reshape(-1), -np.einsum("eq,eqib,eqnb->eni", V, P, g).reshape(-1, 3))
    return f


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("element", list(CELLS))
def test_force_error_is_near_the_rounding_of_F(ctx, element, precision):
    import octopusengine_b200 as ob
    from octopusengine_b200 import capi
    cells = CELLS[element]
    X, T = O.beam_mesh(element, cells, tuple(EDGE * n for n in cells))
    p = (X + np.random.default_rng(7).normal(0.0, 3e-4 * EDGE, X.shape)).astype(np.float32)
    u = p - X
    s = ob.Scene(ctx, element, X, T, material=ob.STABLE_NEOHOOKE, young=YOUNG, poisson=POISSON, precision=precision)
    s.set_position(p)
    f = np.zeros((len(X), 3), np.float32)
    # a time step of 1e6 s takes the inertial part of the residual below 1e-12 of the force
    capi.check(capi.lib().oct_scene_vertex_residuals(s.handle, 1e6, capi.ptr(f, C.c_float)), "residuals")
    exact = _force(element, X, T, u, False)
    floor = np.sqrt(np.mean((_force(element, X, T, u, True) - exact) ** 2))
    error = np.sqrt(np.mean((f - exact) ** 2))
    s.close()
    assert error <= 1.3 * floor, (error / floor, floor)
