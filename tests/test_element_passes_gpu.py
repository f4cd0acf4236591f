"""The element passes of the explicit integrator and of XPBD at the sizes where their blocks change
shape (a single cell, partly filled last blocks, several blocks, distorted elements with a record
per point), for every material, against the FP64 oracle."""
import numpy as np
import pytest

import oracle_lib as O
from scenes import disp_err, rel_err

pytestmark = pytest.mark.gpu

CELLS = [(1, 1, 1), (3, 2, 1), (7, 3, 3), (13, 6, 5)]
MATERIALS = [O.HOOKE, O.STVK, O.NEOHOOKE, O.STABLE_NEOHOOKE]


def _check(ctx, solver, element, cells, material, distorted, substeps, dt, precision=0, damping=0.0):
    import octopusengine_b200 as ob
    X, T = O.beam_mesh(element, cells, tuple(0.1 * c for c in cells))
    if distorted:
        X = X + np.random.default_rng(3).uniform(-0.004, 0.004, X.shape).astype(np.float32)
    m = O.masses(element, X, T, 1000.0, 1)
    fixed = np.nonzero(X[:, 0] < 0.01)[0].astype(np.int32)
    v0 = np.random.default_rng(4).normal(0, 0.5, X.shape).astype(np.float32)
    kind = {"xpbd": ob.SOLVER_XPBD, "explicit": ob.SOLVER_EXPLICIT}[solver]
    s = ob.Scene(ctx, element, X, T, solver=kind, masses=m, material=material, young=1e5, poisson=0.4, fixed_ids=fixed,
                 initial_velocity=v0, gravity=(0.0, 0.0, -9.81), precision=precision, damping=damping)
    kw = dict(material=material, young=1e5, poisson=0.4, fixed=fixed, v0=v0, gravity=(0.0, 0.0, -9.81), damping=damping)
    keep = [O.Scene(element, X, T, m, **kw) for _ in range(2)]
    o32, o64 = O.Solver(solver, keep[0], fp64=False), O.Solver(solver, keep[1], fp64=True)
    s.step(dt, substeps)
    o32.step(dt, substeps)
    o64.step(dt, substeps)
    p, ref = s.get_position(), o64.get(0)
    assert rel_err(p, ref) < 1e-5
    floor = 2.0 * np.finfo(np.float32).eps * np.abs(ref).max() / np.abs(ref - X).max()
    assert disp_err(p, ref, X) <= 3.0 * disp_err(o32.get(0), ref, X) + floor
    s.close()


@pytest.mark.parametrize("cells", CELLS)
@pytest.mark.parametrize("material", MATERIALS)
@pytest.mark.parametrize("element", [O.TETRA, O.HEXA, O.TETRA10])
def test_explicit(ctx, element, material, cells):
    _check(ctx, "explicit", element, cells, material, False, 20, 20 * 2e-5)
    _check(ctx, "explicit", element, cells, material, True, 20, 20 * 2e-5, precision=1)


@pytest.mark.parametrize("element,cells", [(e, c) for e in (O.TETRA, O.HEXA, O.TETRA10) for c in CELLS] +
                         [(O.TETRA20, c) for c in CELLS[:3]])
@pytest.mark.parametrize("material", MATERIALS)
def test_xpbd(ctx, element, cells, material):
    _check(ctx, "xpbd", element, cells, material, False, 2, 1 / 120)
    _check(ctx, "xpbd", element, cells, material, True, 2, 1 / 120)


@pytest.mark.parametrize("cells", CELLS[:3])
@pytest.mark.parametrize("element", [O.TETRA, O.HEXA, O.TETRA10, O.TETRA20, O.HEXA27])
def test_explicit_damped(ctx, element, cells):
    _check(ctx, "explicit", element, cells, O.STABLE_NEOHOOKE, False, 20, 20 * 2e-5, damping=1e-4)
    _check(ctx, "explicit", element, cells, O.NEOHOOKE, True, 20, 20 * 2e-5, precision=1, damping=1e-4)
