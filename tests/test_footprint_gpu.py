"""oct_scene_footprint against what a scene really takes: never less, and for meshes without two equal
elements (a record per quadrature point, nothing shared) not half as much again, for every solver and
element type."""
import ctypes as C

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu

ELEMENTS = [(O.TETRA, (9, 5, 4)), (O.HEXA, (12, 7, 6)), (O.TETRA10, (7, 4, 3)), (O.TETRA20, (5, 3, 3)), (O.HEXA27, (6, 4, 4))]


@pytest.mark.parametrize("lanes", [0, -1, 1, 32])
@pytest.mark.parametrize("distorted", [False, True])
@pytest.mark.parametrize("element,cells", ELEMENTS)
@pytest.mark.parametrize("solver", ["vbd", "xpbd", "explicit"])
def test_estimate_covers_the_scene(built, solver, element, cells, distorted, lanes):
    import octopusengine_b200 as ob
    from octopusengine_b200 import capi
    X, T = O.beam_mesh(element, cells, tuple(0.1 * n for n in cells))
    if distorted:
        X = X + np.random.default_rng(3).uniform(-0.004, 0.004, X.shape).astype(np.float32)
    kind = {"vbd": ob.SOLVER_VBD, "xpbd": ob.SOLVER_XPBD, "explicit": ob.SOLVER_EXPLICIT}[solver]
    kw = dict(solver=kind, fixed_ids=np.arange(len(X) // 3, dtype=np.int32), threads_per_vertex=lanes)
    d, keep = ob.make_desc(element, X, T, **kw)
    need = C.c_size_t()
    assert capi.lib().oct_scene_footprint(C.byref(d), C.byref(need)) == 0
    ctx = ob.Context(0, 1 << 30)
    before = ctx.memory()[0]
    ob.Scene(ctx, element, X, T, **kw)
    used = ctx.memory()[0] - before
    ctx.close()
    assert used <= need.value
    if distorted:
        assert need.value < 1.5 * used, (need.value, used)
