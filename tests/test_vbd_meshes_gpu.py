"""VBD on meshes other than the regular beams: distorted elements, with a quadrature record per point,
in both launch forms of every element type; and fans of Q2 hexahedra around one edge, whose vertices
have as many owners as an item of the point lanes has pair slots (24), one more (two rounds), as many
as the packed mapping takes (32), and one more (lane groups); against the FP64 oracle."""
import numpy as np
import pytest

import oracle_lib as O
from scenes import check_parity

pytestmark = pytest.mark.gpu


def _run(ctx, element, X, T, fixed, precision, lanes=(0,), rho=0.0, damping=0.0):
    import octopusengine_b200 as ob
    m = O.masses(element, X, T, 1000.0, 1)
    colors, n = O.colour(element, T, len(X), 0)
    assert O.conflicts(element, T, len(X), colors) == 0
    kw = dict(young=1e5, poisson=0.4, iterations=4, gravity=(0.0, 0.0, -9.81), rho=rho, damping=damping)
    keep = [O.Scene(element, X, T, m, fixed=fixed, colors=colors, n_colors=n, in_place=True, **kw) for _ in range(2)]
    o32, o64 = O.Solver("vbd", keep[0], fp64=False), O.Solver("vbd", keep[1], fp64=True)
    scenes = [ob.Scene(ctx, element, X, T, masses=m, fixed_ids=fixed, precision=precision, threads_per_vertex=k, **kw)
              for k in lanes]
    twin = ob.Scene(ctx, element, X, T, masses=m, fixed_ids=fixed, precision=precision, **kw)
    batch = ob.Batch(ctx, [twin])
    for _ in range(2):
        batch.step(1 / 60, 2)
        for s in scenes + [o32, o64]:
            s.step(1 / 60, 2)
    for k, s in zip(lanes, scenes):
        check_parity(s.get_position(), o32, o64, X, "e%d lanes %d" % (element, k))
    np.testing.assert_array_equal(twin.get_position(), scenes[0].get_position())
    batch.close()


@pytest.mark.parametrize("precision,rho,damping", [(0, 0.0, 1e-4), (1, 0.9, 0.0)])
@pytest.mark.parametrize("element,cells", [(O.TETRA, (9, 4, 3)), (O.HEXA, (1, 1, 1)), (O.HEXA, (9, 5, 4)),
                                           (O.TETRA10, (1, 1, 1)), (O.TETRA10, (7, 3, 3)), (O.TETRA20, (1, 1, 1)),
                                           (O.TETRA20, (4, 3, 2)), (O.HEXA27, (1, 1, 1)), (O.HEXA27, (6, 4, 3))])
def test_distorted_elements(ctx, element, cells, precision, rho, damping):
    X, T = O.beam_mesh(element, cells, tuple(0.125 * n for n in cells))
    X = X + np.random.default_rng(3).uniform(-0.005, 0.005, X.shape).astype(np.float32)
    fixed = np.nonzero(X[:, 0] < 0.01)[0].astype(np.int32)
    _run(ctx, element, X, T, fixed, precision, lanes=(0, -1, 8), rho=rho, damping=damping)


def _fan(n):
    """(X, T): n Q2 hexahedra around the z axis, each a sector's quadrilateral between z = 0 and 0.3."""
    signs = np.array([(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1),
                      (0, -1, -1), (1, 0, -1), (0, 1, -1), (-1, 0, -1), (-1, -1, 0), (1, -1, 0), (1, 1, 0), (-1, 1, 0),
                      (0, -1, 1), (1, 0, 1), (0, 1, 1), (-1, 0, 1), (0, 0, -1), (0, -1, 0), (1, 0, 0), (0, 1, 0),
                      (-1, 0, 0), (0, 0, 1), (0, 0, 0)])
    w = np.prod(1 + signs[:, None, :] * signs[None, :8, :], axis=2) / 8.0   # node by corner
    at = lambda r, a: (r * np.cos(a), r * np.sin(a))  # noqa: E731
    ids, X, T = {}, [], []
    for k in range(n):
        a, b = 2 * np.pi * k / n, 2 * np.pi * (k + 1) / n
        quad = [(0.0, 0.0), at(1.0, a), at(1.3, (a + b) / 2), at(1.0, b)]
        corners = np.array([(x, y, z) for z in (0.0, 0.3) for x, y in quad])
        T.append([])
        for p in w @ corners:
            key = tuple(np.round(p * 1e6).astype(int) + 0)
            if key not in ids:
                ids[key] = len(X)
                X.append(p)
            T[-1].append(ids[key])
    return np.array(X, np.float32), np.array(T, np.int32)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("owners", [3, 24, 25, 32, 33])
def test_vertices_of_many_owners(ctx, owners, precision):
    X, T = _fan(owners)
    assert np.bincount(T.reshape(-1)).max() == owners
    fixed = np.nonzero(np.hypot(X[:, 0], X[:, 1]) > 1.1)[0].astype(np.int32)
    _run(ctx, O.HEXA27, X, T, fixed, precision, lanes=(0, 8))
