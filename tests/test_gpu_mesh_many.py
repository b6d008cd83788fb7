"""Mesh grids of meshes around the size above which the winding number is
summed in double precision (k_levelset_mesh): the unit cube, its faces cut into
squares, against the cube's own signed distance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cube(m):
    """12 m^2 triangles, outward."""
    g = np.arange(m + 1) / m
    u, v = np.meshgrid(g, g, indexing="ij")
    u, v = u.ravel(), v.ravel()
    i, j = np.meshgrid(np.arange(m), np.arange(m), indexing="ij")
    a = (i * (m + 1) + j).ravel()
    quad = np.stack([a, a + m + 1, a + m + 2, a, a + m + 2, a + 1], 1).reshape(-1, 3)
    verts, tris = [], []
    for d in range(3):
        for side in (0.0, 1.0):
            p = np.zeros((len(u), 3))
            p[:, d], p[:, (d + 1) % 3], p[:, (d + 2) % 3] = side, u, v
            tris.append((quad if side else quad[:, ::-1]) + len(u) * len(verts))
            verts.append(p)
    return np.concatenate(verts), np.concatenate(tris).astype(np.int32)


@pytest.mark.parametrize("m", [3, 590, 592])   # 108, 4,177,200 and 4,205,568 triangles; the rule's 4,194,304
def test_cube_of_many_triangles(fundem, m):
    v, tri = _cube(m)
    h, n = 0.3, (5, 4, 4)
    o = np.array([-0.13, -0.11, 0.07])
    got = fundem.levelset_grid("mesh", None, o, h, n, vertices=v, triangles=tri)
    Z, Y, X = np.meshgrid(*(o[d] + np.arange(n[d]) * h for d in (2, 1, 0)), indexing="ij")
    p = np.stack([X, Y, Z], -1).reshape(-1, 3)
    out = np.linalg.norm(np.maximum(np.maximum(-p, p - 1.0), 0.0), axis=1)
    inner = np.minimum(p, 1.0 - p).min(1)
    ref = np.where(inner > 0, -inner, out)
    assert (ref < 0).any() and (ref > 0).any()
    assert np.abs(got.reshape(-1) - ref).max() < 1e-12
