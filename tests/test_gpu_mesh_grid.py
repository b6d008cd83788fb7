"""Mesh grids: the screened kernel (k_levelset_mesh) gives the values of the
plain double-precision scan over all triangles, bit for bit: closest point
first in triangle order (Ericson's region walk), sign by the winding number.
Sizes at the edges of its node tiles (8 x 4) and triangle stages (128, 32 a
warp); nodes on corners, edges and faces; slivers; an open mesh, whose winding
number is taken again in double precision; a mesh far from the origin and one
much larger than its grid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dot(a, b):
    return a[..., 0] * b[..., 0] + a[..., 1] * b[..., 1] + a[..., 2] * b[..., 2]


def _cross(a, b):
    return np.stack([a[..., 1] * b[..., 2] - a[..., 2] * b[..., 1], a[..., 2] * b[..., 0] - a[..., 0] * b[..., 2],
                     a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]], -1)


def _len(a):
    return np.sqrt(a[..., 0] * a[..., 0] + a[..., 1] * a[..., 1] + a[..., 2] * a[..., 2])


def _closest(p, a, b, c):
    ab, ac, ap, bp, cp = b - a, c - a, p - a, p - b, p - c
    d1, d2, d3, d4, d5, d6 = _dot(ab, ap), _dot(ac, ap), _dot(ab, bp), _dot(ac, bp), _dot(ab, cp), _dot(ac, cp)
    vc, vb, va = d1 * d4 - d3 * d2, d5 * d2 - d1 * d6, d3 * d6 - d5 * d4
    with np.errstate(all="ignore"):
        inv = 1.0 / (va + vb + vc)
        inside = a + ab * (vb * inv)[..., None] + ac * (vc * inv)[..., None]
        on_bc = b + ((d4 - d3) / ((d4 - d3) + (d5 - d6)))[..., None] * (c - b)
        on_ac = a + (d2 / (d2 - d6))[..., None] * ac
        on_ab = a + (d1 / (d1 - d3))[..., None] * ab
    conds = [(d1 <= 0) & (d2 <= 0), (d3 >= 0) & (d4 <= d3), (vc <= 0) & (d1 >= 0) & (d3 <= 0), (d6 >= 0) & (d5 <= d6),
             (vb <= 0) & (d2 >= 0) & (d6 <= 0), (va <= 0) & (d4 - d3 >= 0) & (d5 - d6 >= 0)]
    picks = [a + 0 * p, b + 0 * p, on_ab, c + 0 * p, on_ac, on_bc]
    return np.select([k[..., None] for k in conds], picks, inside)


def _scan(v, tri, o, h, n):
    ax = [o[d] + np.arange(n[d]) * h for d in range(3)]
    Z, Y, X = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    p = np.stack([X, Y, Z], -1).reshape(-1, 3)
    best, near, wind = np.full(len(p), np.finfo(float).max), p.copy(), np.zeros(len(p))
    for t in tri:
        a, b, c = v[t]
        q = _closest(p, a, b, c)
        d2 = _dot(p - q, p - q)
        m = d2 < best
        best[m], near[m] = d2[m], q[m]
        r0, r1, r2 = a - p, b - p, c - p
        l0, l1, l2 = _len(r0), _len(r1), _len(r2)
        den = l0 * l1 * l2 + _dot(r0, r1) * l2 + _dot(r1, r2) * l0 + _dot(r2, r0) * l1
        w = 2.0 * np.arctan2(_dot(r0, _cross(r1, r2)), den)
        wind += np.where((l0 < 1e-30) | (l1 < 1e-30) | (l2 < 1e-30), 0.0, w)
    d = _len(p - near)
    inside = np.abs(wind / (4.0 * np.pi)) > 0.5
    f = np.where(inside, -d, d)
    with np.errstate(all="ignore"):
        u = (p - near) * (1.0 / d)[:, None]
    g = np.where((d > 1e-30)[:, None], np.where(inside[:, None], -u, u), 0.0)
    gn = _len(g)
    with np.errstate(all="ignore"):
        return np.where(gn > 1e-12, f / gn, np.where(f <= 0, -1.0, 1.0) * 0.5 * h)


def _torus(nu, nv, big=1.0, small=0.35):
    u, w = np.meshgrid(2 * np.pi * np.arange(nu) / nu, 2 * np.pi * np.arange(nv) / nv, indexing="ij")
    v = np.stack([(big + small * np.cos(w)) * np.cos(u), (big + small * np.cos(w)) * np.sin(u), small * np.sin(w)], -1)
    i, j = np.meshgrid(np.arange(nu), np.arange(nv), indexing="ij")
    at = lambda a, b: (a % nu) * nv + (b % nv)
    tri = np.concatenate([np.stack([at(i, j), at(i + 1, j), at(i + 1, j + 1)], -1).reshape(-1, 3),
                          np.stack([at(i, j), at(i + 1, j + 1), at(i, j + 1)], -1).reshape(-1, 3)])
    return v.reshape(-1, 3), tri.astype(np.int32)


def _cube(refine=0):
    v = np.array([[x, y, z] for z in (0., 1.) for y in (0., 1.) for x in (0., 1.)])
    tri = np.array([[0, 2, 1], [1, 2, 3], [4, 5, 6], [5, 7, 6], [0, 1, 4], [1, 5, 4], [2, 6, 3], [3, 6, 7], [0, 4, 2],
                    [2, 4, 6], [1, 3, 5], [3, 7, 5]], np.int32)
    return v, tri


def _cases():
    tet = np.array([[0., 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]]), np.array([[0, 2, 1], [0, 1, 3], [0, 3, 2], [1, 2, 3]],
                                                                            np.int32)
    yield "tetrahedron, one node", tet, [0.2, 0.2, 0.2], 0.1, (1, 1, 1)
    yield "tetrahedron, nodes on its corners and edges", tet, [-0.5, -0.5, -0.5], 0.25, (9, 7, 5)
    yield "cube, nodes on its faces", _cube(), [-0.25, -0.25, -0.25], 0.25, (7, 7, 8)
    yield "torus of 128 triangles", _torus(8, 8), [-1.5, -1.5, -0.5], 0.31, (10, 11, 4)
    v, tri = _torus(8, 8)
    yield "nodes a rounding away from corners", (v * (1.0 + 2e-16), tri), [-1.35, -1.35, -0.35], 0.35, (8, 8, 3)
    yield "torus of 132 triangles", _torus(11, 6), [-1.5, -1.5, -0.5], 0.3, (11, 12, 5)
    v, tri = _torus(17, 9)
    yield "far from the origin", (v + 1e3, tri), [998.5, 998.6, 999.4], 0.27, (12, 9, 5)
    yield "micrometres", (v * 1e-6, tri), [-1.5e-6, -1.5e-6, -0.5e-6], 0.27e-6, (12, 9, 5)
    yield "grid small against the mesh", (v, tri), [1.3, -0.05, -0.05], 0.01, (9, 9, 9)
    yield "open mesh", (v, tri[: len(tri) // 2]), [-1.5, -1.5, -0.5], 0.27, (12, 11, 5)
    s, k = _cube()
    s = np.concatenate([s, [[0.5, 1e-9, 0.0], [0.5, 0.0, 0.0]]])
    yield "slivers", (s, np.concatenate([k, [[0, 1, 8], [0, 9, 1], [0, 8, 9]]]).astype(np.int32)), [-0.3, -0.3, -0.3], \
        0.21, (8, 8, 8)


@pytest.mark.parametrize("case", list(_cases()), ids=lambda c: c[0])
def test_mesh_grid_equals_the_double_precision_scan(fundem, case):
    _, (v, tri), origin, h, n = case
    got = fundem.levelset_grid("mesh", None, origin, h, n, vertices=v, triangles=tri)
    assert np.array_equal(got, _scan(np.asarray(v), np.asarray(tri), origin, h, n))
