"""Edge pairs of two convex polyhedra on the GPU at the sizes where the
warp-per-pair kernels change their route: hulls of 6 to 128 edges (one to four
words of edge masks, a last word that is nearly empty or full), as either
shape, against each other and against boxes, deep inside one another (the
lists of edge pairs overflow) to apart.  Bit-exact against the C oracle, on
fresh pairs and with the first frame's caches."""
import numpy as np
import pytest
from scipy.spatial import ConvexHull

import reflib
from reactphysics3d_b200 import _abi as A
from reactphysics3d_b200 import engine, scenes
from test_narrowphase_gpu import _assert_same

pytestmark = pytest.mark.gpu
POLY = A.ALGO_CONVEX_POLYHEDRON_VS_CONVEX_POLYHEDRON


def _hull(points):
    """Triangulated hull with outward winding."""
    p = np.asarray(points, np.float32)
    faces = []
    for t, eq in zip(ConvexHull(p.astype(np.float64)).simplices, ConvexHull(p.astype(np.float64)).equations):
        a, b, c = p[t].astype(np.float64)
        faces.append([int(k) for k in (t if np.dot(np.cross(b - a, c - a), eq[:3]) > 0 else t[::-1])])
    return p, faces


def _sphere(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, 3))
    return _hull(x / np.linalg.norm(x, axis=1, keepdims=True))


def _prism(n):
    ang = 2 * np.pi * np.arange(n) / n
    ring = np.stack([np.cos(ang), np.sin(ang)], 1)
    v = np.concatenate([np.c_[ring, -np.ones(n) * 0.7], np.c_[ring, np.ones(n) * 0.7]]).astype(np.float32)
    faces = [list(range(n))[::-1], list(range(n, 2 * n))]
    faces += [[k, (k + 1) % n, n + (k + 1) % n, n + k] for k in range(n)]
    return v, faces


def _bipyramid(n):
    ang = 2 * np.pi * np.arange(n) / n
    v = np.concatenate([np.stack([np.cos(ang), np.sin(ang), 0 * ang], 1), [[0, 0, 1], [0, 0, -1]]]).astype(np.float32)
    faces = [[k, (k + 1) % n, n] for k in range(n)] + [[(k + 1) % n, k, n + 1] for k in range(n)]
    return v, faces


def _dome(rings):
    """Rings of 16 vertices under an apex: 32 edges a ring."""
    ang = 2 * np.pi * np.arange(16) / 16
    t = np.linspace(-0.6, 1.0, rings)
    v = np.concatenate([np.stack([np.cos(ang) * np.cos(a), np.sin(ang) * np.cos(a), 0 * ang + np.sin(a)], 1) for a in t]
                       + [[[0.0, 0.0, 1.1]]]).astype(np.float32)
    faces = [list(range(16))[::-1]]
    for r in range(rings):
        for k in range(16):
            a, b = 16 * r + k, 16 * r + (k + 1) % 16
            faces.append([a, b, b + 16, a + 16] if r + 1 < rings else [a, b, 16 * rings])
    return v, faces


HULLS = {"tetrahedron": lambda: _sphere(4, 3), "e30": lambda: _sphere(12, 1), "e33": lambda: _bipyramid(11),
         "e48": lambda: _prism(16), "e63": lambda: _sphere(23, 2), "e64": lambda: _dome(2), "e96": lambda: _sphere(34, 4),
         "e126": lambda: _sphere(44, 5),
         "e128": lambda: _dome(4)}


@pytest.mark.parametrize("first,extra", [(k, 0) for k in HULLS] + [("e128", 14)])
def test_hull_edge_pairs_match_oracle(cuda_lib, port, first, extra):
    """extra: further instances, which make the mesh tables too large for shared memory."""
    port.lib.rp3do_reset()
    ctx = engine.Context(0)
    order = [first] + [k for k in HULLS if k != first]
    shapes = np.zeros(len(order) + 2, A.SHAPE_DTYPE)
    for k, name in enumerate(order):
        v, f = HULLS[name]()
        scale = (1.0, 1.0, 1.0) if k % 2 == 0 else (0.7, 1.2, 0.9)
        for e in (ctx, port):
            assert e.create_convex_mesh_shape(e.create_convex_mesh(v, f), scale) == k
        shapes["kind"][k], shapes["mesh"][k] = A.SHAPE_CONVEX_MESH, k
    for k in range(extra):
        ctx.create_convex_mesh_shape(0, (1.0 + k, 2.0, 1.0))
    shapes["kind"][-2:], shapes["mesh"][-2:] = A.SHAPE_BOX, -1
    shapes["params"][-2, :3], shapes["params"][-1, :3] = (0.6, 0.9, 0.4), (4.0, 0.3, 5.0)
    ctx.set_shapes(shapes)
    rng = np.random.default_rng(17)
    n = 97 * len(shapes)
    other = np.arange(n, dtype=np.int32) % len(shapes)
    swap = rng.random(n) < 0.5
    s1, s2 = np.where(swap, other, 0).astype(np.int32), np.where(swap, 0, other).astype(np.int32)
    pos1, pos2 = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos1[:, :3] = rng.uniform(-3, 3, (n, 3))
    # a quarter nearly concentric, the rest from overlapping to just apart
    dist = np.where(rng.random(n) < 0.25, rng.uniform(0, 0.05, n), rng.uniform(0.6, 2.4, n))
    pos2[:, :3] = pos1[:, :3] + scenes.random_unit_vectors(rng, n) * dist[:, None]
    pairs = A.HostPairs(s1, s2, pos1, scenes.random_quaternions(rng, n), pos2, scenes.random_quaternions(rng, n))
    pairs.cache = A.fresh_cache(n)
    collided = 0
    for frame in range(2):
        pg, pp = pairs.slice(0, n), pairs.slice(0, n)
        pg.cache, pp.cache = pairs.cache.copy(), pairs.cache.copy()
        exp, _ = port.narrowphase(POLY, shapes, pp)
        got = ctx.narrowphase_host(POLY, pg)
        _assert_same(got, exp, pg.cache, pp.cache, f"{first} frame {frame}")
        collided += int(np.sum(exp.is_colliding))
        pairs = reflib.perturb_pairs(pp, rng)
        pairs.cache = reflib.next_frame_cache(pp.cache, exp)
    assert n // 4 < collided < 2 * n
    ctx.close()
