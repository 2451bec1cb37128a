"""Convex meshes with few edges in batches large enough for a launch of their
own: contexts whose largest mesh is at the limit below which mesh pairs skip the
side masks (14 edges), just above it (15, 16), and with a large hull beside a
tetrahedron, against each other and against boxes.  Bit-exact against the C
oracle, on fresh pairs and with the first frame's caches."""
import numpy as np
import pytest

import reflib
from reactphysics3d_b200 import _abi as A
from reactphysics3d_b200 import engine, scenes
from test_hull_edges_gpu import HULLS, _prism
from test_narrowphase_gpu import _assert_same

pytestmark = pytest.mark.gpu
POLY = A.ALGO_CONVEX_POLYHEDRON_VS_CONVEX_POLYHEDRON


def _pyramid(n):
    """2 n edges."""
    ang = 2 * np.pi * np.arange(n) / n
    v = np.concatenate([np.stack([np.cos(ang), np.sin(ang), 0 * ang - 0.5], 1), [[0, 0, 1]]]).astype(np.float32)
    return v, [list(range(n))[::-1]] + [[k, (k + 1) % n, n] for k in range(n)]


MESHES = {
    "tetrahedra": [HULLS["tetrahedron"], lambda: _prism(3)],
    "14 edges": [lambda: _pyramid(7), HULLS["tetrahedron"], lambda: _prism(4)],
    "15 edges": [lambda: _prism(5), HULLS["tetrahedron"]],
    "16 edges": [lambda: _pyramid(8), lambda: _pyramid(7)],
    "a hull among them": [HULLS["e128"], HULLS["tetrahedron"], lambda: _prism(4)],
}


@pytest.mark.parametrize("name", MESHES)
def test_small_meshes_match_oracle(cuda_lib, port, name):
    port.lib.rp3do_reset()
    ctx = engine.Context(0)
    meshes = MESHES[name]
    shapes = np.zeros(2 * len(meshes) + 1, A.SHAPE_DTYPE)
    shapes["kind"], shapes["mesh"] = A.SHAPE_CONVEX_MESH, np.arange(len(shapes))
    for k, make in enumerate(meshes + meshes):
        v, f = make()
        for e in (ctx, port):
            assert e.create_convex_mesh_shape(e.create_convex_mesh(v, f), (0.8, 1.1, 0.9) if k % 2 else (1.0, 1.0, 1.0)) == k
    shapes["kind"][-1], shapes["mesh"][-1], shapes["params"][-1, :3] = A.SHAPE_BOX, -1, (0.6, 0.9, 0.4)
    ctx.set_shapes(shapes)
    rng = np.random.default_rng(23)
    n = 6007
    s1, s2 = rng.integers(0, len(shapes), (2, n)).astype(np.int32)
    pos1, pos2 = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos1[:, :3] = rng.uniform(-3, 3, (n, 3))
    dist = np.where(rng.random(n) < 0.25, rng.uniform(0, 0.05, n), rng.uniform(0.5, 2.2, n))
    pos2[:, :3] = pos1[:, :3] + scenes.random_unit_vectors(rng, n) * dist[:, None]
    pairs = A.HostPairs(s1, s2, pos1, scenes.random_quaternions(rng, n), pos2, scenes.random_quaternions(rng, n))
    pairs.cache = A.fresh_cache(n)
    collided = 0
    for frame in range(2):
        pg, pp = pairs.slice(0, n), pairs.slice(0, n)
        pg.cache, pp.cache = pairs.cache.copy(), pairs.cache.copy()
        exp, _ = port.narrowphase(POLY, shapes, pp)
        got = ctx.narrowphase_host(POLY, pg)
        _assert_same(got, exp, pg.cache, pp.cache, f"{name} frame {frame}")
        collided += int(np.sum(exp.is_colliding))
        pairs = reflib.perturb_pairs(pp, rng)
        pairs.cache = reflib.next_frame_cache(pp.cache, exp)
    assert n // 4 < collided < 2 * n
    ctx.close()
