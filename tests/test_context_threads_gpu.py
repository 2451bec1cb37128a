"""Two contexts with mesh tables of different sizes, each used by a thread of its
own: a launch of one must not take away the shared memory that the other's next
launch needs.  The threads take turns, so the order is fixed."""
import threading

import numpy as np
import pytest

from reactphysics3d_b200 import _abi as A
from reactphysics3d_b200 import engine, scenes

pytestmark = pytest.mark.gpu


def _context(instances):
    ctx = engine.Context(0)
    v, f = scenes.load_hull()
    mesh = ctx.create_convex_mesh(v, f)
    for k in range(instances):
        ctx.create_convex_mesh_shape(mesh, (1.0 + 0.01 * k, 1.0, 1.0))
    sh = np.zeros(2, A.SHAPE_DTYPE)
    sh["kind"], sh["mesh"] = A.SHAPE_CONVEX_MESH, (0, instances - 1)
    ctx.set_shapes(sh)
    return ctx


def test_contexts_of_two_threads_keep_their_launches(cuda_lib):
    rng = np.random.default_rng(5)
    n = 300
    p1, p2 = np.zeros((2, n, 4), np.float32)
    p1[:, :3] = rng.uniform(-5, 5, (n, 3))
    p2[:, :3] = p1[:, :3] + scenes.random_unit_vectors(rng, n) * rng.uniform(0.5, 2.5, n)[:, None]
    pairs = A.HostPairs(np.zeros(n), np.ones(n), p1, scenes.random_quaternions(rng, n), p2, scenes.random_quaternions(rng, n))
    big, small = _context(11), _context(6)      # about 93 and 51 KB of tables, staged in shared memory
    results, errors = [], []

    def call(ctx):
        try:
            results.append(ctx.narrowphase_host(A.ALGO_CONVEX_POLYHEDRON_VS_CONVEX_POLYHEDRON, pairs))
        except engine.Rp3dgError as e:
            errors.append(str(e))

    turn = [threading.Event() for _ in range(3)]

    def first():
        call(big)
        turn[0].set()
        turn[1].wait()
        call(big)

    def second():
        turn[0].wait()
        call(small)
        turn[1].set()

    threads = [threading.Thread(target=t) for t in (first, second)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert np.array_equal(results[0].is_colliding, results[2].is_colliding) and results[0].is_colliding.sum() > n // 4
    big.close()
    small.close()
