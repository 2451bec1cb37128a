"""Batch sizes at which the thread-per-pair narrow-phase kernels change how many
pairs a warp takes (one up to 8 warps a multiprocessor, then two, ... 32) and
at which box-box batches start to be grouped: every pair is done once, bit-exact
against the C oracle."""
import numpy as np
import pytest
import torch

import edgecases
import reflib
from reactphysics3d_b200 import _abi as A
from reactphysics3d_b200 import engine, scenes
from test_narrowphase_gpu import _assert_same, _register_hulls

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_warp", [0, 1, 2, 3, 31, 32, 40])
def test_every_batch_size_matches_oracle(cuda_lib, port, per_warp):
    port.lib.rp3do_reset()
    _register_hulls(port)
    ctx = engine.Context(0)
    _register_hulls(ctx)
    warps = 8 * torch.cuda.get_device_properties(0).multi_processor_count
    sizes = (1, 31, 33, 4095, 4096) if per_warp == 0 else (per_warp * warps, per_warp * warps + 1)
    top = max(sizes)
    sc = scenes.narrowphase_scene(total_pairs=7 * top, seed=5, hull=edgecases.load_hull())
    ctx.set_shapes(sc.shapes)
    names = ["box_box", "capsule_box"] if per_warp > 3 else ["sphere_box", "capsule_box", "box_box", "hull_box", "capsule_capsule"]
    for name in names:
        algo, pairs = sc.batches[name]
        full = pairs.slice(0, top)
        full.cache = A.fresh_cache(top)
        exp, _ = port.narrowphase(algo, sc.shapes, full)
        for n in sizes:
            p = pairs.slice(0, n)
            p.cache = A.fresh_cache(n)
            got = ctx.narrowphase_host(algo, p)
            part = A.HostContacts(n, exp.max_contacts)
            for f in ("is_colliding", "nb_contacts"):
                getattr(part, f)[...] = getattr(exp, f)[:n]
            for f in ("normal_depth", "local1", "local2"):
                getattr(part, f)[...] = getattr(exp, f)[:, :n]
            _assert_same(got, part, p.cache, full.cache[:n], f"{name} n={n}")
    ctx.close()


@pytest.mark.parametrize("off", [-700, 0, 1, 2000])
def test_mixed_mesh_combinations_match_oracle(cuda_lib, port, off):
    """Hulls and boxes in every order in one batch, around the size (one pair a
    resident warp) at which the combinations get launches of their own."""
    port.lib.rp3do_reset()
    _register_hulls(port)
    ctx = engine.Context(0)
    _register_hulls(ctx)
    n = 16 * torch.cuda.get_device_properties(0).multi_processor_count + off
    sc = scenes.narrowphase_scene(total_pairs=7 * n, seed=9, hull=edgecases.load_hull())
    ctx.set_shapes(sc.shapes)
    algo, pairs = sc.batches["hull_box"]
    pairs = pairs.slice(0, n)
    rng = np.random.default_rng(4)
    hull, box, turn = pairs.shape1.copy(), pairs.shape2.copy(), rng.integers(0, 4, n)
    pairs.shape1[:] = np.where(turn == 0, hull, np.where(turn == 1, box, np.where(turn == 2, hull, np.roll(box, 1))))
    pairs.shape2[:] = np.where(turn == 0, box, np.where(turn == 1, hull, np.where(turn == 2, np.roll(hull, 1), box)))
    a, b = pairs.slice(0, n), pairs.slice(0, n)
    a.cache, b.cache = A.fresh_cache(n), A.fresh_cache(n)
    exp, _ = port.narrowphase(algo, sc.shapes, a)
    got = ctx.narrowphase_host(algo, b)
    _assert_same(got, exp, b.cache, a.cache, f"n={n}")
    assert len(np.unique(turn)) == 4 and exp.is_colliding.sum() > n // 10
    ctx.close()
