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
