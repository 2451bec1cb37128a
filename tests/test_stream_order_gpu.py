"""Ordering of the context's stream against torch's current stream: inputs
written on that stream just before a call are the ones it reads, results are
there for the stream's next work, on the default stream, a side stream, the
context's own stream and in a captured graph; calls from two threads on two
streams keep their own order."""
import threading

import numpy as np
import pytest
import torch

import reflib
from reactphysics3d_b200 import _abi as A
from reactphysics3d_b200 import engine, scenes

pytestmark = pytest.mark.gpu


def _setup(n):
    ctx = engine.Context(0)
    sc = scenes.narrowphase_scene(total_pairs=7 * n, seed=3)
    ctx.create_convex_mesh_shape(ctx.create_convex_mesh(sc.hull_vertices, sc.hull_faces))
    ctx.set_shapes(sc.shapes)
    algo, pairs = sc.batches["box_box"]
    return ctx, algo, pairs.slice(0, n)


def _late_inputs(ctx, algo, pairs, dp, out, busy, src):
    """The inputs are zero until a copy queued behind slow work fills them."""
    for _ in range(4):
        busy.mul_(1.0001)
    dp.pos1.copy_(src[0])
    dp.pos2.copy_(src[1])
    ctx.narrowphase_device(algo, dp, out)
    res = (out.is_colliding.clone(), out.nb_contacts.clone(), out.normal_depth.clone())
    dp.pos1.zero_()
    dp.pos2.zero_()
    return res


@pytest.mark.parametrize("where", ["default", "side", "own", "graph", "threads"])
def test_calls_are_ordered_with_the_current_stream(cuda_lib, where):
    n = 5000
    ctx, algo, pairs = _setup(n)
    exp = ctx.narrowphase_host(algo, pairs.slice(0, n))

    def job(stream, res):
        with torch.cuda.stream(stream):
            dp, out = engine.DevicePairs(pairs), engine.DeviceContacts(n)
            busy = torch.ones(64 * 1024 * 1024, device="cuda")
            src = dp.pos1.clone(), dp.pos2.clone()
            dp.pos1.zero_()
            dp.pos2.zero_()
            if where == "graph":
                ctx.narrowphase_device(algo, dp, out)   # grows what the call keeps
                torch.cuda.synchronize()
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=stream):
                    r = _late_inputs(ctx, algo, pairs, dp, out, busy, src)
                g.replay()
                g.replay()
                torch.cuda.synchronize()
                r = tuple(x.cpu().numpy() for x in r)
                del g
                res.append(r)
                return
            for _ in range(3):
                r = _late_inputs(ctx, algo, pairs, dp, out, busy, src)
            res.append(tuple(x.cpu().numpy() for x in r))

    results = []
    if where == "threads":
        # one call at a time, from either thread
        for _ in range(2):
            t = threading.Thread(target=job, args=(torch.cuda.Stream(), results))
            t.start()
            t.join()
    else:
        job({"default": torch.cuda.default_stream(), "own": ctx.torch_stream()}.get(where) or torch.cuda.Stream(), results)
    mask = exp.valid_mask()
    for col, nb, nd in results:
        assert np.array_equal(col, exp.is_colliding) and np.array_equal(nb, exp.nb_contacts)
        assert np.array_equal(nd.view(np.uint32)[mask], exp.normal_depth.view(np.uint32)[mask])
    assert exp.is_colliding.sum() > 100
    torch.cuda.synchronize()
    ctx.close()
