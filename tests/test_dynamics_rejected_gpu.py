"""Manifolds that the dynamics stage rejects (no points, too many, a body out of
range, one body twice) in the middle of islands, on every route an island can
take: the stage reports them and solves the rest as if they were not there.
Expected: the C restatement of the reference's stage on the same world without
those manifolds, bit for bit; the rejected ones keep their stored impulses."""
import ctypes as C

import numpy as np
import pytest
import torch

import dynio
import reflib
from reactphysics3d_b200 import dynamics as D
from reactphysics3d_b200 import engine
from test_dynamics_islands_gpu import _world

pytestmark = pytest.mark.gpu
PER_MANIFOLD = ("ids", "point_start", "nb_points", "friction_vector1", "friction_vector2", "friction_impulse")


def _stage(name):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return {
        "warps, eight lanes": [("random", 6, 5)] * 7 + [("random", 40, 60)] * 3 + [("chain", 20, 19)],
        "warps, a lane each": [("wide", 128, 64)] * 3 + [("wide", 40, 60)],
        "threads": [("random", 3, 2)] * (40 * sms),
        "CTAs": [("random", 60, 100), ("random", 150, 300), ("chain", 100, 99)],
        "more than CTAs": [("random", 60, 100)] * (sms + 3) + [("random", 150, 300)] * 2,
        "streamed": [("random", 700, 1100)],
    }[name]


@pytest.mark.parametrize("name", ["warps, eight lanes", "warps, a lane each", "threads", "CTAs", "more than CTAs", "streamed"])
def test_rejected_manifolds_are_skipped(cuda_lib, port, name):
    islands = _stage(name)
    w = _world(islands, len(name))
    rng = np.random.default_rng(len(name))
    nm = len(w.a["ids"])
    bad = np.zeros(nm, bool)
    for s, c in zip(w.a["manifold_start"], w.a["manifold_count"]):
        if c > 1:                                    # the middle, the last, and some more of large islands
            k = rng.integers(0, c, 1 + int(c) // 40)
            bad[s + k[:max(1, int(c) - 1)]] = True
    keep = ~bad
    for i, m in enumerate(np.flatnonzero(bad)):
        if i % 4 == 0:
            w.a["nb_points"][m] = 0
        elif i % 4 == 1:
            w.a["nb_points"][m] = 5
        elif i % 4 == 2:
            w.a["ids"][m, 1] = len(w.a["mass"])
        else:
            w.a["ids"][m, 1] = w.a["ids"][m, 0]
    a = {k: np.array(v, copy=True) for k, v in w.a.items()}
    for k in PER_MANIFOLD:
        a[k] = a[k][keep]
    before = np.concatenate([[0], np.cumsum(keep)])
    a["manifold_start"] = before[w.a["manifold_start"]]
    a["manifold_count"] = before[w.a["manifold_start"].astype(np.int64) + w.a["manifold_count"]] - a["manifold_start"]
    params = D.make_params(split=True)
    ref = dynio.run_oracle(C.CDLL(reflib.PORT_LIB), params, D.DynWorld(a, w.nb_enabled, w.nc_enabled))
    ctx = engine.Context(0)
    dev = D.DynWorld(w.a, w.nb_enabled, w.nc_enabled, device="cuda")
    ctx.dynamics_step(params, dev)
    ctx.synchronize()
    assert ctx.device_errors(clear=True) & 4
    h = dev.host()
    for k in D.OUTPUTS:
        x, y = np.asarray(h[k]), np.asarray(ref[k])
        if k in PER_MANIFOLD:
            assert np.array_equal(x[bad].view(np.uint8), np.asarray(w.a[k])[bad].view(np.uint8)), k
            x = x[keep]
        if k == "inv_inertia_world":
            x, y = x[:3 * w.nb_enabled], y[:3 * w.nb_enabled]
        assert np.array_equal(np.ascontiguousarray(x).view(np.uint8), np.ascontiguousarray(y).view(np.uint8)), k
    ctx.close()
