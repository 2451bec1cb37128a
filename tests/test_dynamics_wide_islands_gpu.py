"""Islands on warps whose levels are wide (a lane a manifold) and narrow (eight
lanes), around the line between the two and at the sizes of the stage, in
stages with more islands above 64 manifolds than SMs, so that the islands stay
on warps: bit for bit against the C restatement of the reference's stage."""
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

# (kind, movable bodies, manifolds); "wide" islands are levels of nb / 2 manifolds
SHAPES = {
    "levels of 8, two chunks": [("wide", 16, 72)],            # 2 chunks a round: eight lanes
    "levels of 9, three chunks": [("wide", 18, 72)],          # 3 chunks a round: one lane
    "levels of 32 and 33": [("wide", 64, 96), ("wide", 66, 99)],
    "random": [("random", 130, 200), ("random", 250, 220), ("random", 60, 65)],
    # the two fixed bodies take slots too: "random" islands reach both
    "304 bodies": [("random", 302, 256), ("wide", 304, 256)],
    "305 bodies": [("random", 303, 256), ("wide", 306, 256)],
    "512 and 513 manifolds": [("random", 90, 512), ("wide", 100, 512), ("random", 90, 513)],
    "chains": [("chain", 66, 65), ("chain", 200, 256)],
}


@pytest.mark.parametrize("split", [True, False])
@pytest.mark.parametrize("name", SHAPES)
def test_islands_on_warps_match_the_restatement(cuda_lib, port, name, split):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    shapes = SHAPES[name]
    islands = (shapes * (1 + (sms + 1) // len(shapes)))[:sms + 1 + len(shapes)]
    w = _world(islands, len(name))
    params = D.make_params(split=split)
    ctx = engine.Context(0)
    dev = D.DynWorld(w.a, w.nb_enabled, w.nc_enabled, device="cuda")
    ref = dynio.run_oracle(C.CDLL(reflib.PORT_LIB), params, w.copy())
    ctx.dynamics_step(params, dev)
    ctx.synchronize()
    assert ctx.device_errors(clear=True) & 4 == 0
    r = ctx.dynamics_routes()
    if name != "512 and 513 manifolds":
        assert r == {"thread": 0, "warp": len(islands), "cta": 0, "streamed": 0}, r
    else:   # 513 do not fit a warp's stage
        assert r["cta"] == sum(m == 513 for _, _, m in islands) and r["warp"] + r["cta"] == len(islands), r
    h = dev.host()
    for k in D.OUTPUTS:
        a, b = np.asarray(h[k]), np.asarray(ref[k])
        if k == "inv_inertia_world":
            a, b = a[:3 * w.nb_enabled], b[:3 * w.nb_enabled]
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8)), k
    ctx.close()
