"""More islands than SMs that no kernel can stage in shared memory, in a stage
whose islands are all of that kind: every island is streamed through global
memory, once, bit for bit against the C restatement of the reference's stage.
(The restatement's order is the reference's, so there is no tolerance.)"""
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


@pytest.mark.parametrize("more", [1, 60])
def test_every_streamed_island_is_solved_once(cuda_lib, port, more):
    # 1,100 manifolds: 187 bytes each, 64 KB of hash and 36 KB of staged rows
    # are more than the 227 KB of a CTA
    islands = torch.cuda.get_device_properties(0).multi_processor_count + more
    w = _world([("random", 700, 1100 + k % 3) for k in range(islands)], 70 + more)
    params = D.make_params(split=True)
    ctx = engine.Context(0)
    dev = D.DynWorld(w.a, w.nb_enabled, w.nc_enabled, device="cuda")
    ref = dynio.run_oracle(C.CDLL(reflib.PORT_LIB), params, w.copy())
    ctx.dynamics_step(params, dev)
    ctx.synchronize()
    assert ctx.device_errors(clear=True) & 4 == 0
    h = dev.host()
    for k in D.OUTPUTS:
        a, b = np.asarray(h[k]), np.asarray(ref[k])
        if k == "inv_inertia_world":
            a, b = a[:3 * w.nb_enabled], b[:3 * w.nb_enabled]
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8)), k
    ctx.close()
