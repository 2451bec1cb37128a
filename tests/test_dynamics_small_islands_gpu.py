"""Where the contact solver stops giving small islands a warp each and gives
them a thread each (24 manifolds a warp of the persistent kernel): one manifold
below, at and above that line, islands of one to ten manifolds, bit for bit
against the C restatement of the reference's stage."""
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


@pytest.mark.parametrize("off", [-1, 0, 1, 500])
def test_small_islands_match_the_restatement(cuda_lib, port, off):
    ctx = engine.Context(0)
    total = 24 * 6 * torch.cuda.get_device_properties(0).multi_processor_count + off
    sizes, left = [], total
    while left > 0:
        sizes.append(min(1 + len(sizes) % 10, left))
        left -= sizes[-1]
    w = _world([("random", 6, m) for m in sizes], 40 + off)
    params = D.make_params(split=True)
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
