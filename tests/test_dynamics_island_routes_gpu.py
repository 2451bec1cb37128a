"""Which islands the contact solver gives a thread each: by the sizes of the
stage's islands and the warps they would share otherwise.  Stages on both sides
of the choice, each checked for the route it takes and bit for bit against the
C restatement of the reference's stage, with and without split impulses."""
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


@pytest.fixture(scope="module")
def ctx(cuda_lib):
    c = engine.Context(0)
    yield c
    c.close()


def _stage(name):
    warps = 6 * torch.cuda.get_device_properties(0).multi_processor_count
    # islands (movable bodies, manifolds), and how many of them get a thread
    one, two, eight, mid = ("random", 2, 1), ("random", 3, 2), ("random", 8, 8), ("random", 30, 40)
    return {
        # an island a warp or less: warps
        "few of one": ([one] * warps, 0),
        # several a warp: a thread's 21 us are less than 8 x 12
        "many of one": ([one] * (8 * warps), 8 * warps),
        # eight manifolds are 266 us on a thread, 4 x 47 on warps
        "some of eight": ([eight] * (4 * warps), 0),
        "many of eight": ([eight] * (7 * warps), 7 * warps),
        # only the small class of a mixture: 21 + 2 x 47 against 4 x 12 + 2 x 47
        "one and eight": ([one, one, eight] * (2 * warps), 4 * warps),
        # beside longer islands on warps the small ones cost nothing there
        "one and mid": ([mid] * 50 + [one] * (4 * warps), 0),
        "two": ([two] * (3 * warps + 1), 0),
        "a single one": ([one], 0),
    }[name]


@pytest.mark.parametrize("split", [True, False])
@pytest.mark.parametrize("name", ["few of one", "many of one", "some of eight", "many of eight", "one and eight",
                                  "one and mid", "two", "a single one"])
def test_routes_and_results(ctx, port, name, split):
    islands, threads = _stage(name)
    w = _world(islands, len(name))
    params = D.make_params(split=split)
    dev = D.DynWorld(w.a, w.nb_enabled, w.nc_enabled, device="cuda")
    ref = dynio.run_oracle(C.CDLL(reflib.PORT_LIB), params, w.copy())
    ctx.dynamics_step(params, dev)
    ctx.synchronize()
    assert ctx.device_errors(clear=True) & 4 == 0
    assert ctx.dynamics_routes() == {"thread": threads, "warp": len(islands) - threads, "cta": 0, "streamed": 0}
    h = dev.host()
    for k in D.OUTPUTS:
        a, b = np.asarray(h[k]), np.asarray(ref[k])
        if k == "inv_inertia_world":
            a, b = a[:3 * w.nb_enabled], b[:3 * w.nb_enabled]
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8)), k
