"""Several threads cast rays at one world that does not change, each with its
own output arrays: every call traces every one of its rays.  The threads start
their calls together, so that their clears, launches and copies interleave on
the world's stream."""
import threading

import numpy as np
import pytest
import torch

from reactphysics3d_b200 import _abi as A
from reactphysics3d_b200 import engine, scenes

pytestmark = pytest.mark.gpu


def test_threads_share_a_world(cuda_lib):
    ctx = engine.Context(0)
    sc = scenes.mixed_world()
    w = engine.World(ctx, sc)
    w.update(1.0 / 60.0, 10)
    p = sc.bodies["position"]
    jobs = []
    for k, n in enumerate((1, 33, 1000, 6000)):
        rays = scenes.world_rays(n, p.min(0) - 1.0, p.max(0) + 1.0, seed=k)
        hits, counts = w.raycast(rays, A.RAYCAST_CLOSEST)     # one thread: the answers, and the tables built
        dev = torch.from_numpy(rays.view(np.uint8)).cuda()
        out = torch.zeros((n, A.RAYCAST_HIT_DTYPE.itemsize), dtype=torch.uint8, device="cuda")
        jobs.append((n, dev, out, torch.zeros(n, dtype=torch.int32, device="cuda"), hits, counts))
    assert sum(int(j[5].sum()) for j in jobs) > 100
    rounds, gate, wrong = 300, threading.Barrier(len(jobs)), []

    def run(job):
        n, dev, out, cnt, hits, counts = job
        with torch.cuda.stream(torch.cuda.Stream()):
            for r in range(rounds):
                cnt.fill_(-1)
                torch.cuda.current_stream().synchronize()
                gate.wait()
                w.raycast_device(dev.data_ptr(), n, out.data_ptr(), cnt.data_ptr(), mode=A.RAYCAST_CLOSEST)
                got = cnt.cpu().numpy()
                rec = out.cpu().numpy().view(A.RAYCAST_HIT_DTYPE).reshape(n)
                hit = counts > 0
                if not (np.array_equal(got, counts) and
                        np.array_equal(rec[hit].view(np.uint8), hits[hit, 0].view(np.uint8))):
                    wrong.append((r, n, int((got < 0).sum())))

    torch.cuda.synchronize()
    threads = [threading.Thread(target=run, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:5]
    w.close()
    ctx.close()
