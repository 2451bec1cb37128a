"""Several threads order the same context's stream against streams of their own
at the same time: work that a thread queues on the context's stream after its
order_in sees what its own stream wrote before, and its own stream sees that
work after its order_out, however the threads' calls interleave."""
import threading

import pytest
import torch

from reactphysics3d_b200 import engine

pytestmark = pytest.mark.gpu


def test_threads_order_their_own_streams(cuda_lib):
    ctx = engine.Context(0)
    ctx.order_in()
    own = ctx.torch_stream()
    nthreads, rounds, n = 4, 60, 1 << 22
    gate, wrong = threading.Barrier(nthreads), []
    bufs = [tuple(torch.zeros(n, device="cuda") for _ in range(3)) for _ in range(nthreads)]
    torch.cuda.synchronize()

    def run(k):
        src, mid, out = bufs[k]
        with torch.cuda.stream(torch.cuda.Stream()):
            for r in range(rounds):
                gate.wait()
                for _ in range(8):          # late: the copies below have to wait for it
                    src.add_(1.0)
                ctx.order_in()
                with torch.cuda.stream(own):
                    mid.copy_(src)
                ctx.order_out()
                out.copy_(mid)
                src.sub_(7.0)               # ... and this for the copy on the context's stream
                if not bool((out == 8.0 + r).all()):
                    wrong.append((k, r))

    threads = [threading.Thread(target=run, args=(k,)) for k in range(nthreads)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:5]
    torch.cuda.synchronize()
    ctx.close()
