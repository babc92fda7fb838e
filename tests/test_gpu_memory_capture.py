"""Closing objects beside another thread's stream capture, and the next objects taking their
device memory while work on them is still queued elsewhere."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def _pointing(ctx, m, mod):
    import torch
    import midapack_b200 as mb
    idx = (torch.arange(m, device="cuda", dtype=torch.int32) % mod)[:, None] * 3 + torch.arange(3, device="cuda", dtype=torch.int32)
    w = torch.ones(3 * m, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return mb.Pointing(ctx, idx.reshape(-1), w, m)


def test_closing_beside_a_capture(gpu_ctx):
    """A thread that closes an operator does not end a capture of another thread (thread-local mode)."""
    import torch
    P = _pointing(gpu_ctx, 1 << 20, 5000)
    y = torch.ones(P.m, dtype=torch.float64, device="cuda")
    x = torch.empty(15000, dtype=torch.float64, device="cuda")
    P.trmatvec(y, x)
    torch.cuda.synchronize()
    go, done = threading.Event(), threading.Event()

    def closer():
        go.wait(30)
        P.close()
        done.set()

    th = threading.Thread(target=closer)
    th.start()
    a = torch.ones(1024, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        b = a * 2
        go.set()
        assert done.wait(30)
        c = b + 1
    th.join()
    g.replay()
    torch.cuda.synchronize()
    assert bool((c == 3).all())


def test_closed_memory_is_taken_after_its_queued_work(gpu_ctx):
    """P^T queued behind 50 ms of other work, the pointing closed and another of the same sizes built on
    another stream: the queued product still sees its own lists."""
    import torch
    import midapack_b200 as mb
    m = 1 << 21
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        ctx2 = mb.Context(0)                        # on the side stream
    y = torch.arange(m, dtype=torch.float64, device="cuda")
    P = _pointing(ctx2, m, 4000)
    x = torch.empty(12000, dtype=torch.float64, device="cuda")
    P.trmatvec(y, x)                                # builds the lists
    ctx2.synchronize()
    ref = x.clone()
    x.fill_(0)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(100_000_000)
    P.trmatvec(y, x)
    P.close()
    Q = _pointing(gpu_ctx, m, 3999)
    q = torch.empty(3 * 3999, dtype=torch.float64, device="cuda")
    Q.trmatvec(y, q)
    torch.cuda.synchronize()
    assert torch.equal(x, ref)
    want = torch.zeros(3999, dtype=torch.float64, device="cuda").index_add_(0, torch.arange(m, device="cuda") % 3999, y)
    assert torch.allclose(q.view(-1, 3)[:, 0], want, rtol=1e-13)
    Q.close()
    ctx2.close()


def test_the_last_context_takes_the_cache_along():
    """In a process of its own: nothing of the library's stays on the device once its contexts are closed."""
    import os
    import subprocess
    import sys
    code = """
import torch, midapack_b200 as mb
def used():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, total = torch.cuda.mem_get_info()
    return total - free
m = 1 << 24
def once():
    idx = (torch.arange(m, device="cuda", dtype=torch.int32) % 5000)[:, None] * 3 + torch.arange(3, device="cuda", dtype=torch.int32)
    w = torch.ones(3 * m, dtype=torch.float64, device="cuda")
    y = torch.ones(m, dtype=torch.float64, device="cuda")
    x = torch.empty(15000, dtype=torch.float64, device="cuda")
    ctx = mb.Context(0)
    P = mb.Pointing(ctx, idx.reshape(-1), w, m)
    P.trmatvec(y, x)
    P.close()
    late = mb.Pointing(ctx, idx.reshape(-1), w, m)
    late.trmatvec(y, x)
    ctx.close()
    late.close()          # after the last context: nothing to keep it for
once()                    # kernels and tables are loaded
ctx = mb.Context(0)
ctx.trim()
ctx.close()
start = used()
once()
print(used() - start)
"""
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, check=True,
                         cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert abs(int(out.stdout.split()[-1])) <= 8 << 20, out.stdout
