"""The library's cache of freed device memory: reused by the next objects, bounded, and
given back by a context's trim."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_freed_memory_is_reused_bounded_and_given_back(gpu_ctx):
    import torch
    import midapack_b200 as mb

    def used():
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free

    m = 1 << 24
    idx = (torch.arange(m, device="cuda", dtype=torch.int32) % 5000)[:, None] * 3 + torch.arange(3, device="cuda", dtype=torch.int32)
    w = torch.ones(3 * m, dtype=torch.float64, device="cuda")
    y = torch.ones(m, dtype=torch.float64, device="cuda")
    x = torch.empty(15000, dtype=torch.float64, device="cuda")
    gpu_ctx.trim()
    start = used()

    def one():
        P = mb.Pointing(gpu_ctx, idx.reshape(-1).contiguous(), w, m)
        P.trmatvec(y, x)
        P.close()
        return x.clone()

    first = one()
    after = used()
    for _ in range(5):
        assert torch.equal(one(), first)
    assert used() <= after + (8 << 20)          # the same blocks again
    assert used() <= start + (2 << 30) + (256 << 20)
    many = [mb.Pointing(gpu_ctx, idx.reshape(-1).contiguous(), w, m) for _ in range(40)]
    for P in many:
        P.trmatvec(y, x)
        P.close()
    del many
    torch.cuda.empty_cache()
    assert used() <= start + (2 << 30) + (256 << 20)
    gpu_ctx.trim()
    assert used() <= start + (64 << 20)
    assert np.isfinite(first.cpu().numpy()).all()
