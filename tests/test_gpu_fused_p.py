"""P fused with the chunk sums of its block means, as one operator application
P^T N^-1 P, at the edges of its row chunks: odd starts and ends, blocks of one or
two rows, chunks that end with a block, and weights that are not 16-byte aligned.
Tolerance: 1e-12 relative, the parity bound of the FP64 operators."""
import numpy as np
import pytest

from oracle import restate as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("sizes,tail", [([1], 0), ([2000] * 70 + [65537] * 30, 5), ([2, 1, 3, 1], 0), ([2047, 2049, 1, 4098, 2], 0), ([4096, 2048, 6145], 0),
                                        ([500, 700], 333)])   # rows past the last block pass through N^-1
def test_operator_over_chunk_edges(gpu_ctx, sizes, tail, shift):
    import torch
    import midapack_b200 as mb
    from midapack_b200.dist import GpuShard
    rng = np.random.default_rng(len(sizes) + shift)
    m, npix, lam = int(sum(sizes)) + tail, 40, 2
    p = rng.integers(0, npix, m)
    p[rng.random(m) < 0.05] = -1
    p[0] = 3
    idx = (3 * p[:, None] + np.arange(3)).astype(np.int32).reshape(-1)
    w = rng.standard_normal(3 * m)
    invtt = np.tile([2.0, -0.7], len(sizes))
    buf = torch.zeros(3 * m + 1, dtype=torch.float64, device="cuda")
    buf[shift:shift + 3 * m] = torch.from_numpy(w).cuda()
    z = torch.zeros(m, dtype=torch.float64, device="cuda")
    shard = GpuShard(gpu_ctx, torch.from_numpy(idx).cuda(), buf[shift:shift + 3 * m], z, z, sizes, lam, invtt)
    pix = np.unique(p[p >= 0])
    x = rng.standard_normal(3 * len(pix))
    q = shard.apply(torch.from_numpy(x).cuda()).cpu().numpy()
    shard.close()
    loc = np.searchsorted(pix, np.maximum(p, 0))
    ok = p >= 0
    y = np.where(ok, (w.reshape(m, 3) * x.reshape(-1, 3)[loc % len(pix)]).sum(1), 0.0)
    n = R.stbmm(y, np.array(sizes), lam, invtt, exact=True)
    ref = np.zeros((len(pix), 3))
    np.add.at(ref, loc[ok], w.reshape(m, 3)[ok] * n[ok][:, None])
    scale = np.linalg.norm(w) * np.linalg.norm(n) + np.linalg.norm(ref)  # a lone row's mean removal leaves zero
    assert np.linalg.norm(q - ref.reshape(-1)) <= 1e-12 * max(scale, np.linalg.norm(y))
