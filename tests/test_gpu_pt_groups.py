"""P^T by map bins at the edges of its slices and groups: bins that fit one slice,
one group and several groups, empty bins, a last bin of few pixels, rows that all hit
one pixel, and unsorted pixels.  FP64 against numpy's sums: 1e-13 relative, the bound of
the pointing tests; two applications equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["one_pixel", "few_bins", "skewed", "random", "two_pixels_far"])
def test_transpose_slices_and_groups(gpu_ctx, kind):
    import torch
    import midapack_b200 as mb
    rng = np.random.default_rng(len(kind))
    m = (1 << 20) + 77
    if kind == "one_pixel":
        p = np.full(m, 5)
    elif kind == "few_bins":                      # 3 bins of 256 pixels, the last one of 7
        p = (np.arange(m) // 3) % (2 * 256 + 7)
    elif kind == "skewed":                        # bins of 1 to 2^19 rows, some empty
        p = np.minimum((2.0 ** (rng.random(m) * 15)).astype(np.int64) * 97 % 40000, 39999)
    elif kind == "random":
        p = rng.integers(0, 30011, m)
    else:                                         # thousands of bins between the two used ones
        p = np.where(np.arange(m) % 1000 == 0, 2_000_000, 3)
    p = p.astype(np.int64)
    p[rng.random(m) < 0.01] = -1
    idx = (3 * p[:, None] + np.arange(3)).astype(np.int32).reshape(-1)
    w = rng.standard_normal(3 * m)
    y = rng.standard_normal(m)
    P = mb.Pointing(gpu_ctx, torch.from_numpy(idx).cuda(), torch.from_numpy(w).cuda(), m)
    d = torch.from_numpy(y).cuda()
    x = torch.full((P.shape()["n_map"],), float("nan"), dtype=torch.float64, device="cuda")
    P.trmatvec(d, x)
    again = torch.full_like(x, float("nan"))
    P.trmatvec(d, again)
    assert torch.equal(x, again)
    pix, loc = np.unique(p[p >= 0], return_inverse=True)
    ok = p >= 0
    ref = np.stack([np.bincount(loc, weights=w.reshape(m, 3)[ok, k] * y[ok], minlength=len(pix)) for k in range(3)], 1)
    mag = np.stack([np.bincount(loc, weights=np.abs(w.reshape(m, 3)[ok, k] * y[ok]), minlength=len(pix)) for k in range(3)], 1)
    assert (np.abs(x.cpu().numpy().reshape(-1, 3) - ref) <= 1e-13 * mag.max()).all()
    assert np.linalg.norm(x.cpu().numpy() - ref.reshape(-1)) <= 1e-13 * np.linalg.norm(mag)
