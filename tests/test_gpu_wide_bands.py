"""N^-1 with the automatic plans at half bandwidths that a right-angle tile of 2^17 samples holds
with little room (2^15 and more) or not at all (above 2^16).

Tolerances: FP64 1e-12 (the N^-1 parity bound).  FP32: a transform of 2^17 points and its inverse
are 34 butterfly stages and at most 8 twiddle and untangle products, each rounding to 2^-24
relative in the worst case, 42 * 2^-24 = 2.5e-6."""
import numpy as np
import pytest

from oracle import restate as R

pytestmark = pytest.mark.gpu
TOL64, TOL32 = 1e-12, 2.5e-6


@pytest.mark.parametrize("lam,sizes", [
    ((1 << 15) + 1, [40001, 200003]),   # a right-angle tile is half useful
    ((1 << 15) + 2, [40001, 200003]),   # and just not
    (40000, [39999, 300001]),
    (1 << 16, [300001]),                # a right-angle tile has two outputs
    ((1 << 16) + 1, [70001, 65536]),    # no right-angle tile
    (98306, [150001]),                  # the longest tile is less than a quarter useful
    (131000, [140001]),
])
def test_automatic_plans_of_wide_bands(gpu_ctx, lam, sizes):
    import torch
    import midapack_b200 as mb
    rng = np.random.default_rng(lam)
    t = np.zeros(lam)
    t[0] = 2.0
    t[1:] = rng.standard_normal(lam - 1) * np.exp(-np.arange(1, lam) / (0.3 * lam))
    invtt = np.tile(t, len(sizes))
    v = rng.standard_normal(int(sum(sizes))) + 3.0
    N = mb.Noise(gpu_ctx, sizes, lam, invtt)
    vin = torch.from_numpy(v).cuda()
    out = torch.full_like(vin, float("nan"))
    N.apply(vin, out)
    v32 = vin.float()
    o32 = torch.full_like(v32, float("nan"))
    N.apply_fp32(v32, o32)
    torch.cuda.synchronize()
    # a tile at least a quarter useful wherever there is one
    for tile in (N.tile(), N.tile_fp32()):
        assert 4 * (tile["fft_n"] - 2 * lam) >= tile["fft_n"] or tile["fft_n"] == 1 << 18
    ref = R.stbmm(v, np.array(sizes), lam, invtt)
    assert np.linalg.norm(out.cpu().numpy() - ref) < TOL64 * np.linalg.norm(ref)
    ref32 = R.stbmm(v32.double().cpu().numpy(), np.array(sizes), lam, invtt)
    assert np.linalg.norm(o32.double().cpu().numpy() - ref32) < TOL32 * np.linalg.norm(ref32)
