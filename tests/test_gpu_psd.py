"""Periodograms of blocks whose transform is longer than one CTA's, at the edges
of the transform lengths and with mixed lengths in one call, against scipy.
Tolerances: 1e-12 relative norm per block (the bound of the periodogram tests) and
1e-8 in log10 per bin, as there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [
    [8192],                               # the shortest power of two: two rows
    [2731, 5461, 5462],                   # n + n/2 at and around 8192
    [16384, 8193, 16384, 10922, 10923, 4],
    [131072, 100003, 99999, 100003],      # a length that comes back after another
    [1 << 20, 174763, 349525],            # 2^8 rows; chirp lengths just past and just within 2^18, 2^19
    [700001] * 9,                         # more blocks of a length than one group holds
    [2796202, 5592405],                   # columns of 1024 and 2048 points
])
def test_long_periodograms(gpu_ctx, sizes):
    import torch
    from scipy.signal import welch
    from midapack_b200 import noise as mbn
    rng = np.random.default_rng(len(sizes) + sizes[0])
    x = rng.standard_normal(sum(sizes)) + 0.3
    at = np.concatenate([[0], np.cumsum(sizes)])
    for b, n in enumerate(sizes):
        x[at[b]:at[b + 1]] += np.linspace(0.0, 2.0 + b, n)
    got = mbn.periodogram(torch.from_numpy(x).cuda(), sizes, 100.0, ctx=gpu_ctx).cpu().numpy()
    o = 0
    for b, n in enumerate(sizes):
        _, ref = welch(x[at[b]:at[b + 1]], 100.0, window="hann", nperseg=n, detrend="linear")
        g = got[o:o + n // 2 + 1]
        o += n // 2 + 1
        assert np.linalg.norm(g - ref) < 1e-12 * np.linalg.norm(ref), (b, n)
        big = ref[1:] > 1e-10 * ref[1:].max()
        assert np.abs(np.log10(g[1:][big]) - np.log10(ref[1:][big])).max() < 1e-8, (b, n)
    assert o == len(got)
