"""Periodograms of long blocks against extended precision: errors of the amplitudes no larger
than those of the radix-2 transforms that took these lengths before (BOUND, measured on these inputs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BOUND = {100003: 3.85e-16, 131072: 2.14e-16, 174763: 3.73e-16}


def amplitude_errors(n, got, x):
    import scipy.fft as sf
    ld = np.longdouble
    t = np.arange(n).astype(ld)
    c = t - ld(n - 1) / 2
    win = ld(0.5) - ld(0.5) * np.cos(8 * np.arctan(ld(1)) * t / n)
    scale = 1 / (100 * (win * win).sum())
    out = []
    for g, v in zip(got, x.astype(ld)):
        v = v - v.sum() / n - c * ((c * v).sum() / (c * c).sum())
        p = np.abs(sf.rfft(v * win)) ** 2 * scale
        p[1:(n + 1) // 2] *= 2
        a, b = np.sqrt(g.astype(ld)), np.sqrt(p)
        out.append(float(np.sqrt(((a - b) ** 2).sum() / (b * b).sum())))
    return out


@pytest.mark.parametrize("n", sorted(BOUND))
def test_amplitude_errors(gpu_ctx, n):
    import torch
    from midapack_b200 import noise as mbn
    x = np.random.default_rng(n).standard_normal((12, n))
    got = mbn.periodogram(torch.from_numpy(x.reshape(-1)).cuda(), [n] * 12, 100.0, ctx=gpu_ctx).cpu().numpy().reshape(12, -1)
    e = amplitude_errors(n, got, x)
    assert np.mean(e) <= BOUND[n]
