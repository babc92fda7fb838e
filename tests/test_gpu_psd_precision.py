"""Periodograms of long blocks against extended precision: errors no larger than those of the
radix-2 transforms that took these lengths before (the bounds, measured on these inputs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BOUND = {100003: 3.85e-16, 131072: 2.14e-16, 174763: 3.73e-16}
BOUND_RED = {4599: 6.25e-16, 12909: 2.68e-16, 65536: 3.44e-16}


def densities(n, x):
    """scipy.signal.welch of one segment, in extended precision."""
    import scipy.fft as sf
    ld = np.longdouble
    t = np.arange(n).astype(ld)
    c = t - ld(n - 1) / 2
    win = ld(0.5) - ld(0.5) * np.cos(8 * np.arctan(ld(1)) * t / n)
    scale = 1 / (100 * (win * win).sum())
    out = []
    for v in x.astype(ld):
        v = v - v.sum() / n - c * ((c * v).sum() / (c * c).sum())
        p = np.abs(sf.rfft(v * win)) ** 2 * scale
        p[1:(n + 1) // 2] *= 2
        out.append(p)
    return out


def rel(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b * b).sum()))


@pytest.mark.parametrize("n", sorted(BOUND))
def test_amplitude_errors(gpu_ctx, n):
    import torch
    from midapack_b200 import noise as mbn
    x = np.random.default_rng(n).standard_normal((12, n))
    got = mbn.periodogram(torch.from_numpy(x.reshape(-1)).cuda(), [n] * 12, 100.0, ctx=gpu_ctx).cpu().numpy().reshape(12, -1)
    e = [rel(np.sqrt(g.astype(np.longdouble)), np.sqrt(p)) for g, p in zip(got, densities(n, x))]
    assert np.mean(e) <= BOUND[n]


@pytest.mark.parametrize("n", sorted(BOUND_RED))
def test_density_errors_of_red_noise(gpu_ctx, n):
    """Data whose lowest bins hold most of the power: the least-squares line's rounding counts."""
    import torch
    from midapack_b200 import noise as mbn
    rng = np.random.default_rng(n)
    x = np.cumsum(rng.standard_normal((24, n)), axis=1) * 0.05 + rng.standard_normal((24, n)) + 3.0
    got = mbn.periodogram(torch.from_numpy(x.reshape(-1)).cuda(), [n] * 24, 100.0, ctx=gpu_ctx).cpu().numpy().reshape(24, -1)
    e = [rel(g, p) for g, p in zip(got, densities(n, x))]
    assert np.mean(e) <= BOUND_RED[n]
