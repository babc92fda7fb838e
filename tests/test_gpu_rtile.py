"""Right-angle tiles of N^-1 (plans "r,log2 rows,log2 row length") at the edges
of their range, against the oracle's exact long-double banded product.

Tolerances: FP64 1e-12 (the N^-1 parity bound).  FP32: a transform and its
inverse are at most 2 * 16 butterfly stages and 2 * 5 twiddle products, each
rounding to 2^-24 relative in the worst case, 42 * 2^-24 = 2.5e-6."""
import numpy as np
import pytest

from oracle import restate as R

pytestmark = pytest.mark.gpu
TOL64, TOL32 = 1e-12, 2.5e-6


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def _row(rng, lam):
    t = np.zeros(lam)
    t[0] = 2.0
    t[1:] = rng.standard_normal(lam - 1) * np.exp(-np.arange(1, lam) / (0.3 * lam))
    return t


@pytest.mark.parametrize("lam,sizes,plan", [
    (2, [9, 50, 64, 1], "r,0,9"),             # blocks far shorter than a tile, an odd number of tiles
    (449, [5000, 600, 1001], "r,0,9"),        # widest band of the shortest tile (an eighth useful)
    (300, [5000, 600], "r,0,10"),
    (64, [4096, 777, 130], "r,0,11"),
    (1000, [30001, 999, 8193], "r,0,12"),     # a block of lambda - 1 samples
    (3585, [20000], "r,0,12"),                # widest band of a one-row tile
    (2048, [20000, 4100, 65537], "r,1,12"),
    (5000, [40000, 9001], "r,2,12"),
    (8192, [70000, 8191], "r,3,12"),
    (16384, [70001, 16383], "r,4,12"),
    (2, [300001], "r,4,12"),                  # windows that end past the block by most of a tile
])
def test_right_angle_tiles_vs_exact(gpu_ctx, lam, sizes, plan):
    """Every shape, FP64 and FP32, with a first row of its own per block."""
    import torch
    import midapack_b200 as mb
    rng = np.random.default_rng(lam + len(sizes))
    invtt = np.concatenate([_row(rng, lam) for _ in sizes])
    v = rng.standard_normal(int(sum(sizes))) + 3.0
    N = mb.Noise(gpu_ctx, sizes, lam, invtt).set_plan(plan).set_plan(plan, fp32=True)
    m1, m2 = (1 << int(x) for x in plan.split(",")[1:])
    for tile in (N.tile(), N.tile_fp32()):
        assert tile["fft_n"] == 2 * m1 * m2
        assert tile.get("split") == ([m1, m2] if m1 > 1 else None)
    vin = torch.from_numpy(v).cuda()
    vout = torch.full_like(vin, float("nan"))
    N.apply(vin, vout)
    v32 = vin.float()
    o32 = torch.full_like(v32, float("nan"))
    N.apply_fp32(v32, o32)
    torch.cuda.synchronize()
    assert _rel(vout.cpu().numpy(), R.stbmm(v, np.array(sizes), lam, invtt, exact=True)) < TOL64
    ref32 = R.stbmm(v32.double().cpu().numpy(), np.array(sizes), lam, invtt, exact=True)
    assert _rel(o32.double().cpu().numpy(), ref32) < TOL32


@pytest.mark.parametrize("plan", ["r,0,12", "r,3,12"])
def test_right_angle_tiles_many_units(gpu_ctx, plan):
    """More tiles than one launch group holds, and gaps between the blocks: uncovered rows pass
    through and nothing outside a block is read into it."""
    import torch
    import midapack_b200 as mb
    rng = np.random.default_rng(5)
    lam, n, nb = 700, 120001, 60
    idv = np.arange(nb, dtype=np.int64) * (n + 3) + 1
    rows = [_row(rng, lam) for _ in range(3)]
    invtt = np.concatenate([rows[b % 3] for b in range(nb)])
    N = mb.Noise(gpu_ctx, [n] * nb, lam, invtt, idv=idv).set_plan(plan).set_plan(plan, fp32=True)
    total = int(idv[-1]) + n
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    v = torch.randn(total, dtype=torch.float64, device="cuda", generator=g) + 2.0
    covered = torch.zeros(total, dtype=torch.bool, device="cuda")
    for s in idv:
        covered[int(s):int(s) + n] = True
    v[~covered] = 1e30  # would dominate any sum it leaked into
    out = torch.full_like(v, float("nan"))
    N.apply(v, out)
    o32 = torch.full(v.shape, float("nan"), dtype=torch.float32, device="cuda")
    v32 = v.float()
    N.apply_fp32(v32, o32)
    torch.cuda.synchronize()
    assert torch.equal(out[~covered], v[~covered]) and torch.equal(o32[~covered], v32[~covered])
    for b in (0, 1, 31, nb - 1):
        s = int(idv[b])
        ref = R.stbmm(v[s:s + n].cpu().numpy(), np.array([n]), lam, rows[b % 3])
        assert _rel(out[s:s + n].cpu().numpy(), ref) < TOL64
        assert _rel(o32[s:s + n].double().cpu().numpy(), ref) < TOL32
