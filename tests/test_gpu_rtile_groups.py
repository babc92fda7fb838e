"""Right-angle tiles of several rows in launch groups that share a scratch: how many groups a call
takes, and its values where groups reuse each other's scratch (three groups and more).

Tolerances: FP64 1e-12 (the N^-1 parity bound); FP32 2.5e-6 (42 roundings of 2^-24, as in the
right-angle tests); solves of the same columns with two FP32 plans 1e-8 (the bound between
multi-RHS and FP64 columns: both refine to a residual of 1e-12)."""
import numpy as np
import pytest

from midapack_b200 import synth

pytestmark = pytest.mark.gpu
E = 131072 - 2 * 2                       # outputs of a 16 x 4096 tile at half bandwidth 3


def _sizes(tiles):
    """Blocks of up to seven tiles, the last tile of each mostly empty."""
    out = []
    while tiles > 0:
        k = min(7, tiles)
        out.append(E * (k - 1) + 1000 + len(out))
        tiles -= k
    return out


@pytest.mark.parametrize("fp32,tiles,groups", [
    (False, 5, 1),      # tiles of 1 MB: one group up to 32 MB
    (False, 31, 1),
    (False, 32, 2),
    (False, 128, 2),    # two halves of 64 MB
    (False, 129, 3),
    (True, 63, 1),      # tiles of 0.5 MB
    (True, 64, 2),
    (True, 257, 3),
    (True, 600, 5),
])
def test_launch_groups(gpu_ctx, fp32, tiles, groups):
    import torch
    import midapack_b200 as mb
    sizes = _sizes(tiles)
    row = np.array([2.0, -0.7, 0.4])
    N = mb.Noise(gpu_ctx, sizes, 3, np.tile(row, len(sizes))).set_plan("r,4,12", fp32=fp32)
    assert (N.tile_fp32() if fp32 else N.tile())["n_tiles"] == tiles
    g = torch.Generator(device="cuda")
    g.manual_seed(tiles)
    v = torch.randn(sum(sizes), dtype=torch.float32 if fp32 else torch.float64, device="cuda", generator=g)
    out = torch.full_like(v, float("nan"))
    n0 = gpu_ctx.launches
    (N.apply_fp32 if fp32 else N.apply)(v, out)
    # three kernels a group; one or two for the block means
    assert (gpu_ctx.launches - n0 - 1) // 3 == groups
    at = 0
    for n in sizes:
        b = v[at:at + n].double()
        b = b - b.mean()
        ref = row[0] * b
        for k in (1, 2):
            ref[k:] += row[k] * b[:-k]
            ref[:-k] += row[k] * b[k:]
        assert torch.linalg.norm(out[at:at + n].double() - ref) < (2.5e-6 if fp32 else 1e-12) * torch.linalg.norm(ref)
        at += n


def test_groups_of_a_batch_with_stopped_columns(gpu_ctx):
    """Eight slots of 48 tiles: three groups; columns of unlike difficulty stop at unlike iterations."""
    import torch
    import midapack_b200 as mb
    wl = synth.small(n_det=16, n_samp=1 << 18, block_len=1 << 18, lam=512, gap_frac=0.01, seed=3)
    m = wl.n_samples
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    noise = torch.randn((9, m), dtype=torch.float32, device="cuda", generator=g)
    noise[1] = noise[1].cumsum(0) * 1e-2
    noise[4, m // 16:] = 0
    got = []
    for plan in ("r,4,12", "r,0,12"):
        P = mb.Pointing(gpu_ctx, d(wl.pix), d(wl.weights), m, 3)
        N = mb.Noise(gpu_ctx, wl.block_sizes, wl.lam, wl.invtt).set_plan(plan, fp32=True)
        x, *_, ci, info = mb.gls_solve_multi(gpu_ctx, P, N, noise, tol=1e-12, maxiter=900, slots=8)
        assert info.slots == 8 and all(c.converged for c in ci)
        got.append(x.clone())
        P.close()
        N.close()
    assert len({c.iterations for c in ci}) > 1
    for a, b in zip(*got):
        assert torch.linalg.norm(a - b) < 1e-8 * torch.linalg.norm(b)
