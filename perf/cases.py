"""Workloads that stand for this framework's use, and how to run one pass of each.

A case is one call that a map-making program makes through the package's
public entry points, on inputs of the survey's kind: detectors that sweep a
flat grid back and forth under a rotating half-wave plate, 1/f noise, one
stationary interval (Toeplitz block) per detector or per piece of a detector,
about 1 % flagged samples, and a noise row of its own for every block, as the
rows estimated from data are.

op            the call
p             Pointing.matvec, map to time stream (FP64)
pt            Pointing.trmatvec, time stream to map (FP64)
ninv          Noise.apply / Noise.apply_fp32, the inverse noise weighting
solve         gls_solve on a resident pointing and noise operator (FP64 PCG)
map           new pointing and noise operator, then gls_solve_mixed: the
              whole way from device arrays to a map
multi         gls_solve_multi, Monte-Carlo columns over one pointing
psd           noise.periodogram, the input side of the noise rows
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import midapack_b200 as mb
from midapack_b200 import noise as mb_noise
from midapack_b200.synth import F_HWP, F_MIN, FS

DEV = "cuda"


# --------------------------------------------------------------------------- the cases
def listed():
    return [
        # one short interval of one detector (the reference's own test stream has 12000
        # samples): the latency of a call, what a quick-look loop over intervals pays
        dict(name="p_interval", op="p", n_det=1, n_samp=12000, side=64, gap=0.01),
        # scanning a map into 16 detectors' streams, every iteration of a large solve
        dict(name="p_scan", op="p", n_det=16, n_samp=1 << 22, side=1024, gap=0.01),
        # binning a few short streams, odd lengths (the pointing stays below the size from
        # which rows are grouped by map bin)
        dict(name="pt_interval", op="pt", n_det=4, n_samp=50001, side=96, gap=0.01),
        # the adjoint on the large map of the at-scale workload, a sixteenth of its samples
        dict(name="pt_scan", op="pt", n_det=16, n_samp=1 << 22, side=2048, gap=0.01),
        # weighting four short intervals: a launch-bound call
        dict(name="ninv_interval", op="ninv", n_blk=4, n=12000, ragged=False, lam=512, fp32=False),
        # the at-scale intervals (2^20 samples, half bandwidth 2^14), FP64 and the FP32 operator of
        # the mixed-precision solves: the call that most of a solve's time goes to
        dict(name="ninv_long", op="ninv", n_blk=64, n=1 << 20, ragged=False, lam=1 << 14, fp32=False),
        dict(name="ninv32_long", op="ninv", n_blk=64, n=1 << 20, ragged=False, lam=1 << 14, fp32=True),
        # intervals as a real schedule cuts them: unequal odd lengths, a band that is no power of two
        dict(name="ninv32_ragged", op="ninv", n_blk=24, n=700001, ragged=True, lam=3001, fp32=True),
        # the CPU-runnable reference configuration (4 detectors x 2^20, 256x192, half bandwidth 2^12),
        # operators resident, as a serving process keeps them
        dict(name="solve_fp64", op="solve", n_det=4, n_samp=1 << 20, side=256, lam=1 << 12, gap=0.01, tol=1e-8),
        # time to map from new data in mixed precision: compression, noise operator, preconditioner, solve,
        # to a residual at which maps of two pipelines can be told apart
        dict(name="map_mixed", op="map", n_det=8, n_samp=1 << 20, side=512, lam=1 << 13, gap=0.01, tol=1e-12),
        # noise realisations over one pointing
        dict(name="multi_rhs", op="multi", n_det=4, n_samp=1 << 19, side=192, lam=1 << 12, gap=0.01, cols=8,
             tol=1e-12),
        # periodograms of unequal intervals of no power-of-two length (the fit that follows them ends on a
        # flat minimum, where rounding alone moves its rows by 1e-7, so the rows themselves say little)
        dict(name="psd_intervals", op="psd", n_blk=32, n=200003, ragged=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["p", "pt", "ninv", "ninv", "ninv", "solve", "map", "multi", "psd"])
    if op in ("p", "pt"):
        n_det = _log(rng, 1, 32)
        n_samp = _log(rng, 8192, min(1 << 23, (1 << 26) // n_det))
        return dict(op=op, n_det=n_det, n_samp=n_samp, side=_log(rng, 64, 2048), gap=rng.choice([0.0, 0.01, 0.03]))
    if op == "ninv":
        n_blk = _log(rng, 1, 64)
        n = _log(rng, 8192, min(1 << 23, (1 << 26) // n_blk))
        lam = _log(rng, 64, min(1 << 14, n // 4))
        return dict(op=op, n_blk=n_blk, n=n, ragged=rng.random() < 0.4, lam=lam, fp32=rng.random() < 0.5)
    if op == "psd":
        n_blk = _log(rng, 1, 32)
        n = rng.choice([_log(rng, 4096, 200003), 1 << rng.randint(12, 18)])
        return dict(op=op, n_blk=n_blk, n=n, ragged=rng.random() < 0.4)
    n_det = _log(rng, 1, 8 if op == "map" else 4)
    n_samp = _log(rng, 1 << 16, (1 << 19) if op == "multi" else (1 << 20))
    # 24 samples a pixel at least, so that no pixel is cut for want of angles
    side = min(_log(rng, 48, 512), int(math.sqrt(n_det * n_samp / 24 * 4 / 3)))
    case = dict(op=op, n_det=n_det, n_samp=n_samp, side=side, lam=_log(rng, 256, min(1 << 13, n_samp // 8)), gap=0.01,
                tol=1e-8 if op == "solve" else 1e-12)
    return dict(case, cols=rng.randint(2, 8)) if op == "multi" else case


# --------------------------------------------------------------------------- inputs
@functools.cache
def _context():
    return mb.Context(0)


def _grid(side):
    """Width and height (4:3); a scan that comes back to a pixel after a multiple of the half-wave
    plate's period would see it under one angle only, so the height is moved off such periods."""
    period = int(FS / (2 * F_HWP))
    w, h = side + (side % period == 0), 3 * side // 4
    while min(w * h % period, -w * h % period) < 3:
        h += 1
    return w, h


def _scan(case, g):
    """(pixel indices int32 [3 Ns], weights FP64 [3 Ns]) of the scan."""
    w, h = _grid(case["side"])
    n_det, n = case["n_det"], case["n_samp"]
    t = torch.arange(n, device=DEV)
    run, u = t // w, t % w
    off = torch.randint(0, 1 << 30, (n_det, 2), generator=g, device=DEV)
    col = (torch.where(run % 2 == 0, u, w - 1 - u)[None] + off[:, 1:]) % w
    p = (((run[None] + off[:, :1]) % h) * w + col).to(torch.int32).reshape(-1)
    if case["gap"] > 0:
        p[torch.rand(p.numel(), generator=g, device=DEV) < case["gap"]] = -1
    pix = (3 * p[:, None] + torch.arange(3, device=DEV, dtype=torch.int32)).reshape(-1)
    two_psi = (math.pi / 2 * (torch.arange(n_det, device=DEV, dtype=torch.float64) % 4)[:, None]
               + 4 * math.pi * F_HWP / FS * t.to(torch.float64)[None]).reshape(-1)
    return pix, torch.stack((torch.ones_like(two_psi), torch.cos(two_psi), torch.sin(two_psi)), dim=1).reshape(-1)


def _psd(n, fknee):
    f = torch.fft.rfftfreq(n, 1 / FS, dtype=torch.float64, device=DEV)
    return 1 + fknee / (f + F_MIN)


def _noise(n, fknee, g):
    """1/f noise of n samples: white noise filtered with the square root of the PSD."""
    m = 1 << (n - 1).bit_length()
    white = torch.randn(m, dtype=torch.float64, device=DEV, generator=g)
    return torch.fft.irfft(torch.fft.rfft(white) * torch.sqrt(_psd(m, fknee)), n=m)[:n]


def _row(n, lam, fknee):
    """First row of a block's inverse-noise matrix: inverse PSD, Gaussian apodisation, lam taps."""
    m = 1 << (n - 1).bit_length()
    k = torch.arange(lam, dtype=torch.float64, device=DEV)
    return torch.fft.irfft(1 / _psd(m, fknee), n=m)[:lam] * torch.exp(-0.5 * (k / (lam / 3)) ** 2)


def _blocks(case):
    """Block lengths: equal, or spread between half the nominal length and it (odd ones among them)."""
    n = case["n"]
    return [n - (7919 * i % (n // 2) if case["ragged"] else 0) for i in range(case["n_blk"])]


def _inputs(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    s = dict(case)
    op = case["op"]
    if op in ("p", "pt"):
        s["pix"], s["w"] = _scan(case, g)
        m = case["n_det"] * case["n_samp"]
        if op == "pt":
            s["tod"] = torch.randn(m, dtype=torch.float64, device=DEV, generator=g)
        else:
            npix = torch.unique(s["pix"][0::3].clamp(min=-1)).numel() - (1 if int(s["pix"].min()) < 0 else 0)
            s["x"] = (torch.randn((npix, 3), dtype=torch.float64, device=DEV, generator=g)
                      * torch.tensor([100.0, 1.0, 1.0], dtype=torch.float64, device=DEV)).reshape(-1)
        return s
    if op in ("ninv", "psd"):
        s["blocks"] = _blocks(case)
        fk = (0.1 * 50 ** torch.rand(len(s["blocks"]), generator=g, device=DEV, dtype=torch.float64)).tolist()
        s["tod"] = torch.cat([_noise(n, f, g) for n, f in zip(s["blocks"], fk)])
        if op == "ninv":
            s["rows"] = torch.stack([_row(n, case["lam"], f) for n, f in zip(s["blocks"], fk)])
            if case["fp32"]:
                s["tod"] = s["tod"].float()
        return s
    # the solves: every detector is one stationary interval with its own knee frequency (0.5 to 2 Hz)
    s["pix"], s["w"] = _scan(case, g)
    n_det, n = case["n_det"], case["n_samp"]
    fk = (0.5 * 4 ** torch.rand(n_det, generator=g, device=DEV, dtype=torch.float64)).tolist()
    w, h = _grid(case["side"])
    sky = torch.randn((w * h, 3), dtype=torch.float64, device=DEV, generator=g)
    sky[:, 0] *= 100
    p = (s["pix"][0::3] // 3).clamp(min=0).long()  # a flagged sample's signal is not used as such
    s["signal"] = (s["w"].view(-1, 3) * sky[p]).sum(1)
    cols = case.get("cols", 1)
    noise = torch.stack([torch.cat([_noise(n, f, g) for f in fk]) for _ in range(cols)])
    s["noise"] = noise.float() if op == "multi" else noise[0]
    s["blocks"] = [n] * n_det
    s["rows"] = torch.stack([_row(n, case["lam"], f) for f in fk])
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    ctx = s["ctx"] = _context()
    if case["op"] != "psd" and "rows" in s:
        s["rows"] = s["rows"].cpu().numpy()
    if case["op"] in ("p", "pt", "solve", "multi"):
        s["P"] = mb.Pointing(ctx, s["pix"], s["w"], s["w"].numel() // 3)
    if case["op"] in ("ninv", "solve", "multi"):
        s["N"] = mb.Noise(ctx, s["blocks"], case["lam"], s["rows"].reshape(-1))
    if case["op"] == "p":
        s["out"] = torch.empty(s["w"].numel() // 3, dtype=torch.float64, device=DEV)
    elif case["op"] == "pt":
        s["out"] = torch.empty(s["P"].shape()["n_map"], dtype=torch.float64, device=DEV)
    elif case["op"] == "ninv":
        s["out"] = torch.empty_like(s["tod"])
    return s


# --------------------------------------------------------------------------- one pass
def run(s):
    op = s["op"]
    if op == "p":
        s["P"].matvec(s["x"], s["out"])
        return s["out"]
    if op == "pt":
        s["P"].trmatvec(s["tod"], s["out"])
        return s["out"]
    if op == "ninv":
        (s["N"].apply_fp32 if s["fp32"] else s["N"].apply)(s["tod"], s["out"])
        return s["out"]
    if op == "psd":
        return mb_noise.periodogram(s["tod"], s["blocks"], FS, ctx=s["ctx"])
    if op == "solve":
        x, ids, cond, hits, _, _ = mb.gls_solve(s["ctx"], s["P"], s["N"], s["signal"], s["noise"], tol=s["tol"])
    elif op == "multi":
        x, ids, cond, hits, _, _ = mb.gls_solve_multi(s["ctx"], s["P"], s["N"], s["noise"], signal=s["signal"],
                                                      signal_col=0, tol=s["tol"])
    else:
        P = mb.Pointing(s["ctx"], s["pix"], s["w"], s["w"].numel() // 3)
        N = mb.Noise(s["ctx"], s["blocks"], s["lam"], s["rows"].reshape(-1))
        x, ids, cond, hits, _, _ = mb.gls_solve_mixed(s["ctx"], P, N, s["signal"], s["noise"], tol=s["tol"])
        P.close()
        N.close()
    return dict(x=x, ids=ids, cond=cond, hits=hits)


# --------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    op = case["op"]
    if op == "psd":
        n = case["n_blk"] * case["n"] * (0.75 if case["ragged"] else 1)
        return {"bytes": 12 * n, "flops": n * (2.5 * math.log2(case["n"]) + 12)}
    if op == "ninv":
        n = case["n_blk"] * case["n"] * (0.75 if case["ragged"] else 1)
        return {"bytes": (8 if case["fp32"] else 16) * n, "flops": n * 6.7 * math.log2(8 * case["lam"])}
    m = case["n_det"] * case["n_samp"]
    w, h = _grid(case["side"])
    n_map = 3 * min(w * h, m)
    if op in ("p", "pt"):  # index, three weights and the stream, a sample; the map
        return {"bytes": 36 * m + 8 * n_map, "flops": 6 * m}
    # an operator application a PCG iteration (P, N^-1, P^T), some 40 iterations; half the bytes in FP32
    it = 40 * case.get("cols", 1)
    size = 8 if op == "solve" else 4
    return {"bytes": it * (m * (8 + 10 * size) + 11 * 8 * n_map), "flops": it * m * (12 + 6.7 * math.log2(8 * case["lam"]))}


# --------------------------------------------------------------------------- the same in 64 bits
def _weight(rows, blocks, v):
    """Block by block: less its mean, times the banded symmetric Toeplitz matrix of its row."""
    out, at = torch.empty_like(v), 0
    for row, n in zip(rows, blocks):
        b = v[at:at + n]
        b = b - b.mean()
        m = 1 << (n + row.numel() - 1).bit_length()
        c = torch.zeros(m, dtype=torch.float64, device=v.device)
        c[:row.numel()] = row
        c[m - row.numel() + 1:] = row[1:].flip(0)
        out[at:at + n] = torch.fft.irfft(torch.fft.rfft(b, n=m) * torch.fft.rfft(c).real, n=m)[:n]
        at += n
    return out


def exact(case, seed):
    s = _inputs(case, seed)
    op = case["op"]
    if op == "ninv":
        return _weight(s["rows"], s["blocks"], s["tod"].double())
    if op == "psd":
        out, at = [], 0
        for n in s["blocks"]:
            t = torch.arange(n, dtype=torch.float64, device=DEV)
            x, c = s["tod"][at:at + n], t - (n - 1) / 2
            x = x - x.mean() - c * ((c * x).sum() / (c * c).sum())
            win = 0.5 - 0.5 * torch.cos(2 * math.pi * t / n)
            p = torch.fft.rfft(x * win).abs().square() / (FS * win.square().sum())
            p[1:(n + 1) // 2] *= 2  # all but the zero and (n even) the Nyquist frequency
            out.append(p)
            at += n
        return torch.cat(out)
    seen, local = torch.unique(s["pix"][0::3].clamp(min=-3) // 3, return_inverse=True)
    gap = int(seen[0] < 0)
    npix, valid, local = seen.numel() - gap, local >= gap, (local - gap).clamp(min=0)
    w = s["w"].view(-1, 3) * valid[:, None]
    if op == "p":
        return (w * s["x"].view(-1, 3)[local]).sum(1)

    def adjoint(y):
        return torch.zeros((npix, 3), dtype=torch.float64, device=DEV).index_add_(0, local, w * y[:, None])

    if op == "pt":
        return adjoint(s["tod"]).reshape(-1)
    # the solution of (P^T N^-1 P) x = P^T N^-1 d, by block-Jacobi CG to rounding
    t0 = torch.repeat_interleave(s["rows"][:, 0].cpu(), torch.tensor(s["blocks"])).to(DEV)
    W = torch.zeros((npix, 9), dtype=torch.float64, device=DEV)
    W.index_add_(0, local, (w[:, :, None] * w[:, None, :]).view(-1, 9) * t0[:, None])
    inv, info = torch.linalg.inv_ex(W.view(-1, 3, 3))
    rcond = 1 / (inv.abs().sum(1).amax(1) * W.view(-1, 3, 3).abs().sum(1).amax(1))
    if int(info.max()) or float(rcond.min()) < 0.11:
        return None  # near the solver's cut of badly seen pixels

    def solve(d):
        r = adjoint(_weight(s["rows"], s["blocks"], d))
        x, first, rz, h = torch.zeros_like(r), r.square().sum(), None, None
        for _ in range(400):
            z = (inv @ r[:, :, None])[:, :, 0]
            new = (r * z).sum()
            h = z if h is None else z + (new / rz) * h
            q = adjoint(_weight(s["rows"], s["blocks"], (w * h[local]).sum(1)))
            a = new / (h * q).sum()
            x, r, rz = x + a * h, r - a * q, new
            if r.square().sum() <= 1e-28 * first:
                break
        return x.reshape(-1)

    if op == "multi":
        x = torch.stack([solve(v.double() + (s["signal"] if k == 0 else 0)) for k, v in enumerate(s["noise"])])
    else:
        x = solve(s["signal"] + s["noise"])
    return dict(x=x, ids=None, cond=None, hits=None)
