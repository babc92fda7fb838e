"""N^-1 of the longest block there is, 2^31 - 1 samples: the last tiles' windows reach past the
range of a 32-bit sample index.  FP32 against the three-term product in FP64 at both ends:
2.5e-6 relative (42 roundings of 2^-24, as in the right-angle tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("plan", ["r,4,12", "r,0,12"])
def test_longest_block(gpu_ctx, plan):
    import torch
    import midapack_b200 as mb
    n, k = (1 << 31) - 1, 400000
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    v = torch.randn(n, dtype=torch.float32, device="cuda", generator=g)
    out = torch.full((n,), float("nan"), dtype=torch.float32, device="cuda")
    row = np.array([2.0, -0.7, 0.4])
    N = mb.Noise(gpu_ctx, [n], 3, row).set_plan(plan, fp32=True)
    N.apply_fp32(v, out)
    torch.cuda.synchronize()
    mean = sum(float(c.double().sum()) for c in v.split(1 << 28)) / n
    for end in (v[:k], v[-k:]):
        b = end.double() - mean
        ref = row[0] * b
        for j in (1, 2):
            ref[j:] += row[j] * b[:-j]
            ref[:-j] += row[j] * b[j:]
        first = end.data_ptr() == v.data_ptr()
        got = (out[:k] if first else out[-k:]).double()
        cut = slice(0, k - 2) if first else slice(2, k)  # the cut edge lacks its neighbours
        assert torch.linalg.norm(got[cut] - ref[cut]) < 2.5e-6 * torch.linalg.norm(ref[cut])
    N.close()
    del v, out
    torch.cuda.empty_cache()
