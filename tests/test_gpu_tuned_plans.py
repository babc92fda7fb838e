"""A tile plan that was timed for one half bandwidth is taken over for another of the same class
only where it is one of that band's own candidates: an eighth of its tile useful."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[12000] * 4, [5003], [40000] * 2])
@pytest.mark.parametrize("lams", [[513, 769, 1000, 1024], [257, 400, 512], [129, 255, 256], [1025, 2000]])
def test_plan_of_a_narrow_band_is_not_kept_for_a_wide_one(gpu_ctx, sizes, lams):
    import midapack_b200 as mb
    for lam in lams:                              # the narrowest first, as it is then timed first
        row = np.zeros(lam)
        row[0] = 1.0
        N = mb.Noise(gpu_ctx, sizes, lam, np.tile(row, len(sizes)))
        for tile in (N.tile(), N.tile_fp32()):
            n = tile["fft_n"]
            assert 8 * (n - 2 * (lam - 1)) >= n, (lam, tile)
        N.close()
