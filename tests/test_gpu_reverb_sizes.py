"""estimate_reverb on the GPU at histogram lengths around its block's chunks (128
threads, 8 bins a step of the late sum) and up to its longest curve, against the
oracle's FP64 estimate. The level is an f32 sum in the reference's order on both
sides: equal to f32 rounding of its square root. RT60 reads two bin indices and
an f32 quotient of FP64 levels: within 1e-6; the least-squares fit, FP64 sums in
another order, within 1e-6 too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_bins", [1, 2, 31, 127, 128, 129, 300, 2000, 4095, 19370])
@pytest.mark.parametrize("nb", [1, 3, 8])
def test_reverb_at_every_length_equals_the_oracle(ctx, oracle, n_bins, nb):
    rng = np.random.default_rng(n_bins * 10 + nb)
    t = np.arange(n_bins)[:, None]
    decay = rng.uniform(0.5, 8.0, nb)[None, :]
    bins = (rng.uniform(0.2, 1.0, (n_bins, nb)) * np.exp(-decay * t / n_bins) * 1e-3).astype(np.float32)
    bins[rng.random((n_bins, nb)) < 0.2] = 0.0
    if n_bins == 300:
        bins[:, 0] = 0.0                                   # a silent band: the defaults
    dt = 0.001 if n_bins > 300 else 0.01
    got = ctx.estimate_reverb(bins, dt)
    rt, lv, fit = oracle.estimate_reverb(bins, dt, level_f32=True)
    assert np.allclose(got.level, lv, rtol=2e-7, atol=0)
    assert np.allclose(got.rt60, rt, rtol=1e-6, atol=0)
    assert np.allclose(got.rt60_fit, fit, rtol=1e-6, atol=0)
