"""estimate_reverb on few and on many curves: one warp or four take a curve, by the number
of curves and of bins. A job's values do not depend on its company.

Tolerance: the FP64 sums are split differently (relative 1e-12 apart at most), so the f32
results may round to neighbours: 2^-22 relative. The late level is one f32 sum in order:
equal.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [3, 8])
@pytest.mark.parametrize("n_bins", [1, 31, 129, 767, 768, 4096, 4097])
def test_job_alone_and_in_company(ctx, nb, n_bins):
    rng = np.random.default_rng(n_bins + nb)
    # more than 384 curves, and a job fewer than each line of the rule
    for n in (152 // nb, 152 // nb + 1, 384 // nb, 384 // nb + 1):
        t = np.arange(n_bins)[None, :, None] / n_bins
        x = (rng.random((n, n_bins, nb)) * np.exp(-t * rng.uniform(0.5, 40.0, (n, 1, nb)))).astype(np.float32)
        x[0] = 0.0
        many = ctx.estimate_reverb(x, 0.005)
        for i in sorted({0, 1, n // 2, n - 1}):
            one = ctx.estimate_reverb(x[i], 0.005)
            np.testing.assert_array_equal(many[i].level, one.level)
            for a, b in ((many[i].rt60, one.rt60), (many[i].rt60_fit, one.rt60_fit)):
                np.testing.assert_allclose(a, b, rtol=2.0 ** -22, atol=0)
