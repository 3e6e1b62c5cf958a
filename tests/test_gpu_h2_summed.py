"""h2 with a median takes the aggregate pass's sums from the median's first sweep
(from 16,384 SNPs on): the same results as without a median but for the order of
those sums, and the exact median; odd sizes put every other trait off 16-byte
alignment."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [16383, 16384, 16385, 20011])
@pytest.mark.parametrize("traits,kw", [(1, {}), (5, {}), (3, {"intercept": 1.0})])
def test_h2_with_and_without_median(ctx, m, traits, kw):
    from ldsc_b200.api import h2_batch
    rng = np.random.default_rng(m + traits)
    ld = 1.0 + rng.gamma(2.0, 20.0, m)
    w = np.maximum(ld * rng.uniform(0.8, 1.2, m), 0.5)
    n = np.exp(rng.uniform(np.log(2e4), np.log(3e5), traits))
    chi2 = (1.0 + 1e-7 * n[:, None] * ld) * rng.standard_normal((traits, m)) ** 2
    a = h2_batch(ctx, chi2, n, ld, w, 1e6, 200, lambda_gc=True, **kw)
    b = h2_batch(ctx, chi2, n, ld, w, 1e6, 200, lambda_gc=False, **kw)
    for f in a.dtype.names:
        if f == "lambda_gc":
            np.testing.assert_array_equal(a[f], np.median(chi2, axis=1) / 0.4549)
        else:   # sums of m terms in another order, through two re-weightings
            np.testing.assert_allclose(a[f], b[f], rtol=1e-10, err_msg=f)
