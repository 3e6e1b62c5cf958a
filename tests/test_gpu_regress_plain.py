"""The batched regressions' plain sums (scalar sample sizes) at the edges of a
warp's steps, one job and many jobs per warp, and the median's two-sweep select
and its fallbacks."""
import numpy as np
import pytest

from oracle import regress_oracle as R

pytestmark = pytest.mark.gpu

# estimates and errors: blocks summed in another order, 2 x 2 normal equations
# for the reference's QR, a reciprocal rounded once more: a relative 1e-8
RTOL = 1e-8


def _inputs(m, T, seed):
    rng = np.random.default_rng(seed)
    ld = 1.0 + rng.gamma(2.0, 20.0, m)
    wld = np.maximum(ld * rng.uniform(0.5, 1.2, m), 0.3)
    n = np.exp(rng.uniform(np.log(2e4), np.log(4e5), T))
    z = np.sqrt(n[:, None] * 0.3 * ld / 1e6) * rng.standard_normal((T, m)) + rng.standard_normal((T, m))
    return rng, ld, wld, n, z


# SNPs per block: 3, 31, 32, 33, 63, 64, 65, 255..257 (the ring holds 4 steps of 64)
@pytest.mark.parametrize("per_block,nb,T", [(3, 20, 1), (31, 10, 2), (32, 10, 3), (33, 10, 1), (63, 8, 2), (64, 8, 5),
                                            (65, 8, 1), (257, 4, 3), (64, 160, 33), (37, 200, 26)])
def test_h2_and_rg_at_block_edges(ctx, per_block, nb, T):
    from ldsc_b200.api import h2_batch, rg_batch
    m = per_block * nb + (nb // 3 if per_block > 3 else 0)   # uneven blocks
    rng, ld, wld, n, z = _inputs(m, T, per_block)
    got = h2_batch(ctx, z * z, n, ld, wld, 1e6, nb)
    for t in {0, T // 2, T - 1}:
        want = R.run_h2(z[t] ** 2, ld, wld, n[t], 1e6, nb)
        for k in ("h2", "h2_se", "intercept", "intercept_se", "mean_chi2"):
            assert abs(got[t][k] - want[k]) <= RTOL * abs(want[k]) + 1e-12, (k, t)
        assert got[t]["lambda_gc"] == want["lambda_gc"]
    z2 = 0.5 * z + rng.standard_normal(z.shape)
    rg = rg_batch(ctx, z, z2, n, n * 1.5, ld, wld, 1e6, nb)
    for t in {0, T - 1}:
        want = R.run_rg(z[t], z2[t], ld, wld, n[t], 1.5 * n[t], 1e6, nb)
        for k in ("gencov", "gencov_se", "h2_1", "h2_2"):
            w = want[k] if isinstance(want, dict) else getattr(want, k)
            assert abs(rg[t][k] - w) <= RTOL * abs(w) + 1e-12, (k, t)
    # a job's result does not depend on the jobs beside it
    one = h2_batch(ctx, z[T - 1:] ** 2, n[T - 1:], ld, wld, 1e6, nb)
    for k in one.dtype.names:
        np.testing.assert_array_equal(one[0][k], got[T - 1][k])


def test_weights_far_from_one_take_the_division(ctx):
    """An overcounting LD score of 2^1018 puts the denominators of the second
    trait's largest weights (2 t^2 of it, t from 1 to between 2.8 and 5.7) above
    2^1021, outside the range of the reciprocal's iteration and short of
    overflow.  It scales the weights alike and cancels.  (Fixed intercept: the
    free one's determinant multiplies two sums of weights and underflows.)"""
    from ldsc_b200.api import h2_batch
    m, nb = 4000, 20
    _, ld, _, _, z = _inputs(m, 2, 5)
    n, one = np.array([1e4, 2e4]), np.ones(m)
    a = h2_batch(ctx, z * z, n, ld, one * 2.0 ** 1018, 1e6, nb, intercept=1.0, lambda_gc=False)
    b = h2_batch(ctx, z * z, n, ld, one, 1e6, nb, intercept=1.0, lambda_gc=False)
    for k in ("h2", "h2_se"):
        np.testing.assert_allclose(a[k], b[k], rtol=1e-6)


def _values(kind, m, rng):
    i = np.arange(m)
    x = rng.chisquare(1, m)
    if kind == "chi2":
        return x
    if kind == "sorted":
        return np.sort(x)
    if kind == "sample_misleads":   # the evenly spaced sample sees only large values
        x[(np.arange(1024) * m) // 1024] = 1e6 + i[:1024]
        return x
    if kind == "ties":
        return np.round(x, 1)
    if kind == "two_values":
        return np.where(rng.random(m) < 0.5, 1.0, 2.0)
    if kind == "constant":
        return np.full(m, 0.25)
    if kind == "signs":
        return rng.standard_normal(m)
    if kind == "wide":
        return np.exp(rng.uniform(-300, 300, m))
    x[:: 7] = np.inf
    return x


@pytest.mark.parametrize("kind", ["chi2", "sorted", "sample_misleads", "ties", "two_values", "constant", "signs", "wide",
                                  "infinities"])
@pytest.mark.parametrize("m", [16384, 16385, 40000, 70001])
def test_lambda_gc_two_sweeps(ctx, kind, m):
    from ldsc_b200.api import h2_batch
    rng = np.random.default_rng(m)
    y = _values(kind, m, rng)
    ld = 1.0 + rng.gamma(2.0, 20.0, m)
    got = h2_batch(ctx, np.stack([y, y[::-1].copy()]), [1e5, 1e5], ld, ld, 1e6, 7)
    for t in range(2):
        assert got[t]["lambda_gc"] == np.median(y) / 0.4549


@pytest.mark.parametrize("case", ["nan_chi2", "huge_n"])
def test_a_job_beside_one_out_of_range(ctx, case):
    """A neighbour whose weights are NaN, or so small that their denominators leave
    the reciprocal's range, changes no bit of the other jobs' results.  (The
    reciprocal and the division differ by one place in 1 of 3,400 weights, and
    few of those reach a result: many jobs of few SNPs.)"""
    from ldsc_b200.api import h2_batch, rg_batch
    m, nb, T = 150, 50, 20_000
    _, ld, wld, n, z = _inputs(m, T, 11)
    want = h2_batch(ctx, z * z, n, ld, wld, 1e6, nb)
    bad = np.arange(1, T, 2)
    rest = np.arange(0, T, 2)
    chi2, n_bad = z * z, n.copy()
    if case == "nan_chi2":
        chi2[bad, 100] = np.nan
    else:
        n_bad[bad] = 1e300
    got = h2_batch(ctx, chi2, n_bad, ld, wld, 1e6, nb)
    for k in want.dtype.names:
        np.testing.assert_array_equal(got[k][rest], want[k][rest])
    # the two h2 fits of a pair lie in one warp
    z1, n1, z2, n2 = z[::2], n[::2], z[1::2], n[1::2]
    want = rg_batch(ctx, z1, z2, n1, n2, ld, wld, 1e6, nb)
    got = rg_batch(ctx, z1, z2, np.full(T // 2, np.nan if case == "nan_chi2" else 1e300), n2, ld, wld, 1e6, nb)
    for k in ("h2_2", "h2_2_se"):
        np.testing.assert_array_equal(got[k], want[k])
