"""Edges of the partitioned kernels against the oracle: the Gram's units of
4 x 5 groups of 8 columns and their split k-steps, and the solve's register
tiles, over the column count q = annotations + free intercept + chi2.

The oracle solves with numpy's LU where the device eliminates by Gauss-Jordan,
both with partial pivoting: agreement to 1e-8, or 1e-13 times the condition
number of the estimates' covariance where that is larger.
"""
import numpy as np
import pytest

from oracle import regress_oracle as R

pytestmark = pytest.mark.gpu


def _inputs(k, seed, m=5_003):
    rng = np.random.default_rng(seed)
    base = 1.0 + rng.gamma(2.0, 15.0, m)
    l2 = base[:, None] * rng.dirichlet(np.ones(k), size=m) * rng.uniform(0.5, 1.5, (m, k))
    wld = np.maximum(base * rng.uniform(0.8, 1.2, m), 0.5)
    z2 = (1.0 + 0.02 * l2.sum(1)) * rng.standard_normal(m) ** 2
    z2[rng.random(m) < 0.1] = 1e6      # above the chi2 cut: not kept
    n = rng.uniform(5e4, 2e5, m)
    n[rng.random(m) < 0.01] = 0.0      # their LD scores carry no weight, the intercept does
    return l2, wld, z2, n


# (annotations, free intercept): q = 2, 3 | 8, 9 | 17 | 32, 33, 34 | 40, 41 | 64, 65, 66 | 113, 114 | 161, 161
EDGES = [(1, False), (1, True), (6, True), (8, False), (15, True), (31, False), (31, True), (32, True),
         (38, True), (40, False), (62, True), (63, True), (64, True), (112, False), (112, True), (159, True),
         (160, False)]


@pytest.mark.parametrize("k,free", EDGES)
def test_partitioned_column_edges(ctx, k, free):
    from ldsc_b200.partitioned import h2_partitioned
    l2, wld, chi2, n = _inputs(k, 900 + k)
    m_vec = np.full(k, 1e3)
    kw = {} if free else {"no_intercept": True}
    got = h2_partitioned(ctx, chi2, n, l2, wld, m_vec, 13, **kw)
    want = R.fit_h2_partitioned(chi2, l2, wld, n, m_vec, 13, **kw)
    assert got.n_obs == want["n_obs"] and got.n_blocks == want["n_blocks"]
    cond = np.linalg.cond(want["cov"]) if k > 1 or free else 1.0
    tol = max(1e-8, min(1e-4, 1e-13 * cond))
    for name in ("est", "delete_values"):
        w = np.asarray(want[name])
        np.testing.assert_allclose(getattr(got, name), w, rtol=tol, atol=tol * np.abs(w).max(), err_msg=name)
    assert got.h2_total == pytest.approx(want["h2_total"], rel=tol)
