"""The annotation contraction over half blocks: output rows on either side of
64 and 128, tiles cut to quarters of one half or of both, and column chunks,
against the definition.  Sums of f64 terms: 1e-9 of the largest."""
import numpy as np
import pytest

from conftest import brute_force_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [2, 63, 65, 129, 193, 300])
@pytest.mark.parametrize("k,half", [(2, 5), (9, 40), (97, 100), (130, 70)])
def test_contraction_halves(ctx, m, k, half):
    from ldsc_b200.api import WindowMode, run_l2
    from test_gpu_l2 import table
    n = 120
    rng = np.random.default_rng(1000 * m + k)
    body = rng.integers(0, 256, (m, n // 4), dtype=np.uint8)
    cm = np.arange(m) * 1.0
    snps = table(np.ones(m), cm, np.arange(1, m + 1))
    annot = rng.standard_normal((m, k))
    panel = ctx.upload(body, n)
    left = np.maximum(np.arange(m) - half, 0)
    want, _ = brute_force_l2(body, n, np.ones(m), cm, np.arange(1, m + 1), left, annot=annot)
    for precision in ("int8", "fp64"):
        l2, _, _ = run_l2(ctx, snps, panel, WindowMode.Cm(half + 0.5), 1, annot=annot, precision=precision,
                          snp_level_masking=True, yes_really=True)
        np.testing.assert_allclose(l2, want, rtol=0, atol=1e-9 * np.abs(want).max())
