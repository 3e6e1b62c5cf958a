"""The MAF-aware bias inversion at the smallest sketches, where d - 3 - 2 kappa
of a pair lies on either side of 4 (kappa reaches 1 for a singleton), against
the oracle.

The oracle adds N f32 terms per dot product (N 2^-24 relative, twice that on the
square), and r^2 moves by up to four times as much per pair: 1.6e-4 at N = 300,
1e-2 over 60 pairs.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [8, 9, 10, 11, 12, 40])
@pytest.mark.parametrize("maf_aware", [False, True])
def test_small_sketch_correction(ctx, d, maf_aware):
    from ldsc_b200.api import WindowMode, run_l2
    from oracle import OracleL2Args, oracle_l2
    from test_gpu_l2 import table
    n, m = 300, 60
    rng = np.random.default_rng(d)
    codes = rng.choice(np.array([3, 2, 0, 1], np.uint8), p=[0.5, 0.35, 0.13, 0.02], size=(m, n))
    codes[::7] = 3                                  # singletons: one heterozygote
    for j in range(0, m, 7):
        codes[j, rng.integers(n)] = 2
    body = (codes.reshape(m, n // 4, 4) << np.array([0, 2, 4, 6], np.uint8)).sum(2).astype(np.uint8).reshape(-1)
    chr_, cm, bp = np.ones(m, np.uint8), np.arange(m) * 0.001, np.arange(1, m + 1) * 1000
    ref, _, _, _ = oracle_l2(OracleL2Args(bed_body=body, n_file_indiv=n, chr=chr_, cm=cm, bp=bp, chunk_c=50,
                                          sketch_d=d, sketch_maf_aware=maf_aware, use_f32=True))
    panel = ctx.upload(body, n)
    l2, _, _ = run_l2(ctx, table(chr_, cm, bp), panel, WindowMode.Cm(1.0), 50, sketch=d,
                      sketch_maf_aware=maf_aware, yes_really=True)
    np.testing.assert_allclose(l2, ref, rtol=0, atol=1e-2)
