"""The band Gram's 128 x 128 record tiles at their edges: record counts around
a tile, windows narrower and wider than one, one and several annotation
columns, in the INT8 forms (against the brute-force definition) and the
CountSketch form (against the oracle's f32 path)."""
import numpy as np
import pytest

from ldsc_b200 import synth
from ldsc_b200.plink import BimTable

pytestmark = pytest.mark.gpu

# INT8 sums are exact and every r2u is formed in f64: what differs is the f64
# rounding of up to 520 summed terms (520 x 2^-53 ~ 6e-14), squared sums no more
EXACT_TOL = 1e-9
# f32 bucket values and dot products against the oracle's f32 path at d = 50
SKETCH_TOL = 3e-5


def _panel(m, n, per_cm, seed):
    spec = synth.PanelSpec(n_indiv=n, chrom_sizes=[m - m // 3, m // 3] if m > 3 else [m],
                           chrom_cm=[(m - m // 3) / per_cm, max(m // 3, 1) / per_cm] if m > 3 else [m / per_cm],
                           founders=9, miss=0.03, seed=seed)
    chr_, cm, bp = synth.positions(spec)
    snps = BimTable(chr_, [f"rs{i}" for i in range(m)], cm, bp, np.arange(m, dtype=np.int64))
    return synth.bed_body(spec), snps


@pytest.mark.parametrize("K", [1, 3])
@pytest.mark.parametrize("m,per_cm", [(1, 10), (2, 10), (33, 60), (127, 20), (128, 300), (129, 45), (257, 90),
                                      (520, 170), (520, 2000)])
def test_int8_tiles_match_the_definition(ctx, m, per_cm, K):
    from conftest import brute_force_l2
    from ldsc_b200.api import Context, WindowMode, left_limits, run_l2
    n = 133
    body, snps = _panel(m, n, per_cm, seed=m + per_cm)
    A = None if K == 1 else np.random.default_rng(m).standard_normal((m, K))
    with Context(0, fused_operands=True) as fused:
        for c in (ctx, fused):
            panel = c.upload(body, n)
            for masking in (True, False):
                l2, maf, _ = run_l2(c, snps, panel, WindowMode.Cm(1.0), 40, annot=A, snp_level_masking=masking,
                                    precision="int8", yes_really=True)
                left = left_limits(snps, WindowMode.Cm(1.0), 40, snp_level_masking=masking)
                ref, ref_maf = brute_force_l2(body, n, snps.chr, snps.cm, snps.bp, left, annot=A)
                assert np.max(np.abs(l2 - ref) / np.maximum(np.abs(ref), 1.0)) < EXACT_TOL
                np.testing.assert_allclose(maf, ref_maf, atol=1e-15)
            panel.close()


@pytest.mark.parametrize("maf_aware", [False, True])
@pytest.mark.parametrize("m,per_cm", [(2, 10), (127, 20), (129, 45), (257, 300)])
def test_sketch_tiles_match_the_oracle(ctx, m, per_cm, maf_aware):
    from ldsc_b200.api import WindowMode, run_l2
    from oracle import OracleL2Args, oracle_l2
    n, d = 203, 50
    body, snps = _panel(m, n, per_cm, seed=m + per_cm)
    panel = ctx.upload(body, n)
    got, _, _ = run_l2(ctx, snps, panel, WindowMode.Cm(1.0), 40, sketch=d, sketch_maf_aware=maf_aware,
                       snp_level_masking=True, yes_really=True)
    ref = oracle_l2(OracleL2Args(bed_body=body, n_file_indiv=n, chr=snps.chr, cm=snps.cm, bp=snps.bp, chunk_c=40,
                                 masking=True, use_f32=True, sketch_d=d, sketch_maf_aware=maf_aware))[0]
    panel.close()
    assert np.max(np.abs(got - ref)) < SKETCH_TOL


@pytest.mark.parametrize("K", [1, 3])
@pytest.mark.parametrize("m,per_cm,n", [(1, 10, 5), (2, 10, 16), (31, 60, 17), (32, 20, 130), (33, 300, 15),
                                        (129, 45, 64), (300, 90, 133), (300, 2000, 31)])
def test_fp64_blocks_match_the_definition(ctx, m, per_cm, n, K):
    """The FP64 form's 32 x 32 blocks at their edges, words of sixteen individuals
    that end in the row, and a record list."""
    from conftest import brute_force_l2
    from ldsc_b200.api import WindowMode, left_limits, run_l2
    body, snps = _panel(m, n, per_cm, seed=m + per_cm + n)
    pick = np.arange(0, m, 2) if m > 32 else np.arange(m)
    for idx in (np.arange(m), pick):
        sub = BimTable(snps.chr[idx], [f"rs{i}" for i in idx], snps.cm[idx], snps.bp[idx], idx.astype(np.int64))
        A = None if K == 1 else np.random.default_rng(m).standard_normal((len(idx), K))
        panel = ctx.upload(body, n)
        for masking in (True, False):
            l2, _, _ = run_l2(ctx, sub, panel, WindowMode.Cm(1.0), 40, annot=A, snp_level_masking=masking,
                              precision="fp64", yes_really=True)
            left = left_limits(sub, WindowMode.Cm(1.0), 40, snp_level_masking=masking)
            ref, _ = brute_force_l2(body[idx], n, sub.chr, sub.cm, sub.bp, left, annot=A)
            assert np.max(np.abs(l2 - ref) / np.maximum(np.abs(ref), 1.0)) < EXACT_TOL
        panel.close()
