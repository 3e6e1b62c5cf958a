"""--keep: rows compacted to the kept individuals before the decode, against the
brute-force definition: words that end inside the list, lists in any order with
repeats, record lists, and rows too long to be staged."""
import numpy as np
import pytest

from ldsc_b200 import synth
from ldsc_b200.plink import BimTable

pytestmark = pytest.mark.gpu

EXACT_TOL = 1e-9   # exact integers into f64 (int8), f64 sums of a few hundred terms (fp64)


def _keep(kind, n, rng):
    if kind == "sorted":
        return np.sort(rng.permutation(n)[: max(3, 2 * n // 3)])
    if kind == "shuffled_repeats":
        return rng.integers(0, n, n + 5)
    return np.arange(n)[: n // 16 * 16 + 1]   # one individual into the last word


@pytest.mark.parametrize("precision", ["int8", "fp64"])
@pytest.mark.parametrize("extract", [False, True])
@pytest.mark.parametrize("kind", ["sorted", "shuffled_repeats", "word_edge"])
@pytest.mark.parametrize("n", [37, 133, 1026])
def test_keep_matches_the_definition(ctx, n, kind, extract, precision):
    from conftest import brute_force_l2
    from ldsc_b200.api import WindowMode, left_limits, run_l2, snp_stats
    spec = synth.PanelSpec(n_indiv=n, chrom_sizes=[150, 70], chrom_cm=[2.0, 1.0], founders=7, miss=0.05, seed=n)
    body, (chr_, cm, bp) = synth.bed_body(spec), synth.positions(spec)
    rng = np.random.default_rng(n)
    keep = _keep(kind, n, rng).astype(np.int64)
    idx = np.sort(rng.permutation(spec.m)[:140]) if extract else np.arange(spec.m)
    snps = BimTable(chr_[idx], [f"rs{i}" for i in idx], cm[idx], bp[idx], idx.astype(np.int64))
    panel = ctx.upload(body, n)
    l2, maf, _ = run_l2(ctx, snps, panel, WindowMode.Cm(1.0), 50, iid_indices=keep, precision=precision,
                        yes_really=True)
    left = left_limits(snps, WindowMode.Cm(1.0), 50)
    ref, ref_maf = brute_force_l2(body[idx], n, snps.chr, snps.cm, snps.bp, left, iid=keep)
    stat_maf, _ = snp_stats(ctx, snps, panel, keep)
    panel.close()
    assert np.max(np.abs(l2 - ref) / np.maximum(np.abs(ref), 1.0)) < EXACT_TOL
    np.testing.assert_allclose(maf, ref_maf, atol=1e-15)
    np.testing.assert_allclose(stat_maf, ref_maf, atol=1e-15)


@pytest.mark.parametrize("n", [196_600, 196_700, 260_003])   # two rows of 49,152 bytes fit; longer ones do not
def test_keep_on_long_rows(ctx, n):
    from ldsc_b200.api import snp_stats
    from ldsc_b200.plink import decode_genotypes
    rng = np.random.default_rng(n)
    body = rng.integers(0, 256, (5, (n + 3) // 4), dtype=np.uint8)
    keep = np.sort(rng.permutation(n)[: n // 2]).astype(np.int64)
    snps = BimTable(np.ones(5, np.uint8), [f"rs{i}" for i in range(5)], np.arange(5.0), np.arange(5, dtype=np.uint32),
                    np.arange(5, dtype=np.int64))
    panel = ctx.upload(body, n)
    maf, ok = snp_stats(ctx, snps, panel, keep)
    panel.close()
    G = decode_genotypes(body, n)[:, keep]
    f = np.nansum(G, 1) / (2.0 * np.sum(~np.isnan(G), 1))
    np.testing.assert_allclose(maf, np.minimum(f, 1 - f), atol=1e-15)
    assert np.array_equal(ok, np.sum(np.isnan(G) | (G == 1), 1) < len(keep))
