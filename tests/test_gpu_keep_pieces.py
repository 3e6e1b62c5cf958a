"""--keep on panels whose compacted rows go through the bounded buffer in several
pieces: the records at the pieces' edges against calls on those records alone,
and the INT8 form against the FP64 one, which keeps all compacted rows."""
import numpy as np
import pytest

from ldsc_b200.plink import BimTable

pytestmark = pytest.mark.gpu

EXACT_TOL = 1e-9   # exact integers into f64 (int8), f64 sums of a few dozen terms (fp64)
BUFFER = 64 << 20


def _case(m, n, n_keep, seed):
    rng = np.random.default_rng(seed)
    body = rng.integers(0, 256, (m, (n + 3) // 4), dtype=np.uint8)
    keep = np.sort(rng.permutation(n)[:n_keep]).astype(np.int64)
    snps = BimTable(np.ones(m, np.uint8), [f"rs{i}" for i in range(m)], 0.01 * np.arange(m),
                    np.arange(m, dtype=np.uint32), np.arange(m, dtype=np.int64))
    return body, keep, snps


def _subset(snps, rows):
    return BimTable(snps.chr[rows], [f"rs{i}" for i in rows], snps.cm[rows], snps.bp[rows], rows.astype(np.int64))


@pytest.mark.parametrize("extract", [False, True])
def test_statistics_over_pieces(ctx, extract):
    from ldsc_b200.api import snp_stats
    m, n, n_keep = 50_001, 12_003, 11_111
    body, keep, snps = _case(m, n, n_keep, 1)
    rows = np.arange(m) if not extract else np.delete(np.arange(m), [7, 20_000])
    piece = BUFFER // ((n_keep + 63) // 64 * 16)
    assert 2 * piece < m
    panel = ctx.upload(body, n)
    maf, ok = snp_stats(ctx, _subset(snps, rows), panel, keep)
    at = np.unique(np.clip(np.concatenate([[0, 1], [k * piece + o for k in (1, 2) for o in (-1, 0, 1)], [len(rows) - 1]]),
                           0, len(rows) - 1))
    one_maf, one_ok = snp_stats(ctx, _subset(snps, rows[at]), panel, keep)
    panel.close()
    np.testing.assert_array_equal(maf[at], one_maf)
    np.testing.assert_array_equal(ok[at], one_ok)
    assert len(np.unique(maf)) > m // 100   # (no piece repeated)


@pytest.mark.parametrize("annot", [False, True])
@pytest.mark.parametrize("m,n,n_keep", [(9_001, 33_003, 30_001), (40_003, 12_003, 11_111)])   # plain; overlapped with the Gram
def test_int8_over_pieces_matches_fp64(ctx, m, n, n_keep, annot):
    from ldsc_b200.api import WindowMode, run_l2
    body, keep, snps = _case(m, n, n_keep, m)
    assert m * ((n_keep + 63) // 64 * 16) > BUFFER
    A = np.random.default_rng(2).normal(size=(m, 2)) if annot else None
    panel = ctx.upload(body, n)
    got = {}
    for precision in ("int8", "fp64"):
        l2, maf, _ = run_l2(ctx, snps, panel, WindowMode.Snp(20), 50, iid_indices=keep, precision=precision, annot=A,
                            snp_level_masking=True, yes_really=True)
        got[precision] = l2, maf
    panel.close()
    np.testing.assert_array_equal(got["int8"][1], got["fp64"][1])
    ref = got["fp64"][0]
    assert np.max(np.abs(got["int8"][0] - ref) / np.maximum(np.abs(ref), 1.0)) < EXACT_TOL


def test_streamed_file_over_pieces(ctx):
    from ldsc_b200.api import WindowMode, l2_from_bed_bytes, run_l2
    m, n, n_keep = 20_003, 20_011, 19_007
    body, keep, snps = _case(m, n, n_keep, 5)
    image = np.concatenate([np.array([0x6C, 0x1B, 0x01], np.uint8), body.reshape(-1)])
    panel = ctx.upload(body, n)
    want, want_maf, _ = run_l2(ctx, snps, panel, WindowMode.Snp(20), 50, iid_indices=keep, precision="int8",
                               snp_level_masking=True, yes_really=True)
    panel.close()
    got, maf, _ = l2_from_bed_bytes(ctx, image, n, snps, WindowMode.Snp(20), 50, iid_indices=keep, precision="int8",
                                    snp_level_masking=True, yes_really=True)
    np.testing.assert_array_equal(got, want)
    np.testing.assert_array_equal(maf, want_maf)
