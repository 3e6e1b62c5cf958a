"""Annotations that are inf, NaN or very large: a record's l2 takes them from the
pairs inside its window alone, in every Gram form.  A negative exponent of p q
makes the annotation of a monomorphic record inf."""
import numpy as np
import pytest

from ldsc_b200 import synth
from ldsc_b200.plink import BimTable

pytestmark = pytest.mark.gpu

EXACT_TOL = 1e-9   # exact integers into f64 (int8), f64 sums of a few hundred terms (fp64)

FORMS = {
    "fp64": dict(precision="fp64"),
    "int8": dict(precision="int8"),
    "int8_long_rows": dict(precision="int8"),     # 100 K steps and more: whole tiles, 8 epilogue warps
    "int8_fused": dict(precision="int8"),
    "sketch": dict(sketch=32),
    "sketch_few": dict(sketch=5),                 # the f64 form of the bias inversion
    "sketch_maf": dict(sketch=32, sketch_maf_aware=True),
}


@pytest.fixture(scope="module")
def fused_ctx():
    from ldsc_b200.api import Context
    c = Context(0, fused_operands=True)
    yield c
    c.close()


def _panel(n, mono):
    """Random genotypes (no record monomorphic by chance), windows of about 130 records to each side: some
    32 x 32 blocks lie inside the band, some across its edge."""
    spec = synth.PanelSpec(n_indiv=n, chrom_sizes=[1200, 150], chrom_cm=[12.0, 1.5], seed=n)
    chr_, cm, bp = synth.positions(spec)
    body = np.random.default_rng(n).integers(0, 256, (spec.m, (n + 3) // 4), dtype=np.uint8)
    for i, r in enumerate(mono):
        body[r] = 0x00 if i % 2 == 0 else 0x55     # all of one genotype; all missing
    snps = BimTable(chr_, [f"rs{i}" for i in range(spec.m)], cm, bp, np.arange(spec.m, dtype=np.int64))
    return body, snps


def _same(got, want, tol=EXACT_TOL):
    fin = np.isfinite(want)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[~fin & ~np.isnan(want)], want[~fin & ~np.isnan(want)])
    assert np.max(np.abs(got[fin] - want[fin]) / np.maximum(np.abs(want[fin]), 1.0)) < tol


@pytest.mark.parametrize("masking", [True, False])
@pytest.mark.parametrize("form", ["fp64", "int8", "int8_fused"])
def test_negative_pq_exponent_with_monomorphic_records(ctx, fused_ctx, form, masking):
    from conftest import brute_force_l2
    from ldsc_b200.api import WindowMode, left_limits, run_l2
    n, mono = 150, [3, 300, 310, 1300]
    body, snps = _panel(n, mono)
    c = fused_ctx if form == "int8_fused" else ctx
    panel = c.upload(body, n)
    l2, maf, _ = run_l2(c, snps, panel, WindowMode.Cm(1.3), 50, snp_level_masking=masking, pq_exp=-0.5,
                        yes_really=True, **FORMS[form])
    panel.close()
    left = left_limits(snps, WindowMode.Cm(1.3), 50, snp_level_masking=masking)
    with np.errstate(divide="ignore"):
        pq = (maf * (1 - maf)) ** -0.5
    assert np.isinf(pq[mono]).all() and np.isfinite(np.delete(pq, mono)).all()
    with np.errstate(invalid="ignore"):
        want, _ = brute_force_l2(body, n, snps.chr, snps.cm, snps.bp, left, pq=pq)
    assert np.isfinite(want).sum() > 100 and np.isinf(want).sum() > 50
    _same(l2[:, 0], want[:, 0])


@pytest.mark.parametrize("masking", [True, False])
@pytest.mark.parametrize("form", list(FORMS))
def test_annotation_values_reach_the_window_only(ctx, fused_ctx, form, masking):
    """l2 is linear in the annotation: the run without the special values plus, for
    each of them, its record's r^2 (a run with that record's annotation alone)
    times the value, over the pairs in the band."""
    from ldsc_b200.api import WindowMode, left_limits, run_l2
    n = 13_000 if form == "int8_long_rows" else 333
    body, snps = _panel(n, [310])
    m = len(snps.chr)
    c = fused_ctx if form == "int8_fused" else ctx
    panel = c.upload(body, n)

    def l2_of(a):
        out, _, _ = run_l2(c, snps, panel, WindowMode.Cm(1.3), 50, snp_level_masking=masking, annot=a[:, None],
                           yes_really=True, **FORMS[form])
        return out[:, 0]

    left = left_limits(snps, WindowMode.Cm(1.3), 50, snp_level_masking=masking)
    special = {5: np.inf, 300: -np.inf, 310: np.nan, 700: 1e300, 705: 1e-310, 1100: np.inf, 1349: -np.inf}
    a = np.random.default_rng(7).normal(size=m)
    for r in special:
        a[r] = 0.0
    want = l2_of(a)
    k, j = np.arange(m)[:, None], np.arange(m)[None, :]
    band = (k < j) & (left[None, :] <= k)
    band |= band.T
    for r, v in special.items():
        one = np.zeros(m)
        one[r] = 1.0
        r2u = l2_of(one)
        with np.errstate(invalid="ignore"):
            want = want + np.where(band[r], r2u * v, 0.0)
        want[r] += v
        a[r] = v
    got = l2_of(a)
    panel.close()
    assert np.isfinite(want).sum() > 300
    _same(got, want)


@pytest.mark.parametrize("masking", [True, False])
@pytest.mark.parametrize("k_annot", [2, 20, 131])     # fragments of one and two, and a second chunk of columns
@pytest.mark.parametrize("form", ["fp64", "int8", "int8_fused", "sketch"])
def test_columns_with_special_values(ctx, fused_ctx, form, k_annot, masking):
    """Several columns: each with its own special values equals the run on that
    column alone, and the columns without any are what they are without them."""
    from ldsc_b200.api import WindowMode, run_l2
    n = 333
    body, snps = _panel(n, [310])
    m = len(snps.chr)
    c = fused_ctx if form == "int8_fused" else ctx
    panel = c.upload(body, n)

    def l2_of(A, **kw):
        out, _, _ = run_l2(c, snps, panel, WindowMode.Cm(1.3), 50, snp_level_masking=masking, annot=A,
                           yes_really=True, **kw, **FORMS[form])
        return out

    rng = np.random.default_rng(k_annot)
    A = rng.normal(size=(m, k_annot))
    plain = l2_of(A)
    B = A.copy()
    B[5, 0], B[300, 0], B[310, 0] = np.inf, -np.inf, np.nan
    B[1349, k_annot - 1] = -np.inf
    got = l2_of(B)
    mixed = sorted({0, k_annot - 1})
    for col in mixed:
        _same(got[:, col], l2_of(B[:, col:col + 1])[:, 0])
        assert 300 < np.isfinite(got[:, col]).sum() < m
    rest = [x for x in range(k_annot) if x not in mixed]
    assert np.array_equal(got[:, rest], plain[:, rest])
    if form != "sketch":   # negative exponent: every column of the monomorphic record is inf
        pq = l2_of(A, pq_exp=-0.5)
        for col in mixed:
            _same(pq[:, col], l2_of(A[:, col:col + 1], pq_exp=-0.5)[:, 0])
    panel.close()
