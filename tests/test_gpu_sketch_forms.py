"""The CountSketch projection's kernel forms over the sizes where they change or
could go wrong: row lengths around whole quads and whole stretches, buckets
fewer than threads, both thread counts, stored counts per quad and per word,
rows too long for the row form, and runs around the longest it takes.

Each bucket is the f32 rounding of an exactly known number, and the row's scale
is an f32 of a norm over those: a few f32 roundings, 2^-21 relative.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = 3


def _layout(n, d, rng, run):
    """Random buckets and signs; with run, that many individuals form bucket d / 2's positive run."""
    bucket = rng.integers(0, d, n)
    sign = np.where(rng.random(n) < 0.5, np.float32(-1), np.float32(1))
    if run:
        b = d // 2
        bucket[bucket == b] = (b + 1) % d
        who = rng.permutation(n)[:run]
        bucket[who] = b
        sign[who] = 1
    return bucket.astype(np.uint32), sign


@pytest.mark.parametrize("n,d,run", [
    (3, 2, 0), (63, 5, 0), (64, 5, 0), (65, 40, 0), (8191, 200, 0), (8192, 127, 0), (8193, 129, 0), (24576, 200, 0),
    (20011, 1, 0), (20011, 1000, 0), (100003, 200, 0), (100003, 1000, 0), (50000, 2560, 0), (16384, 2561, 0),
    (16320, 12288, 0), (280000, 50, 0), (400000, 300, 0), (300000, 2600, 0),
    (60000, 200, 16383), (60000, 200, 16384), (60000, 200, 40000), (60000, 2600, 16383), (60000, 2600, 20000)])
def test_sketch_project_forms(ctx, n, d, run):
    from ldsc_b200.api import sketch_project
    from ldsc_b200.plink import decode_genotypes
    rng = np.random.default_rng(n + d + run)
    bpr = (n + 3) // 4
    body = rng.integers(0, 256, (ROWS, bpr), dtype=np.uint8)
    body[1, :bpr // 2] = 0x55   # half a row missing
    if n % 4:
        body[:, -1] &= (1 << (2 * (n % 4))) - 1
    bucket, sign = _layout(n, d, rng, run)
    panel = ctx.upload(body, n)
    got = sketch_project(ctx, panel, 0, ROWS, bucket, sign, d)
    G = decode_genotypes(body, n)
    for j in range(ROWS):
        pres = ~np.isnan(G[j])
        g = np.where(pres, G[j], 0.0)
        cnt = int(pres.sum())
        mean = g.sum() / cnt if cnt else 0.0
        sd = np.sqrt((np.sum(g * g) - cnt * mean * mean) / n)
        inv = float(np.float32(1.0 / sd)) if sd > 0 else 0.0
        s1 = np.bincount(bucket, weights=sign * g, minlength=d)
        s0 = np.bincount(bucket, weights=sign * pres, minlength=d)
        col = inv * (s1 - float(np.float32(mean)) * s0)
        nrm = np.sum(col * col)
        if nrm > 0:
            col *= np.sqrt(n / nrm)
        np.testing.assert_allclose(got[j], col, rtol=2.0 ** -21, atol=1e-9, err_msg=str(j))
