"""A file that streams in several chunks gives the resident panel's results,
bit for bit: one chunk, one row more, a last chunk of one right block, rows that
skip whole chunks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 200_000                        # 50,000 bytes per row: 503 rows to a chunk of 24 MB


@pytest.mark.parametrize("rows,take", [(503, None), (504, None), (755, None), (1400, None), (1400, "sparse"),
                                       (1400, "tail")])
def test_streamed_file_equals_panel(ctx, rows, take):
    from ldsc_b200.api import WindowMode, l2_from_bed_bytes, run_l2
    from test_gpu_l2 import table
    rng = np.random.default_rng(rows)
    body = rng.integers(0, 256, rows * (N // 4), dtype=np.uint8)
    idx = {None: np.arange(rows), "sparse": np.arange(0, rows, 97), "tail": np.arange(rows - 40, rows)}[take]
    snps = table(np.ones(len(idx)), idx * 0.001, idx * 1000 + 1)
    snps.bed_idx = idx.astype(np.int64)
    kw = dict(precision="int8", snp_level_masking=True, yes_really=True)
    image = np.concatenate([np.array([0x6C, 0x1B, 0x01], np.uint8), body])
    l2, maf, _ = l2_from_bed_bytes(ctx, image, N, snps, WindowMode.Cm(0.2), 50, **kw)
    want, wmaf, _ = run_l2(ctx, snps, ctx.upload(body, N), WindowMode.Cm(0.2), 50, **kw)
    assert np.array_equal(l2, want)
    assert np.array_equal(maf, wmaf)
