"""The allocation-free entry point on bands with few pairs: most records have an
empty window, so the tile list is much shorter than the records' blocks."""
import ctypes as C

import numpy as np
import pytest

from ldsc_b200.plink import BimTable

pytestmark = pytest.mark.gpu

TOL = 1e-9   # as in the other exact-mode parity tests


@pytest.mark.parametrize("m", [4224, 4353, 13000])
@pytest.mark.parametrize("kind", ["no_pair", "dense_head", "pairs"])
def test_sparse_bands_match_the_resident_entry_point(ctx, kind, m):
    import torch
    from ldsc_b200.api import WindowMode, left_limits, run_l2
    n = 70
    rng = np.random.default_rng(m)
    body = rng.integers(0, 256, (m, (n + 3) // 4), dtype=np.uint8)
    cm = 10.0 * np.arange(m)                       # every record alone in a 1 cM window
    if kind == "dense_head":
        cm[:128] = 0.001 * np.arange(128)
    elif kind == "pairs":
        cm[1::50] = cm[0::50][: len(cm[1::50])] + 0.5
    chr_, bp = np.ones(m, np.uint8), np.arange(m, dtype=np.uint32)
    snps = BimTable(chr_, [f"rs{i}" for i in range(m)], cm, bp, np.arange(m, dtype=np.int64))
    panel = ctx.upload(body, n)
    ref, ref_maf, _ = run_l2(ctx, snps, panel, WindowMode.Cm(1.0), 50, snp_level_masking=True, precision="fp64",
                             yes_really=True)
    panel.close()
    left = np.ascontiguousarray(left_limits(snps, WindowMode.Cm(1.0), 50, snp_level_masking=True), dtype=np.int64)
    rows = np.zeros((m, 32), dtype=np.uint8)
    rows[:, : body.shape[1]] = body
    d_rows = torch.from_numpy(rows).cuda()
    l2 = torch.full((m,), np.nan, dtype=torch.float64, device="cuda")
    maf = torch.full((m,), np.nan, dtype=torch.float64, device="cuda")
    rc = ctx.lib.ldsc_l2_int8_noalloc(C.c_void_p(d_rows.data_ptr()), 32, n, m, left.ctypes.data,
                                      C.c_void_p(l2.data_ptr()), C.c_void_p(maf.data_ptr()),
                                      C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    got = l2.cpu().numpy()
    assert np.max(np.abs(got - ref[:, 0]) / np.maximum(np.abs(ref[:, 0]), 1.0)) < TOL
    np.testing.assert_allclose(maf.cpu().numpy(), ref_maf, atol=1e-15)
