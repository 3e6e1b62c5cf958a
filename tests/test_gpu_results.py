"""Results through the context's pinned memory, and those too large for it
(8 MiB), equal the device's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k", [(1, 1), (16384, 63), (16385, 63)])   # 16384 x (63 + 1) doubles = 8 MiB
def test_host_results_equal_device_results(ctx, m, k):
    import torch
    from ldsc_b200.api import WindowMode, run_l2
    from test_gpu_l2 import table
    n = 64
    rng = np.random.default_rng(m)
    body = rng.integers(0, 256, (m, n // 4), dtype=np.uint8)
    snps = table(np.ones(m), np.arange(m) * 0.01, np.arange(1, m + 1))
    annot = np.asfortranarray(rng.random((m, k)))
    panel = ctx.upload(body, n)
    kw = dict(annot=annot, yes_really=True, precision="int8", snp_level_masking=True)
    l2, maf, _ = run_l2(ctx, snps, panel, WindowMode.Cm(0.5), 50, **kw)
    dl2 = torch.empty((k, m), dtype=torch.float64, device="cuda")
    dmaf = torch.empty(m, dtype=torch.float64, device="cuda")
    run_l2(ctx, snps, panel, WindowMode.Cm(0.5), 50, out_device=(dl2, dmaf), **kw)
    assert np.array_equal(np.asarray(l2).reshape(m, k), dl2.cpu().numpy().T)
    assert np.array_equal(maf, dmaf.cpu().numpy())
