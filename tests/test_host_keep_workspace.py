"""--keep: the rows compacted for a decode go through a bounded buffer, so the
workspace that admission and slicing count on does not grow with the panel by
more than the operand rows."""
import ctypes as C

import numpy as np
import pytest

from ldsc_b200.plink import BimTable


def _workspace(m, n, keep, precision):
    from ldsc_b200 import _lib as L
    from ldsc_b200.api import WindowMode, _ArgPack
    snps = BimTable(np.ones(m, np.uint8), [""] * m, 0.001 * np.arange(m), np.arange(m, dtype=np.uint32),
                    np.arange(m, dtype=np.int64))
    pack = _ArgPack(snps, WindowMode.Cm(0.01), 200, None, keep, None, True, False, None, False, True, precision, False,
                    None)
    out = C.c_uint64()
    assert L.load().ldsc_l2_workspace_bytes(C.byref(pack.args), n, C.byref(out)) == 0
    return out.value


@pytest.mark.parametrize("m,n", [(1000, 2000), (60_000, 20_000)])
def test_kept_rows_take_a_bounded_buffer(m, n):
    keep = np.arange(n, dtype=np.int64)   # the same individuals, by list
    more = _workspace(m, n, keep, "int8") - _workspace(m, n, None, "int8")
    pitch = (n + 63) // 64 * 16
    assert 8 * n <= more <= 8 * n + min(m * pitch, 64 << 20)
    # the FP64 Gram reads them all
    more = _workspace(m, n, keep, "fp64") - _workspace(m, n, None, "fp64")
    assert more == 8 * n + m * pitch
