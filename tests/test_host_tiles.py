"""The Gram's tile list (host plan) against its definition: every in-band pair
lies in exactly one tile, whole or trimmed, for windows of every width."""
import numpy as np
import pytest


@pytest.mark.parametrize("m", [1, 31, 32, 33, 127, 128, 129, 300, 641])
@pytest.mark.parametrize("trim,max_quarters", [(0, 4), (1, 4), (1, 2), (1, 1)])
def test_every_pair_lies_in_one_tile(m, trim, max_quarters):
    from ldsc_b200 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(m)
    for width in (0, 1, 17, 130, 10 ** 6):
        # non-decreasing limits with jumps (chromosome starts), and one list that is not monotone
        left = np.maximum.accumulate(np.maximum(np.arange(m) - rng.integers(0, width + 1, m), 0))
        for lim in (left, np.maximum(np.arange(m) - rng.integers(0, width + 1, m), 0)):
            lim = np.ascontiguousarray(lim, dtype=np.int64)
            out = np.zeros((4 * (m // 128 + 1) ** 2 + 4, 4), dtype=np.uint32)
            n = lib.ldsc_debug_gram_tiles(lim.ctypes.data, m, trim, max_quarters, out.ctypes.data, len(out))
            assert 0 <= n <= len(out)
            seen = np.zeros((m + 128, m + 128), dtype=np.int32)
            for a, b, q0, nq in out[:n]:
                assert q0 + nq <= 4 and nq <= max_quarters
                seen[128 * a:128 * a + 128, 128 * b + 32 * q0:128 * b + 32 * (q0 + nq)] += 1
            for j in range(m):
                assert (seen[lim[j]:j, j] == 1).all()
            assert seen.max(initial=0) <= 1
