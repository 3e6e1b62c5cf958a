"""The Gram's tile list holds no tile without an in-band pair, and whole tiles
are never more than the 64 x 128 band tiles that the allocation-free entry point
reserves room for."""
import ctypes as C

import numpy as np
import pytest


def _tiles(left, trim, max_quarters):
    from ldsc_b200 import _lib
    lib = _lib.load()
    left = np.ascontiguousarray(left, dtype=np.int64)
    n = lib.ldsc_debug_gram_tiles(left.ctypes.data, len(left), trim, max_quarters, None, 0)
    out = np.zeros((n, 4), dtype=np.uint32)
    assert lib.ldsc_debug_gram_tiles(left.ctypes.data, len(left), trim, max_quarters,
                                     out.ctypes.data_as(C.c_void_p), n) == n
    return out.astype(np.int64)


def _pairs_in(left, k0, k1, j0, j1):
    """In-band pairs left[j] <= k < j with k in [k0, k1), j in [j0, j1)."""
    j = np.arange(j0, min(j1, len(left)))
    return int(np.maximum(0, np.minimum(j, k1) - np.maximum(left[j0:j1], k0)).sum())


def _lefts(kind, m):
    rng = np.random.default_rng(m)
    j = np.arange(m)
    if kind == "no_pair":
        return j
    if kind == "dense_head":          # one full block, then records alone
        return np.where(j < 128, 0, j)
    if kind == "few":                 # a partner here and there
        return np.maximum.accumulate(j - (rng.random(m) < 0.01))
    return np.maximum.accumulate(np.maximum(j - rng.geometric(0.6, m) + 1, 0))


@pytest.mark.parametrize("kind", ["no_pair", "dense_head", "few", "short_gaps"])
@pytest.mark.parametrize("m", [1, 33, 129, 4224, 13000])
def test_every_tile_holds_a_pair(kind, m):
    left = _lefts(kind, m)
    for trim, mq in ((0, 4), (1, 4), (1, 2), (1, 1)):
        for a, b, q0, nq in _tiles(left, trim, mq):
            j0 = 128 * b + 32 * q0
            if trim:   # the outer quarters of a trimmed tile, or the whole piece
                assert _pairs_in(left, 128 * a, 128 * a + 128, 128 * b, 128 * b + 128) > 0
                if mq == 4:
                    assert _pairs_in(left, 128 * a, 128 * a + 128, j0, j0 + 32) > 0
                    assert _pairs_in(left, 128 * a, 128 * a + 128, j0 + 32 * (nq - 1), j0 + 32 * nq) > 0
            else:
                assert _pairs_in(left, 128 * a, 128 * a + 128, j0, j0 + 128) > 0


@pytest.mark.parametrize("kind", ["no_pair", "dense_head", "few", "short_gaps"])
@pytest.mark.parametrize("m", [129, 4224, 4225, 13000])
def test_no_more_tiles_than_band_tiles(kind, m):
    left = _lefts(kind, m)
    band = sum(_pairs_in(left, a, a + 64, b, b + 128) > 0
               for b in range(0, m, 128) for a in range(int(left[b:b + 128].min()) // 64 * 64, min(b + 128, m), 64))
    for trim in (0, 1):
        assert len(_tiles(left, trim, 4)) <= band
