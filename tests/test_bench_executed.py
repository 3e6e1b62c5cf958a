"""The sketch Gram's executed pairs, as the bench counts them: 32 right records a
quarter where tiles are cut, whole tiles for long rows."""
import numpy as np
import pytest


@pytest.mark.parametrize("d,trimmed", [(200, True), (3168, True), (3169, False), (5000, False)])
def test_executed_pairs(d, trimmed):
    import bench
    m = 2000
    left = np.maximum(np.arange(m) - 133, 0)
    tiles, pairs = bench.sketch_gram_executed(left, d)
    want_tiles = want = 0
    for b in range(0, m, 128):
        for a in range(0, b + 128, 128):
            hit = [q for q in range(4) if any(max(left[j], a) <= min(j - 1, a + 127)
                                              for j in range(b + 32 * q, min(b + 32 * q + 32, m)))]
            if hit:
                want_tiles += 1
                want += 128 * 32 * (hit[-1] - hit[0] + 1 if trimmed else 4)
    assert (tiles, pairs) == (want_tiles, want)
    assert pairs < tiles * 128 * 128 if trimmed else pairs == tiles * 128 * 128
