"""The bit-sliced pair test where its tiling can go wrong: word counts around
its units of 64 columns, tiles of 1024 and bands of 256 rows, and every length
with every threshold class (levels editDist <= 5, deltas above, thresholds of
the length or more).  Integer work: bit-exact comparisons with the oracle."""
import numpy as np
import pytest

from test_gpu_modes import planted

pytestmark = pytest.mark.gpu


def _check(ctx, oracle, w, L, d):
    from indexgen_b200 import build_conflict_graph, count_conflicts

    rp, cols = oracle.conflict_upper(w, L, d)
    with build_conflict_graph(w, L, d, ctx) as G:
        r, c = G.upper_csr()
    assert np.array_equal(r, rp) and np.array_equal(c, cols), (len(w), L, d)
    assert count_conflicts(w, L, d, ctx) == int(rp[-1]), (len(w), L, d)


@pytest.mark.parametrize("n", [2, 31, 33, 63, 64, 65, 127, 129, 255, 256, 257, 319, 1023, 1024, 1025, 1088, 1281])
def test_word_counts_around_tiles(igctx, oracle, n):
    for L, d in ((12, 4), (16, 5), (11, 3), (13, 7)):
        _check(igctx, oracle, planted(n, L, 7000 + n), L, d)


@pytest.mark.parametrize("L", [3, 5, 6, 9, 11, 14, 16])
def test_every_threshold_class(igctx, oracle, L):
    w = planted(300, L, 7100 + L)
    for d in range(1, L + 3):
        _check(igctx, oracle, w, L, d)


def test_dense_words_fill_slot_chunks(igctx, oracle):
    """Nearly every pair a hit: a warp's hits of one unit exceed a slot chunk."""
    w = planted(700, 8, 7200)
    for d in (7, 8, 9):
        _check(igctx, oracle, w, 8, d)
    _check(igctx, oracle, np.repeat(planted(40, 12, 7201), 20), 12, 4)
