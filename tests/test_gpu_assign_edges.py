"""Nearest-centre assignment around the centre counts at which a length goes from
one word against each centre in turn to one word against 32 centres at a time.
Integer work: exact equality with the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [8, 10, 11, 12, 13, 14, 15, 16])
def test_counts_around_the_change(igctx, oracle, L):
    from indexgen_b200 import assign_centers, workloads as W

    single = np.array([c * 0x55555555 & ((1 << 2 * L) - 1) for c in range(4)], np.uint32)
    for k in range(8, 15):
        w = np.concatenate([W.uniform_words(701, L, 8200 + k), np.repeat(single, 9)])
        c = W.uniform_words(k, L, 8201 + k)
        c[k - 1] = c[0]
        assert np.array_equal(assign_centers(w, c, L, igctx), oracle.assign_centers(w, c, L)), (L, k)
        c = np.concatenate([single[:1], np.repeat(single[2:3], k - 1)])  # far from most words, ties
        assert np.array_equal(assign_centers(w, c, L, igctx), oracle.assign_centers(w, c, L)), (L, k)


@pytest.mark.parametrize("n", [(1 << 19) - 1, 1 << 19])
@pytest.mark.parametrize("L,k", [(11, 9), (13, 9), (14, 10), (15, 11), (15, 12)])
def test_word_count_of_the_change(igctx, oracle, L, k, n):
    from indexgen_b200 import assign_centers, workloads as W

    w, c = W.uniform_words(n, L, 8300 + L), W.uniform_words(k, L, 8301 + L)
    assert np.array_equal(assign_centers(w, c, L, igctx), oracle.assign_centers(w, c, L))
