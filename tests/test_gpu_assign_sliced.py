"""The bit-sliced nearest-centre kernel where it can go wrong: centre counts
around its words of 32, units of 64 and passes of 2,048, every band width it
picks, words whose nearest centre lies outside the band (the full matrix), ties
across words and units.  Integer work: exact equality with the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [8, 9, 31, 32, 33, 63, 64, 65, 96, 97, 129, 2047, 2048, 2049, 2112])
def test_centre_counts(igctx, oracle, k):
    from indexgen_b200 import assign_centers, workloads as W

    for L, n in ((7, 300), (13, 515), (16, 257)):
        w = W.uniform_words(n, L, 8000 + k)
        c = W.uniform_words(k, L, 8001 + L)
        c[k - 1] = c[0]
        c[k // 2] = c[1]
        assert np.array_equal(assign_centers(w, c, L, igctx), oracle.assign_centers(w, c, L)), (L, k)


@pytest.mark.parametrize("L", [8, 10, 12, 13, 14, 15, 16])
def test_every_band_and_far_words(igctx, oracle, L):
    """Centre counts on both sides of each band's limit, and centres far from
    some words (single-letter words), which the full matrix must settle."""
    from indexgen_b200 import assign_centers, workloads as W

    single = np.array([c * 0x55555555 & ((1 << 2 * L) - 1) for c in range(4)], np.uint32)
    for k in (9, 10, 11, 14, 16, 17, 24, 45, 88, 89, 181, 182):
        w = np.concatenate([W.uniform_words(700, L, 8100 + k), np.repeat(single, 10)])
        c = W.uniform_words(k, L, 8101 + k)
        assert np.array_equal(assign_centers(w, c, L, igctx), oracle.assign_centers(w, c, L)), (L, k)
    for k in (12, 40, 2100):  # every centre far from the words of the other letters
        c = np.full(k, single[0], np.uint32)
        c[k // 3:] = single[1]
        assert np.array_equal(assign_centers(w, c, L, igctx), oracle.assign_centers(w, c, L)), (L, k)
