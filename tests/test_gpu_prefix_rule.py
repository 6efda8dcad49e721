"""Which lone builds run shared prefixes once (the tiling tells: a width and no
segments): up to a word count that depends on length and threshold, builds of
more edges by the general pass alone, and a build of too many edges for its
size wastes no compaction on the pass it gives up.  The graphs are the general
pass's, which a second, tiny job in the batch selects.  Bit-exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _general(w, L, d, ctx):
    from indexgen_b200 import build_batch

    with build_batch([(w, L, d), (w[:2], L, d)], ctx) as G:
        rp, cols = G.upper_csr()
        _, n, e = G.job_stats(0)
    return rp[:n + 1], cols[:e]


@pytest.mark.parametrize("L,d,n,shared", [
    (10, 3, 100000, True), (10, 4, 32768, False), (10, 4, 90000, False), (11, 3, 40000, True), (11, 4, 140000, True),
    (11, 4, 140001, False), (12, 4, 60000, True), (12, 5, 32768, False), (12, 5, 90000, False), (13, 5, 206000, True),
    (13, 5, 206001, False), (16, 5, 40000, True), (10, 5, 40000, False), (13, 6, 40000, False), (12, 2, 40000, False),
])
def test_route(igctx, L, d, n, shared):
    from indexgen_b200 import build_conflict_graph, workloads as W

    w = W.uniform_words(n, L, 9900 + L)
    rp, cols = _general(w, L, d, igctx)
    igctx.set_profiling(True)
    try:
        with build_conflict_graph(w, L, d, igctx) as G:
            assert (G.job_tiling(0)[1] == 0) == shared
            assert igctx.phase_time(0)[1] == 1  # one pair pass: none thrown away
            r, c = G.upper_csr()
    finally:
        igctx.set_profiling(False)
    assert np.array_equal(r, rp) and np.array_equal(c, cols)


def test_a_pass_given_up_is_not_compacted(igctx):
    """50,000 words of ten distinct ones: 2,500 edges a word.  On a context whose
    buffers hold them all, compacting them twice took five times as long as
    once."""
    from indexgen_b200 import build_batch, build_conflict_graph, workloads as W

    w = W.uniform_words(2000, 14, 9950)[np.random.default_rng(4).integers(0, 10, 50000)]
    rp, cols = _general(w, 14, 3, igctx)
    assert rp[-1] > 2000 * len(w)
    ms = []
    for build in (lambda: build_batch([(w, 14, 3), (w[:2], 14, 3)], igctx), lambda: build_conflict_graph(w, 14, 3, igctx)):
        build().close()
        igctx.set_profiling(True)
        with build() as G:
            r, c = G.upper_csr()
        ms.append(igctx.phase_time(1)[0])
        igctx.set_profiling(False)
    assert np.array_equal(r, rp) and np.array_equal(c, cols)
    assert ms[1] < 2.5 * ms[0], ms
