"""The pass that runs shared prefixes once (lone sparse jobs of 32,768 words or
more, L >= 10, editDist 3..5) against the general pass, which a second, tiny job
in the batch selects: word counts around its column blocks of 2,048 and its
row tiles of 16, every length and threshold it takes, both prefix
lengths, sorted, reversed and repeated words, long rows, and the fall-back for
graphs of many edges.  Integer work: bit-exact comparisons; the oracle checks
sampled rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _general(w, L, d, ctx):
    from indexgen_b200 import build_batch

    with build_batch([(w, L, d), (w[:2], L, d)], ctx) as G:
        rp, cols = G.upper_csr()
        _, n, e = G.job_stats(0)
    return rp[:n + 1], cols[:e]


def _check(w, L, d, ctx):
    from indexgen_b200 import build_conflict_graph, count_conflicts

    rp, cols = _general(w, L, d, ctx)
    with build_conflict_graph(w, L, d, ctx) as G:
        r, c = G.upper_csr()
    assert np.array_equal(r, rp) and np.array_equal(c, cols), (len(w), L, d)
    assert count_conflicts(w, L, d, ctx) == int(rp[-1]), (len(w), L, d)
    return rp, cols


@pytest.mark.parametrize("n", [32767, 32768, 32769, 32799, 34815, 34817, 40959, 40960, 40961, 49153])
def test_word_counts(igctx, n):
    from indexgen_b200 import workloads as W

    _check(W.uniform_words(n, 13, 9300 + n), 13, 4, igctx)


@pytest.mark.parametrize("L", [10, 11, 12, 13, 14, 15, 16])
def test_lengths_and_thresholds(igctx, oracle, L):
    from indexgen_b200 import workloads as W

    w = W.uniform_words(50011, L, 9400 + L)
    rows = np.sort(np.random.default_rng(L).choice(len(w), 12, replace=False)).astype(np.int32)
    for d in (3, 4, 5):
        rp, cols = _check(w, L, d, igctx)
        want = oracle.row_neighbours(w, L, d, rows)
        owner = np.repeat(np.arange(len(w), dtype=np.int32), np.diff(rp))
        for k, r in enumerate(rows):
            got = np.concatenate([np.sort(owner[cols == r]), cols[rp[r]:rp[r + 1]]])
            assert np.array_equal(got, want[k]), (L, d, int(r))


@pytest.mark.parametrize("L,d", [(12, 4), (15, 3), (16, 5)])
def test_longer_prefix(igctx, L, d):
    from indexgen_b200 import workloads as W

    _check(W.uniform_words(160001, L, 9500 + L), L, d, igctx)


def test_word_orders_and_repeats(igctx):
    from indexgen_b200 import workloads as W

    w = W.uniform_words(50000, 12, 9600)
    _check(np.sort(w), 12, 4, igctx)
    _check(np.sort(w)[::-1].copy(), 12, 4, igctx)
    twice = np.concatenate([w[:30000], w[:30000]])
    _check(twice, 12, 4, igctx)
    # rows of a few hundred to some thousand columns beside short ones
    few = np.concatenate([W.uniform_words(60000, 16, 9601), np.repeat(W.uniform_words(3, 16, 9602), (150, 700, 3000))])
    np.random.default_rng(1).shuffle(few)
    _check(few, 16, 4, igctx)


def test_many_edges_fall_back(igctx):
    """Words from a small set: over 256 edges a word, so the general pass
    finishes the build."""
    from indexgen_b200 import workloads as W

    w = W.uniform_words(2000, 14, 9700)[np.random.default_rng(2).integers(0, 60, 50000)]
    rp, _ = _check(w, 14, 3, igctx)
    assert rp[-1] > 256 * len(w)


def test_bounded_wait_and_recovery():
    from indexgen_b200 import FAULT_TILE_COPY, Context, IndexGenError, build_conflict_graph, workloads as W

    w = W.uniform_words(60000, 13, 9800)
    ctx = Context(0)
    try:
        ctx.set_wait_limit(20_000_000)  # about 10 ms of SM clock
        with build_conflict_graph(w, 13, 4, ctx) as G:
            want = G.upper_csr()
        ctx.inject_fault(FAULT_TILE_COPY)
        with pytest.raises(IndexGenError) as ei:
            build_conflict_graph(w, 13, 4, ctx)
        assert ei.value.status == 5 and "did not land" not in str(ei.value)
        with build_conflict_graph(w, 13, 4, ctx) as G:
            got = G.upper_csr()
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    finally:
        ctx.close()
