"""The pass that runs shared prefixes once, where an item has several row tiles:
every length and threshold at both prefix lengths, a withheld copy with other
tiles in flight, rows long enough for the bitmap sort in each of its windows of
131,072 ids, and failing allocations.  Against the general pass, which a second,
tiny job in the batch selects.  Bit-exact."""
import numpy as np
import pytest

from test_gpu_prefix import _general

pytestmark = pytest.mark.gpu


# 7, 7 and 8 shared characters; items of two to four row tiles, then of four or more
@pytest.mark.parametrize("n", [100003, 131071, 131073])
@pytest.mark.parametrize("L", [10, 11, 12, 13, 14, 15, 16])
def test_items_of_several_tiles(igctx, L, n):
    from indexgen_b200 import build_batch, build_conflict_graph, count_conflicts, workloads as W

    w = W.uniform_words(n, L, 9400 + L)
    for d in (3, 4, 5):
        if d >= L // 2 and n != 100003:
            continue
        with build_conflict_graph(w, L, d, igctx) as G:
            lone, edges = G.job_tiling(0)[1] == 0, G.edges
            got = G.upper_csr() if lone else None
        assert count_conflicts(w, L, d, igctx) == edges, (L, d)
        if lone:
            rp, cols = _general(w, L, d, igctx)
            assert np.array_equal(got[0], rp) and np.array_equal(got[1], cols), (L, d)
        else:  # too many edges for the pass to build: its count against the general build's
            with build_batch([(w, L, d), (w[:2], L, d)], igctx) as G:
                assert G.job_stats(0)[2] == edges, (L, d)


def test_withheld_copy_with_other_tiles_in_flight():
    from indexgen_b200 import (FAULT_TILE_COPY, Context, IndexGenError, build_conflict_graph, count_conflicts,
                               workloads as W)

    w = W.uniform_words(131071, 14, 9801)
    ctx = Context(0)
    try:
        ctx.set_wait_limit(20_000_000)  # about 10 ms of SM clock
        with build_conflict_graph(w, 14, 4, ctx) as G:
            assert G.job_tiling(0)[1] == 0
            want = G.upper_csr()
        for call in (build_conflict_graph, count_conflicts):
            ctx.inject_fault(FAULT_TILE_COPY)
            with pytest.raises(IndexGenError) as ei:
                call(w, 14, 4, ctx)
            assert ei.value.status == 5 and "did not land" not in str(ei.value)
            with build_conflict_graph(w, 14, 4, ctx) as G:
                got = G.upper_csr()
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    finally:
        ctx.close()


@pytest.mark.parametrize("L,d", [(16, 3), (15, 4)])
def test_long_rows_across_the_sort_windows(igctx, L, d):
    """300,000 shuffled words, some of them 300 to 3,000 times: rows of more than
    256 columns that start in each window of 131,072 ids and reach the last."""
    from indexgen_b200 import build_conflict_graph, workloads as W

    many = np.repeat(W.uniform_words(6, L, 9651), (300, 500, 900, 1500, 2200, 3000))
    w = np.concatenate([W.uniform_words(300000 - len(many), L, 9652), many])
    np.random.default_rng(7).shuffle(w)
    rp, cols = _general(w, L, d, igctx)
    with build_conflict_graph(w, L, d, igctx) as G:
        assert G.job_tiling(0)[1] == 0
        r, c = G.upper_csr()
    assert np.array_equal(r, rp) and np.array_equal(c, cols)
    long_rows = np.flatnonzero(np.diff(rp) > 256)
    assert set(long_rows // 131072) == {0, 1, 2}
    for k in (0, 1, 2):  # columns in every window from the row's own on
        assert any(len(set(cols[rp[q]:rp[q + 1]] // 131072)) == 3 - k for q in long_rows[long_rows // 131072 == k])


def test_every_allocation_can_fail():
    from indexgen_b200 import build_conflict_graph, count_conflicts, workloads as W
    from test_gpu_general_pass import alloc_sweep

    w = W.uniform_words(33000, 13, 9850)
    want = []

    def run(ctx):
        edges = count_conflicts(w, 13, 4, ctx)
        with build_conflict_graph(w, 13, 4, ctx) as G:
            assert G.job_tiling(0)[1] == 0
            return G.upper_csr() + (edges,)

    def check(out):
        want.append(out)
        assert all(np.array_equal(a, b) for a, b in zip(out, want[0]))
        assert out[2] == out[0][-1] > 0

    # words, tables, scan words, row offsets, records, columns, the graph's own columns
    assert len(alloc_sweep(run, check)) == 7
