"""The general pair pass on the paths that lone large jobs no longer take it
through: a withheld tile copy with a second copy in flight in both pair kernels,
builds and counts; every work split; both pair kernels in one captured graph;
edge records that outgrow their first buffer; and failing allocations on the
way.  Bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OOM, TIMEOUT = 3, 5


def _check(G, oracle, jobs):
    rp, cols = G.upper_csr()
    for j, (w, L, d) in enumerate(jobs):
        first, n, e = G.job_stats(j)
        orp, ocols = oracle.conflict_upper(w, L, d)
        assert e == orp[-1], j
        assert np.array_equal(rp[first:first + n + 1] - rp[first], orp), j
        assert np.array_equal(cols[rp[first]:rp[first + n]] - first, ocols), j


@pytest.mark.parametrize("L,d,n", [(12, 4, 40000), (16, 5, 40000), (16, 6, 24000)])
def test_withheld_copy_with_another_in_flight(oracle, L, d, n):
    """(12, 4) and (16, 5) run pair_levels, (16, 6) pair_deltas.  One item per
    CTA makes the first item's segment two staged tiles wide or more; the tiny
    second job keeps the build on the general pass."""
    from indexgen_b200 import FAULT_TILE_COPY, Context, IndexGenError, build_batch, lane_form, workloads as W

    w = W.uniform_words(n, L, 41 + L)
    jobs = [(w, L, d), (w[:2], L, d)]
    ctx = Context(0)
    try:
        ctx.set_work_split(lane_form(L, d), 1)
        ctx.set_wait_limit(20_000_000)  # about 10 ms of SM clock
        with build_batch(jobs, ctx) as G:
            width, segments = G.job_tiling(0)
            assert width >= 2048 and segments > 0
            _check(G, oracle, jobs)
            want = G.upper_csr()
        ctx.inject_fault(FAULT_TILE_COPY)
        with pytest.raises(IndexGenError) as ei:
            build_batch(jobs, ctx)
        assert ei.value.status == TIMEOUT
        assert "did not arrive" in str(ei.value) and "did not land" not in str(ei.value)
        for _ in range(2):
            with build_batch(jobs, ctx) as G:
                got = G.upper_csr()
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    finally:
        ctx.close()


def test_withheld_copy_in_a_count_of_each_kernel(oracle):
    from indexgen_b200 import FAULT_TILE_COPY, Context, IndexGenError, count_conflicts, lane_form, workloads as W

    for L, d, n in ((11, 5, 32000), (16, 6, 24000)):
        w = W.uniform_words(n, L, 43 + L)
        ctx = Context(0)
        try:
            ctx.set_work_split(lane_form(L, d), 1)
            ctx.set_wait_limit(20_000_000)
            want = count_conflicts(w, L, d, ctx)
            assert want == int(oracle.conflict_upper(w, L, d)[0][-1])
            ctx.inject_fault(FAULT_TILE_COPY)
            with pytest.raises(IndexGenError) as ei:
                count_conflicts(w, L, d, ctx)
            assert ei.value.status == TIMEOUT and "did not land" not in str(ei.value)
            assert count_conflicts(w, L, d, ctx) == want
        finally:
            ctx.close()


@pytest.mark.parametrize("L,d,n", [(12, 4, 60000), (16, 7, 30000)])
def test_graph_independent_of_work_split(oracle, L, d, n):
    from indexgen_b200 import Context, build_batch, lane_form, workloads as W

    w = W.uniform_words(n, L, 2025)
    form = lane_form(L, d)
    ctx = Context(0)
    try:
        ctx.set_autotune(False)
        ref, widths = None, set()
        for split in (1, 6, 24, 96, 4096):
            ctx.set_work_split(form, split)
            with build_batch([(w, L, d), (w[:6000], L, d)], ctx) as G:
                got = G.upper_csr()
                widths.add(G.job_tiling(0)[0])
                if ref is None:
                    ref = got
                    first, m, _ = G.job_stats(1)
                    orp, ocols = oracle.conflict_upper(w[:6000], L, d)
                    assert np.array_equal(got[0][first:first + m + 1] - got[0][first], orp)
                    assert np.array_equal(got[1][got[0][first]:] - first, ocols)
            assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1]), split
        assert len(widths) >= 3  # the splits did cut the job differently
    finally:
        ctx.close()


def test_both_pair_kernels_in_one_graph_and_record_growth(oracle):
    """45,000 words at L = 10, editDist 4 (pair_levels) have some 6 x 10^6 edges,
    more than the first record buffer; (13, 9) runs pair_deltas; (10, 5) keeps
    hit words beside the records."""
    from indexgen_b200 import Context, build_batch, build_conflict_graph, workloads as W

    grows = (W.uniform_words(45000, 10, 78), 10, 4)
    jobs = [grows, (W.uniform_words(900, 13, 5), 13, 9), (W.uniform_words(8300, 10, 6), 10, 5)]
    ctx, lone = Context(0), Context(0)
    try:
        ctx.set_autotune(False)
        for _ in range(2):
            with build_batch(jobs, ctx) as G:
                assert G.job_stats(0)[2] > (1 << 22)
                _check(G, oracle, jobs)
        launches, inst, upd = ctx.graph_stats()
        assert launches == 3  # the first build's pass ran twice
        for _ in range(2):
            with build_conflict_graph(*grows, lone) as G:
                assert G.job_tiling(0)[1] > 0
                _check(G, oracle, [grows])
        assert lone.graph_stats()[0] == 3
    finally:
        ctx.close()
        lone.close()


def alloc_sweep(run, check):
    """Fails the k-th device allocation of a fresh context for every k that the
    run reaches; the run is refused as out of memory, or goes on with a smaller
    buffer and is exact, and so are the runs after it.  The ks refused."""
    from indexgen_b200 import FAULT_DEVICE_ALLOC, FAULT_NONE, Context, IndexGenError

    refused = []
    for k in range(1, 64):
        ctx = Context(0)
        try:
            ctx.inject_fault(FAULT_DEVICE_ALLOC, k)
            try:
                check(run(ctx))
            except IndexGenError as e:
                assert e.status == OOM, (k, str(e))
                refused.append(k)
            reached = ctx.device_allocs >= k
            ctx.inject_fault(FAULT_NONE)
            check(run(ctx))
            check(run(ctx))
        finally:
            ctx.close()
        if not reached:
            return refused
    raise AssertionError("the sweep never ran past the last allocation")


def test_every_allocation_of_growing_records_can_fail(oracle):
    from indexgen_b200 import build_conflict_graph, workloads as W

    w = W.uniform_words(45000, 10, 78)
    rp, cols = oracle.conflict_upper(w, 10, 4)

    def run(ctx):
        with build_conflict_graph(w, 10, 4, ctx) as G:
            return G.upper_csr()

    def check(out):
        assert np.array_equal(out[0], rp) and np.array_equal(out[1], cols)

    # words, row offsets, records, columns, units, counts, scan words, grown records and columns
    assert len(alloc_sweep(run, check)) == 9
