"""Dense jobs (8,192 words or more at editDist >= L/2), whose pair pass keeps
hit words: word counts around the words' units and blocks, list overflow (more
than a quarter of the pairs), wide segments, batches beside sparse jobs, and a
first build on a fresh context, which outgrows its column workspace.  Integer
work: bit-exact comparisons with the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(G, oracle, w, L, d):
    rp, cols = oracle.conflict_upper(w, L, d)
    r, c = G.upper_csr()
    assert np.array_equal(r, rp) and np.array_equal(c, cols), (len(w), L, d)


@pytest.mark.parametrize("n", [8191, 8192, 8193, 8255, 8257, 8447, 8449])
@pytest.mark.parametrize("L,d", [(10, 5), (13, 7), (12, 9)])
def test_sizes_and_densities(igctx, oracle, n, L, d):
    from indexgen_b200 import build_conflict_graph, workloads as W

    w = W.uniform_words(n, L, 9000 + n)
    with build_conflict_graph(w, L, d, igctx) as G:
        _same(G, oracle, w, L, d)


@pytest.mark.parametrize("split", [1, 24, 4096])
def test_segment_widths_and_a_fresh_context(oracle, split):
    from indexgen_b200 import Context, build_conflict_graph, lane_form, workloads as W

    w = W.uniform_words(20011, 10, 9100)
    ctx = Context(0)
    try:
        ctx.set_work_split(lane_form(10, 5), split)
        for _ in range(2):
            with build_conflict_graph(w, 10, 5, ctx) as G:
                _same(G, oracle, w, 10, 5)
    finally:
        ctx.close()


def test_batch_with_sparse_jobs(igctx, oracle):
    from indexgen_b200 import build_batch, workloads as W

    jobs = [(W.uniform_words(n, L, 9200 + n), L, d)
            for n, L, d in ((9001, 10, 5), (3000, 12, 4), (8300, 14, 3), (8700, 11, 6), (2, 10, 5), (8200, 6, 7))]
    with build_batch(jobs, igctx) as G:
        rp, cols = G.upper_csr()
        for j, (w, L, d) in enumerate(jobs):
            first, n, e = G.job_stats(j)
            orp, ocols = oracle.conflict_upper(w, L, d)
            assert e == orp[-1], j
            assert np.array_equal(rp[first:first + n + 1] - rp[first], orp), j
            assert np.array_equal(cols[rp[first]:rp[first + n]] - first, ocols), j
