"""The tiling a graph reports is the one its pair pass used: column segments of
the general pass, column blocks and no segments where shared prefixes ran once,
the general pass's again where such a build had too many edges, zeros without
pair tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_tiling_of_each_pass():
    from indexgen_b200 import Context, build_batch, build_conflict_graph, lane_form, workloads as W

    w = W.uniform_words(40000, 13, 71)
    few = W.uniform_words(2000, 14, 72)[np.random.default_rng(3).integers(0, 40, 40000)]  # 500 edges a word
    ctx = Context(0)
    try:
        ctx.set_work_split(lane_form(13, 4), 1)
        with build_conflict_graph(w, 13, 4, ctx) as G:
            assert G.job_tiling(0) == (2048, 0)
        with build_batch([(w, 13, 4), (w[:1], 13, 4), (w[:2], 13, 4)], ctx) as G:
            width, segments = G.job_tiling(0)
            assert width >= 1024 and segments == -(-len(w) // width)
            assert G.job_tiling(1) == (0, 0)
        with build_conflict_graph(w[:8000], 13, 4, ctx) as G:
            width, segments = G.job_tiling(0)
            assert width >= 256 and segments == -(-8000 // width)
        with build_conflict_graph(few, 14, 3, ctx) as G:
            width, segments = G.job_tiling(0)
            assert G.edges > 400 * G.n and segments == -(-len(few) // width)
        with build_conflict_graph(w[:1], 13, 4, ctx) as G:
            assert G.job_tiling(0) == (0, 0)
    finally:
        ctx.close()
