"""A dense build whose hit words (or the columns sized by them) do not get their
memory goes on with edge records: every device allocation of such a build but
that of its words may fail once and the graph is still the oracle's.  Failures
are injected on the host (IG_FAULT_DEVICE_ALLOC)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", ["fresh", "grown"])
def test_every_allocation_of_a_dense_build_may_fail_once(oracle, first):
    from indexgen_b200 import FAULT_DEVICE_ALLOC, FAULT_NONE, Context, IndexGenError, build_batch, build_conflict_graph
    from indexgen_b200 import workloads as W

    w = W.uniform_words(12000, 10, 81)
    sparse = W.uniform_words(3000, 12, 82)
    rp, cols = oracle.conflict_upper(w, 10, 5)
    srp, scols = oracle.conflict_upper(sparse, 12, 4)

    def build(ctx):
        with build_batch([(w, 10, 5), (sparse, 12, 4)], ctx) as G:
            r, c = G.upper_csr()
        n = len(w)
        assert np.array_equal(r[:n + 1], rp) and np.array_equal(c[:rp[-1]], cols)
        assert np.array_equal(r[n:] - r[n], srp) and np.array_equal(c[rp[-1]:] - n, scols)

    refused = []
    for k in range(1, 64):
        ctx = Context(0)
        try:
            ctx.set_autotune(False)
            if first == "grown":  # workspaces of a smaller dense job before it
                with build_conflict_graph(w[:9000], 10, 5, ctx):
                    pass
            before = ctx.device_allocs
            ctx.inject_fault(FAULT_DEVICE_ALLOC, k)
            try:
                build(ctx)
            except IndexGenError as e:
                assert e.status == 3, str(e)
                refused.append(k)
            done = ctx.device_allocs - before < k
            ctx.inject_fault(FAULT_NONE)
            build(ctx)
            build(ctx)
        finally:
            ctx.close()
        if done:
            break
    assert done and k > 8
    assert refused == [1], refused  # the words' own buffer; everything after it is tried again without hit words
