"""A build returns with the device done: nothing of it is left on the context's
stream, and the CSR read through the device pointers from another stream, right
after the call, is the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Array:
    def __init__(self, address, count, typestr):
        self.__cuda_array_interface__ = dict(shape=(count,), typestr=typestr, data=(address, False), version=2)


@pytest.mark.parametrize("batch", [False, True])
def test_stream_is_idle_and_columns_are_there(oracle, batch):
    import torch

    from indexgen_b200 import Context, build_batch, build_conflict_graph, workloads as W

    w = W.uniform_words(36000, 10, 61)  # 2.7 x 10^7 edges, copied out of a larger workspace
    rp, cols = oracle.conflict_upper(w, 10, 5)
    ctx = Context(0)
    try:
        with build_conflict_graph(W.uniform_words(60000, 10, 62), 10, 5, ctx):
            pass
        stream, other = torch.cuda.ExternalStream(ctx.stream), torch.cuda.Stream()
        for _ in range(20):
            with (build_batch([(w, 10, 5)], ctx) if batch else build_conflict_graph(w, 10, 5, ctx)) as G:
                idle = stream.query()
                d_rp, d_cols = G.device_csr()
                with torch.cuda.stream(other):
                    r = torch.as_tensor(_Array(d_rp, G.n + 1, "<i8"), device="cuda").cpu().numpy()
                    c = torch.as_tensor(_Array(d_cols, G.edges, "<i4"), device="cuda").cpu().numpy()
                assert idle
                assert np.array_equal(r, rp) and np.array_equal(c, cols)
    finally:
        ctx.close()
