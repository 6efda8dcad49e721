"""Neighbour lists that name a vertex twice, or their own: the greedy deletes
each vertex of a ball once, on one thread and on two, as the oracle's
restatement of the reference's AdjList does.  Host-only; bit-exact."""
import numpy as np
import pytest


@pytest.fixture
def G():
    from indexgen_b200 import build as B

    B.build()
    import indexgen_b200 as G

    yield G
    G.set_greedy_threads(-1, -1)


def _lists(n, pairs, loops):
    rows = [[] for _ in range(n)]
    for u, v in pairs:
        rows[u].append(int(v))
        rows[v].append(int(u))
    for x in loops:
        rows[x].insert(len(rows[x]) // 2, int(x))
    ap = np.zeros(n + 1, np.int64)
    ap[1:] = np.cumsum([len(r) for r in rows])
    return ap, np.array([y for r in rows for y in r], np.int32)


@pytest.mark.parametrize("helpers", [0, 1])
@pytest.mark.parametrize("kind", ["self", "repeats", "both"])
def test_repeated_neighbours(G, oracle, kind, helpers):
    rng = np.random.default_rng(5)
    G.set_greedy_threads(helpers, 0)
    for _ in range(60):
        n = int(rng.integers(2, 60))
        p = rng.integers(0, n, (int(rng.integers(1, 400)), 2))
        p = p[p[:, 0] != p[:, 1]]
        if kind == "self":
            p = np.unique(np.sort(p, axis=1), axis=0)
        loops = rng.choice(n, n // 3, replace=False) if kind != "repeats" else []
        ap, adj = _lists(n, p, loops)
        assert np.array_equal(G.codebook_from_adjacency(ap, adj, n), oracle.greedy(ap, adj, n))
    # a list longer than the chunk its row is walked in
    ap, adj = _lists(3, [(0, 1)] * 6000 + [(1, 2)] * 5000, [0, 2])
    assert np.array_equal(G.codebook_from_adjacency(ap, adj, 3), oracle.greedy(ap, adj, 3))


def test_repeated_edges_of_an_upper_csr(G, oracle):
    rp = np.array([0, 4, 6, 6], np.int64)
    cols = np.array([1, 1, 2, 1, 2, 2], np.int32)
    for helpers in (0, 1):
        G.set_greedy_threads(helpers, 0)
        for order_threads in (1, 3):
            assert np.array_equal(G.codebook_from_upper_csr(rp, cols, 3, order_threads),
                                  oracle.codebook(rp, cols, 3, order_threads))
