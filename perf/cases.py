"""Cases by which the speed of the conflict-graph path is measured.

Each case is one call (or a build and its device CSR) through the package's
public entry points, on candidate sets like the ones the codebook generator
makes: filtered uniform words (maxRun 3, GC content 0.3 to 0.7) or cosets of
the [12,9,3] GF(4) code, lengths 10 to 16, editDist 3 to 7.

    listed()             the fixed cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  candidates in hand before the call, from the seed alone
    run(state)           one pass; returns its outputs whole
    work(case)           bytes and cell updates a pass cannot do without
    exact(case, seed)    the outputs by plain dynamic programming, where quick
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import indexgen_b200 as ig
from indexgen_b200 import workloads

FILTERS = dict(max_run=3, min_gc=0.3, max_gc=0.7)


def listed():
    return [
        # One small cluster, the size a many-way clustering leaves: launches
        # and latency are all of it.
        dict(name="build_2k_l12_d4", kind="build", source="uniform", n=2000, L=12, d=4),
        # 20,000 uniform n=11 draws after the filters: the generator's ordinary
        # quick run, an odd word count.
        dict(name="build_14k_l11_d4", kind="build", source="uniform", n=14375, L=11, d=4),
        # The linear-code method at its benchmark size: [12,9,3] code + random
        # coset, about 207,000 words after the filters, of which 201,601 are taken.
        dict(name="build_code12_d4", kind="build", source="code", n=201601, L=12, d=4),
        # Many long words, the smallest threshold in use: a sparse graph.
        dict(name="build_150k_l15_d3", kind="build", source="uniform", n=150001, L=15, d=3),
        # The largest call: n=16 at editDist 5, the big sparse graph.
        dict(name="build_300k_l16_d5", kind="build", source="uniform", n=300000, L=16, d=5),
        # Short words at editDist 5: a dense graph, some 3 x 10^7 edges from 40,000 words.
        dict(name="build_40k_l10_d5", kind="build", source="uniform", n=40000, L=10, d=5),
        # A deep threshold on a medium set: every tenth pair or so conflicts.
        dict(name="build_20k_l13_d7", kind="build", source="uniform", n=19999, L=13, d=7),
        # A serving tick: sixteen small jobs of mixed lengths and thresholds in one build.
        dict(name="batch_mixed_16x3k", kind="batch_build", jobs=16, n=3000),
        # The clustered generator: 32 clusters of Zipf sizes, graphs and codebooks in one call.
        dict(name="solve_batch_32_l14_d4", kind="solve_batch", jobs=32, n=250000, L=14, d=4),
        # Words to codebook for one job, the library's whole service.
        dict(name="solve_30k_l12_d4", kind="solve", source="uniform", n=30000, L=12, d=4),
        # Verifying a large codebook's distance from host words: a count and no graph.
        dict(name="count_100k_l16_d4", kind="count", source="uniform", n=100003, L=16, d=4),
        # random_cluster's step: a million words to their nearest of 64 centres.
        dict(name="assign_1m_l14_k64", kind="assign", n=1000000, L=14, k=64),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["build", "build", "build", "build", "batch_build", "solve_batch", "solve", "count", "assign"])
    if kind == "assign":
        return dict(kind=kind, n=_log_uniform(rng, 10000, 1000000), L=rng.randint(10, 16), k=rng.randint(5, 64))
    if kind == "batch_build":
        return dict(kind=kind, jobs=rng.randint(4, 24), n=_log_uniform(rng, 500, 5000))
    if kind == "solve_batch":
        jobs = rng.randint(8, 32)
        return dict(kind=kind, jobs=jobs, n=_log_uniform(rng, 3000 * jobs, 7000 * jobs), L=rng.randint(12, 16), d=4)
    L = rng.randint(10, 16)
    d = rng.choice([3, 4, 4, 5, 5, rng.randint(6, 7) if kind == "build" else 4])
    # as many words as the edges leave room for: 3e7 for a graph, 2e6 for a greedy
    most = {"build": 250000, "solve": 60000, "count": 250000}[kind]
    edges = {"build": 3e7, "solve": 2e6, "count": 3e7}[kind]
    most = int(min(most, math.sqrt(2 * edges / _density(L, d)), _population(L) // 2))
    n = _log_uniform(rng, 2000, max(most, 2100))
    return dict(kind=kind, source="uniform", n=n, L=L, d=d)


def _population(L):
    """About how many words of length L pass the filters."""
    return int(0.6 * 4 ** L)


@functools.lru_cache(maxsize=None)
def _sampled_distances(L):
    """How many of 10^6 uniform word pairs of length L lie at each distance."""
    rng = np.random.default_rng(L)
    a, b = (torch.from_numpy(rng.integers(0, 4, size=(1000000, L), dtype=np.int8)) for _ in range(2))
    return np.bincount(_distance(a, b).numpy(), minlength=L + 1)


def _density(L, d):
    """Share of the pairs of uniform words of length L with distance < d."""
    return max(int(_sampled_distances(L)[:d].sum()), 1) / 1e6


def _distance(a, b):
    """Levenshtein distances by dynamic programming, one row at a time, of the
    digit arrays a [..., L] and b [..., L] (broadcast against each other)."""
    L = a.shape[-1]
    shape = torch.broadcast_shapes(a.shape[:-1], b.shape[:-1])
    row = [torch.full(shape, j, dtype=torch.int8, device=a.device) for j in range(L + 1)]
    for i in range(L):
        diag, row[0] = row[0], torch.full(shape, i + 1, dtype=torch.int8, device=a.device)
        for j in range(L):
            sub = diag + (a[..., i] != b[..., j]).to(torch.int8)
            diag = row[j + 1]
            row[j + 1] = torch.minimum(sub, torch.minimum(diag, row[j]) + 1)
    return row[L]


def _words(source, n, L, seed):
    if source == "code":
        bias = np.random.default_rng(seed).integers(0, 4, size=L)
        w = workloads.linear_code_words(L, bias)
        w = w[workloads.filter_words(w, L, FILTERS["max_run"], FILTERS["min_gc"], FILTERS["max_gc"])]
        if len(w) < n:
            raise ValueError("the coset leaves fewer words than the case takes")
        return w[:n]
    return workloads.uniform_until(n, L, seed, **FILTERS)


def _mixed_shapes(case):
    """(n, L, editDist) of a mixed batch: lengths 10 to 16, thresholds 3 to 5
    in turn, sizes within a factor of two either way."""
    rng = np.random.default_rng(case["jobs"])
    return [(int(case["n"] * 2.0 ** rng.uniform(-1, 1)), int(rng.integers(10, 17)), 3 + j % 3)
            for j in range(case["jobs"])]


def _mixed_jobs(case, seed):
    rng = np.random.default_rng(seed)
    return [(workloads.uniform_until(n, L, int(rng.integers(1 << 31)), **FILTERS), L, d)
            for n, L, d in _mixed_shapes(case)]


def _cluster_jobs(case, seed):
    L, k, n = case["L"], case["jobs"], case["n"]
    w = workloads.uniform_until(n, L, seed, **FILTERS)
    sizes = workloads.zipf_sizes(n, k, lo=min(2000, n // k), hi=60000)
    return [(w[p], L, case["d"]) for p in workloads.assign_clusters(w, L, sizes, seed + 1)]


def _on_device(words):
    return torch.from_numpy(words.view(np.int32)).cuda()


def _room(shapes):
    """Columns a caller sets aside for the edges of (n, L, editDist) jobs."""
    edges = sum(n * (n - 1) / 2 * _density(L, d) for n, L, d in shapes)
    return int(2 * edges) + 8192


def _build_shapes(case):
    return _mixed_shapes(case) if case["kind"] == "batch_build" else [(case["n"], case["L"], case["d"])]


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case)
    if kind == "batch_build":
        state["jobs"] = _mixed_jobs(case, seed)
    elif kind == "solve_batch":
        state["jobs"] = _cluster_jobs(case, seed)
    else:
        words = _words(case.get("source"), case["n"], case["L"], seed)
        if kind == "assign":
            pick = np.random.default_rng(seed + 1).choice(len(words), case["k"], replace=False)
            state["centres"] = _on_device(words[pick])
        # a build takes words already on the GPU; the host calls take host words
        state["words"] = _on_device(words) if kind in ("build", "assign") else words
    # results go to arrays of the caller's, -1 behind their end
    if kind in ("build", "batch_build"):
        shapes = _build_shapes(case)
        rows = sum(n for n, _, _ in shapes)
        state["row_ptr"] = torch.full((rows + 1,), -1, dtype=torch.int64, device="cuda")
        state["cols"] = torch.full((_room(shapes),), -1, dtype=torch.int32, device="cuda")
    elif kind in ("solve", "solve_batch"):
        state["book"] = np.full(case["n"], -1, np.int32)
    ig.default_context()
    torch.cuda.synchronize()
    return state


class _DeviceArray:
    """A device array of a graph as torch sees it."""

    def __init__(self, address, count, typestr):
        self.__cuda_array_interface__ = dict(shape=(count,), typestr=typestr, data=(address, False), version=2)


def _take_csr(graph, state):
    """The graph's device CSR into the caller's arrays; frees the graph."""
    with graph:
        row_ptr, cols = graph.device_csr()
        state["row_ptr"].copy_(torch.as_tensor(_DeviceArray(row_ptr, graph.n + 1, "<i8"), device="cuda"))
        if graph.edges:
            state["cols"][:graph.edges].copy_(torch.as_tensor(_DeviceArray(cols, graph.edges, "<i4"), device="cuda"))
        torch.cuda.current_stream().synchronize()  # the copies, before their source goes
    return state["row_ptr"], state["cols"]


def run(state):
    kind = state["kind"]
    if kind == "build":
        return _take_csr(ig.build_conflict_graph(state["words"], state["L"], state["d"]), state)
    if kind == "batch_build":
        return _take_csr(ig.build_batch(state["jobs"]), state)
    if kind == "solve_batch":
        books, edges = ig.solve_batch(state["jobs"])
        first = 0
        for (words, _, _), book in zip(state["jobs"], books):
            state["book"][first:first + len(book)] = book
            first += len(words)
        return state["book"], edges
    if kind == "solve":
        book, edges = ig.solve(state["words"], state["L"], state["d"])
        state["book"][:len(book)] = book
        return state["book"], edges
    if kind == "count":
        return ig.count_conflicts(state["words"], state["L"], state["d"])
    return ig.assign_centers(state["words"], state["centres"], state["L"])


def _pairs_cells(n, L, d):
    """Pair tests of a job and the distance cells each needs: the band of
    half-width (d-1)/2 around the diagonal."""
    pairs = n * (n - 1) // 2
    w = min((d - 1) // 2, L - 1)
    return pairs, L * (2 * w + 1) - w * (w + 1)


def work(case):
    """Bytes: words in, results out.  Operations: one per distance cell."""
    kind = case["kind"]
    if kind == "assign":
        return dict(bytes=4 * case["n"] + 4 * case["k"] + 4 * case["n"], flops=case["n"] * case["k"] * case["L"] ** 2)
    if kind == "batch_build":
        jobs = _mixed_shapes(case)
    elif kind == "solve_batch":
        jobs = [(case["n"] // case["jobs"], case["L"], case["d"])] * case["jobs"]
    else:
        jobs = [(case["n"], case["L"], case["d"])]
    nbytes = ops = 0
    for n, L, d in jobs:
        pairs, cells = _pairs_cells(n, L, d)
        ops += pairs * cells
        nbytes += 4 * n
        if kind != "count":
            nbytes += 8 * n
            nbytes += int(4 * pairs * _density(L, d)) if kind in ("build", "batch_build") else 4 * n
    return dict(bytes=nbytes, flops=ops)


_EXACT_PAIRS = 1 << 27  # some seconds on a GPU


def _digits(words, L):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return torch.from_numpy(workloads.unpack_digits(words, L)).to(dev)


def _exact_csr(words, L, d):
    """Row counts and ascending columns (int64 numpy) of one job's upper graph."""
    x = _digits(words, L)
    n = len(words)
    counts, cols = [], []
    step = max(1, (1 << 22) // max(n, 1))
    for r0 in range(0, n, step):
        rows = x[r0:r0 + step]
        hit = _distance(rows[:, None, :], x[None, :, :]) < d
        hit &= torch.arange(n, device=x.device)[None, :] > torch.arange(r0, r0 + len(rows), device=x.device)[:, None]
        counts.append(hit.sum(dim=1).cpu().numpy())
        cols.append(hit.nonzero()[:, 1].cpu().numpy())
    return np.concatenate(counts), np.concatenate(cols)


def exact(case, seed):
    kind = case["kind"]
    if kind == "assign":
        if case["n"] * case["k"] > _EXACT_PAIRS:
            return None
        words = _words(None, case["n"], case["L"], seed)
        pick = np.random.default_rng(seed + 1).choice(len(words), case["k"], replace=False)
        x, c = _digits(words, case["L"]), _digits(words[pick], case["L"])
        best = torch.full((len(words),), 127, dtype=torch.int8, device=x.device)
        arg = torch.zeros(len(words), dtype=torch.int32, device=x.device)
        for i in range(len(c)):
            dist = _distance(x, c[i][None, :])
            nearer = dist < best
            best[nearer] = dist[nearer]
            arg[nearer] = i
        return arg
    if kind == "solve_batch":
        return None
    if kind == "batch_build":
        jobs = _mixed_jobs(case, seed)
    else:
        if case["n"] ** 2 > 2 * _EXACT_PAIRS:
            return None
        jobs = [(_words(case["source"], case["n"], case["L"], seed), case["L"], case["d"])]
    if sum(len(w) ** 2 for w, _, _ in jobs) > 2 * _EXACT_PAIRS:
        return None
    counts, cols, first = [], [], 0
    for w, L, d in jobs:
        n_row, col = _exact_csr(w, L, d)
        counts.append(n_row)
        cols.append(col + first)
        first += len(w)
    edges = int(sum(len(c) for c in cols))
    if kind == "count":
        return edges
    if kind == "solve":
        return None, edges
    row_ptr = np.concatenate([[0], np.cumsum(np.concatenate(counts))])
    out = np.full(_room(_build_shapes(case)), -1, np.int32)
    out[:edges] = np.concatenate(cols)
    return torch.from_numpy(row_ptr.astype(np.int64)), torch.from_numpy(out)
