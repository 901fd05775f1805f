"""Union run of a batch: per-graph sums split over several blocks (few graphs)
or one block per graph, page-locked graphs gathered in chunks that start and
end inside graphs, and the incremental weight update with stopped graphs beside
running ones.  Every graph must come out as in its own run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.cuda.init()
    return torch


def _graph(ffi, n, deg, weighted, seed):
    """Planted graph of n vertices in blocks of about 40 ids."""
    rng = np.random.default_rng(seed)
    m = max(1, n * deg // 2)
    u = rng.integers(0, n, m)
    v = np.where(rng.random(m) < 0.7, np.minimum(n - 1, u // 40 * 40 + rng.integers(0, 40, m)), rng.integers(0, n, m))
    u, v = np.concatenate([u, [0]]), np.concatenate([v, [n - 1]])
    lo, hi = np.minimum(u, v), np.maximum(u, v)
    key = np.unique((lo * n + hi)[lo != hi])
    lo, hi = key // n, key % n
    a, b = np.concatenate([lo, hi]), np.concatenate([hi, lo])
    k = np.argsort(a * n + b)
    offs = np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n))]).astype(np.int64)
    w = (1 + (lo + hi) % 5) if weighted else None
    return ffi.Graph.from_csr(offs, b[k].astype(np.int32), None if w is None else np.concatenate([w, w])[k].astype(np.int32))


# sizes around the gather's 8192-entry chunks and the slices of the sums
BATCHES = {
    "few": [(2, 2, False), (3, 2, False), (700, 12, False), (9000, 16, False), (65, 4, False)],
    "weighted": [(5000, 10, True), (2, 2, False), (20000, 12, False), (640, 13, True)],
    "one": [(30000, 14, False)],
    "many": [(2 + (i * 37) % 900, 6, i % 3 == 0) for i in range(400)],
}


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("name", sorted(BATCHES))
def test_union_run_equals_single_runs(ffi, torch_cuda, name, pinned):
    graphs = [_graph(ffi, n, d, w, 100 + i) for i, (n, d, w) in enumerate(BATCHES[name])]
    if pinned:
        for g in graphs:
            g.pin()
    infos = [g.info() for g in graphs]
    ctx = ffi.Context(sum(i[0] for i in infos), sum(i[1] for i in infos))
    singles = [ctx.louvain(g) for g in graphs]
    for mode in (0, 1, 2):
        ctx.set_update_mode(mode)
        r = ctx.louvain_batch(graphs, batch_mode=1)
        for i, s in enumerate(singles):
            assert np.array_equal(r["labels"][i], s["labels"]), (mode, i)
            assert r["modularity"][i] == s["modularity"], (mode, i)
            assert r["communities"][i] == s["num_communities"], (mode, i)
    ctx.close()
