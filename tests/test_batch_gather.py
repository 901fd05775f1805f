"""Batches whose CTAs copy their graphs from page-locked memory themselves:
vertex and entry counts at the edges of the copy's 512-thread, 8-wide tiles,
graphs without entries, weighted and unweighted graphs in one batch, against
the staged copy of the same graphs and single runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ring(n, chords, weighted, seed):
    """n vertices, 2 (n + chords) entries for n > 2."""
    rng = np.random.default_rng(seed)
    pairs = {(i, i + 1) for i in range(n - 1)}
    if n > 2:
        pairs.add((0, n - 1))
        while len(pairs) < n + chords:
            a, b = sorted(int(x) for x in rng.integers(0, n, 2))
            if a != b:
                pairs.add((a, b))
    p = np.array(sorted(pairs), dtype=np.int64).reshape(-1, 2)
    wt = rng.integers(1, 9, p.shape[0])
    src, dst = np.concatenate([p[:, 0], p[:, 1]]), np.concatenate([p[:, 1], p[:, 0]])
    order = np.lexsort((dst, src))
    offs = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int64)
    return offs, dst[order].astype(np.int32), np.concatenate([wt, wt])[order].astype(np.int32) if weighted else None


# (vertices, chords): entries 2 (n + chords), around 512, 4096 and 8192
SIZES = [(1, 0), (2, 0), (64, 191), (64, 192), (64, 193), (511, 0), (512, 1536), (513, 1536), (700, 1347), (700, 1349),
         (4095, 1), (4096, 0), (4096, 1)]


@pytest.mark.parametrize("weights", ["none", "all", "mixed"])
def test_pinned_batch_equals_staged_batch_and_single_runs(ffi, weights):
    csr = [_ring(n, c, weights == "all" or (weights == "mixed" and i % 2 == 1), i) for i, (n, c) in enumerate(SIZES)]
    csr.append((np.zeros(8, dtype=np.int64), np.zeros(0, dtype=np.int32), None))  # no entries
    csr.append(csr[5])
    n, e = sum(c[0].shape[0] - 1 for c in csr), sum(int(c[0][-1]) for c in csr)
    ctx = ffi.Context(n, e)
    staged = ctx.louvain_batch([ffi.Graph.from_csr(*c) for c in csr], batch_mode=0)
    graphs = [ffi.Graph.from_csr(*c) for c in csr]
    for g in graphs:
        try:
            g.pin()
        except ffi.GalaError:
            pass  # arrays sharing a page with one already registered: the batch is staged
    pinned = ctx.louvain_batch(graphs, batch_mode=0)
    assert np.array_equal(pinned["modularity"], staged["modularity"])
    assert np.array_equal(pinned["communities"], staged["communities"])
    for i, c in enumerate(csr):
        assert np.array_equal(pinned["labels"][i], staged["labels"][i]), SIZES[i]
        if c[1].size:
            one = ctx.louvain(ffi.Graph.from_csr(*c))
            assert np.array_equal(pinned["labels"][i], one["labels"]), SIZES[i]
            assert pinned["modularity"][i] == one["modularity"]
    ctx.close()
