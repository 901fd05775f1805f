"""Levels of few entries are contracted in one cooperative launch: its classes
end at 32, 256 (128 for float weights) and 4096 (2048) stream entries, longer
communities take global tables, and rows of over 4096 entries are copied by all
blocks.  Against the general contraction, which set_long_rows(1) selects, and
the oracle."""
import numpy as np
import pytest

from test_gpu_parity import _assert_same, _sym_graph

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.cuda.init()
    return torch


def _cliques(sizes, seed):
    """Cliques of the given sizes (dense communities of known entry counts)
    joined in a ring, random other edges."""
    rng = np.random.default_rng(seed)
    u, v, base = [], [], 0
    for s in sizes:
        a, b = np.triu_indices(s, 1)
        u.append(a + base)
        v.append(b + base)
        base += s
    starts = np.concatenate([[0], np.cumsum(sizes)])[:-1]
    u.append(starts)
    v.append(np.roll(starts, 1))
    u.append(rng.integers(0, base, base // 3))
    v.append(rng.integers(0, base, base // 3))
    u, v = np.concatenate(u), np.concatenate(v)
    lo, hi = np.minimum(u, v).astype(np.int64), np.maximum(u, v)
    key = np.unique((lo * base + hi)[lo != hi])
    lo, hi = key // base, key % base
    a, b = np.concatenate([lo, hi]), np.concatenate([hi, lo])
    k = np.argsort(a * base + b)
    offs = np.concatenate([[0], np.cumsum(np.bincount(a, minlength=base))]).astype(np.int64)
    return offs, b[k].astype(np.int32), lo, hi, k


# clique of s vertices: s (s - 1) entries and a few more
SIZES = [2, 3, 5, 6, 7, 11, 12, 16, 17, 23, 45, 46, 64, 65, 91, 120, 260]


@pytest.mark.parametrize("kind", ["unit", "int", "float"])
def test_community_sizes(ffi, oracle, torch_cuda, kind):
    offs, nbr, lo, hi, k = _cliques(SIZES, 3)
    n = offs.shape[0] - 1
    w = (1 + (lo * 5 + hi * 3) % 7)
    w = np.concatenate([w, w])[k].astype(np.int32)
    if kind == "float":
        wf = (w * 0.3).astype(np.float32)
        g, o = ffi.Graph.from_csr_f32(offs, nbr, wf), oracle.louvain_f32(offs, nbr, wf)
    else:
        w = w if kind == "int" else None
        g, o = ffi.Graph.from_csr(offs, nbr, w), oracle.louvain(offs, nbr, w)
    ctx = ffi.Context(n, offs[-1])
    r = ctx.louvain(g)
    ctx.set_long_rows(1)
    general = ctx.louvain(g)
    ctx.close()
    assert r["iter_q"] == o["iter_q"] and np.array_equal(r["labels"], o["labels"])
    assert general["iter_q"] == r["iter_q"] and general["level_c"] == r["level_c"]
    assert [x["entries"] for x in general["levels"]] == [x["entries"] for x in r["levels"]]


@pytest.mark.parametrize("n,m,hubs", [(3, 2, ()), (40, 70, ()), (5000, 20000, [(1, 4999), (2, 4500)]),
                                      (60000, 90000, [(7, 9000), (8, 13000)]), (65537, 60000, ())])
def test_random_graphs(ffi, oracle, torch_cuda, n, m, hubs):
    """Hub rows, isolated vertices, vertex counts on both sides of the limit."""
    offs, nbr, w = _sym_graph(np.random.default_rng(n), n, m, True, hubs=hubs)
    ctx = ffi.Context(n, max(1, offs[-1]))
    r = ctx.louvain(ffi.Graph.from_csr(offs, nbr, w))
    ctx.close()
    _assert_same(r, oracle.louvain(offs, nbr, w))
