"""Levels of few entries run all their sweeps in one cooperative launch; its
degree bins end at other row lengths than those of the one-bin launches, and a
level of many sweeps takes several launches.  Labels and every iteration's
modularity must equal the oracle's bit for bit, and the one-bin launches'
(which the forced incremental weight update selects)."""
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


def _run(ffi, g, mode=0):
    n, e, _ = g.info()
    ctx = ffi.Context(n, e)
    ctx.set_update_mode(mode)
    r = ctx.louvain(g)
    ctx.close()
    return r


def _path(n, w):
    """Path 0 - 1 - ... - n-1 with edge weights w."""
    u = np.arange(n - 1, dtype=np.int64)
    a, b = np.concatenate([u, u + 1]), np.concatenate([u + 1, u])
    k = np.argsort(a * n + b)
    offs = np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n))]).astype(np.int64)
    return offs, b[k].astype(np.int32), np.concatenate([w, w])[k].astype(np.int32)


@pytest.mark.parametrize("n", [2, 3, 700])
def test_many_sweeps(ffi, oracle, torch_cuda, n):
    """Rising weights move one vertex after the other: 700 vertices take over
    1000 sweeps, several launches' worth."""
    offs, nbr, w = _path(n, np.arange(1, n))
    r = _run(ffi, ffi.Graph.from_csr(offs, nbr, w))
    _assert_same(r, oracle.louvain(offs, nbr, w))
    assert n < 700 or max(r["level_iters"]) > 300


# rows around every limit: warp tables (128 / 256 entries), CTA tables (2048 /
# 4096), hub rows of one and of several 4096-entry chunks
ROWS = [4, 5, 8, 9, 16, 17, 32, 33, 127, 128, 129, 255, 256, 257, 2047, 2048, 2049, 4095, 4096, 4097, 8192, 8193, 13000]


@pytest.mark.parametrize("kind", ["unit", "int", "float"])
def test_row_length_limits(ffi, oracle, torch_cuda, kind):
    rng = np.random.default_rng(5)
    n = 16000
    u, v = [], []
    for i, d in enumerate(ROWS):  # vertex i gets a row of exactly d entries
        u.append(np.full(d, i))
        v.append(len(ROWS) + rng.permutation(n - len(ROWS))[:d])
    u, v = np.concatenate(u), np.concatenate(v)
    a, b = np.concatenate([u, v]).astype(np.int64), np.concatenate([v, u]).astype(np.int64)
    k = np.argsort(a * n + b)
    offs = np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n))]).astype(np.int64)
    assert list(np.diff(offs)[:len(ROWS)]) == ROWS
    nbr = b[k].astype(np.int32)
    w = (1 + ((np.minimum(a, b) * 7 + np.maximum(a, b) * 13) % 11))[k].astype(np.int32)
    if kind == "float":
        g = ffi.Graph.from_csr_f32(offs, nbr, (w * 0.37).astype(np.float32))
        o = oracle.louvain_f32(offs, nbr, (w * 0.37).astype(np.float32), nthreads=4)
    else:
        w = w if kind == "int" else None
        g = ffi.Graph.from_csr(offs, nbr, w)
        o = oracle.louvain(offs, nbr, w)
    r = _run(ffi, g)
    assert r["iter_q"] == o["iter_q"]
    assert np.array_equal(r["labels"], o["labels"])
    full = _run(ffi, g, mode=2)
    assert full["iter_q"] == r["iter_q"] and full["level_iters"] == r["level_iters"]
    assert full["decisions"] == r["decisions"]
    assert [x["movers"] for x in full["levels"]] == [x["movers"] for x in r["levels"]]
    assert [x["active_entries"] for x in full["levels"]] == [x["active_entries"] for x in r["levels"]]
    assert np.array_equal(full["labels"], r["labels"])


@pytest.mark.parametrize("m,weighted", [(40, True), (3000, False), (200000, True)])
def test_random_levels(ffi, oracle, torch_cuda, m, weighted):
    offs, nbr, w = _sym_graph(np.random.default_rng(m), max(8, m // 8), m, weighted)
    r = _run(ffi, ffi.Graph.from_csr(offs, nbr, w))
    _assert_same(r, oracle.louvain(offs, nbr, w))
