"""Phase 1 of a small level over several launches (256 sweeps each) with float
weights and with hub rows: totals, active lists and hub tables carry over."""
import numpy as np
import pytest

from test_batch import torch_cuda  # noqa: F401


def _path_with_hubs(n, leaves):
    """Path 0 - 1 - ... - n-1 of rising weights (one vertex moves after the other),
    and stars of `leaves` leaves whose centres are joined to the path's end."""
    u = np.arange(n - 1, dtype=np.int64)
    a, b, w = [u], [u + 1], [u + 1]
    first = n
    for k in leaves:
        a.append(np.full(k + 1, first, dtype=np.int64))
        b.append(np.concatenate([[n - 1], np.arange(first + 1, first + 1 + k)]))
        w.append(np.concatenate([[n], np.ones(k, dtype=np.int64)]))
        first += k + 1
    a, b, w = np.concatenate(a), np.concatenate(b), np.concatenate(w)
    a, b, w = np.concatenate([a, b]), np.concatenate([b, a]), np.concatenate([w, w])
    order = np.argsort(a * first + b)
    offs = np.concatenate([[0], np.cumsum(np.bincount(a, minlength=first))]).astype(np.int64)
    return offs, b[order].astype(np.int32), w[order].astype(np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["int", "float"])
@pytest.mark.parametrize("leaves", [[], [5000], [3000]])
def test_many_sweeps(ffi, oracle, torch_cuda, kind, leaves):  # noqa: F811
    offs, nbr, w = _path_with_hubs(400, leaves)
    if kind == "float":
        w = w.astype(np.float32) * np.float32(0.37)
        g, o = ffi.Graph.from_csr_f32(offs, nbr, w), oracle.louvain_f32(offs, nbr, w, nthreads=4)
    else:
        g, o = ffi.Graph.from_csr(offs, nbr, w), oracle.louvain(offs, nbr, w)
    assert max(o["level_iters"]) > 300
    ctx = ffi.Context(offs.shape[0] - 1, offs[-1])
    r = ctx.louvain(g)
    ctx.close()
    assert r["iter_q"] == o["iter_q"] and r["level_iters"] == o["level_iters"]
    assert np.array_equal(r["labels"], o["labels"])
