"""Small unweighted levels with many hub rows are left to the one-bin kernels: the
same results on both sides of the line (320 rows above 4096 entries), with and
without refinement, and the launches of each route."""
import numpy as np
import pytest

from test_batch import torch_cuda  # noqa: F401


def _bipartite(k, d, n):
    rng = np.random.default_rng(k)
    a = np.repeat(np.arange(k, dtype=np.int64), d)
    b = np.concatenate([k + rng.permutation(n - k)[:d] for _ in range(k)])
    a, b = np.concatenate([a, b]), np.concatenate([b, a])
    order = np.argsort(a * n + b)
    return np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n))]).astype(np.int64), b[order].astype(np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("k,separate", [(320, False), (321, True), (700, True)])
def test_many_hub_rows(ffi, oracle, torch_cuda, k, separate):  # noqa: F811
    offs, nbr = _bipartite(k, 4200, 30000)
    assert offs[-1] <= 1 << 23
    g = ffi.Graph.from_csr(offs, nbr, None)
    ctx = ffi.Context(30000, offs[-1])
    for refine in (False, True):
        r = ctx.louvain(g, refine=refine)
        o = oracle.louvain(offs, nbr, None, nthreads=8, refine=refine)
        assert np.array_equal(r["labels"], o["labels"]) and r["iter_q"] == o["iter_q"]
        assert r["level_iters"] == o["level_iters"]
    assert (ctx.louvain(g, max_levels=1)["kernel_launches"] > 16) == separate
    # with weights one launch keeps the level
    w = (1 + (np.repeat(np.arange(30000), np.diff(offs)) + nbr) % 3).astype(np.int32)
    g = ffi.Graph.from_csr(offs, nbr, w)
    r, o = ctx.louvain(g), oracle.louvain(offs, nbr, w, nthreads=8)
    assert np.array_equal(r["labels"], o["labels"]) and r["iter_q"] == o["iter_q"]
    assert ctx.louvain(g, max_levels=1)["kernel_launches"] <= 16
    ctx.close()
