"""The one-launch contraction of a level whose vertices mostly stay on their own:
thousands of short community rows and few vertices per block.  The rows are dealt
to all warps, so that it takes no longer than the general path (which long-rows
mode 1 selects; 0.86 ms against 0.2 with 32 rows to every warp, 0.15 so)."""
import numpy as np
import pytest

from test_batch import torch_cuda  # noqa: F401


@pytest.mark.gpu
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("k,d,n", [(49, 2400, 4814), (3, 900, 2000), (40, 1384, 3205)])
def test_unmerged_level(ffi, oracle, torch_cuda, weighted, k, d, n):  # noqa: F811
    rng = np.random.default_rng(k)
    a = np.repeat(np.arange(k, dtype=np.int64), d)
    b = np.concatenate([k + rng.permutation(n - k)[:d] for _ in range(k)])
    a, b = np.concatenate([a, b]), np.concatenate([b, a])
    order = np.argsort(a * n + b)
    a, b = a[order], b[order]
    offs = np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n))]).astype(np.int64)
    w = (1 + (a + b) % 3).astype(np.int32) if weighted else None
    assert offs[-1] <= 1 << 18
    g = ffi.Graph.from_csr(offs, b.astype(np.int32), w)
    o = oracle.louvain(offs, b.astype(np.int32), w)
    ctx = ffi.Context(n, offs[-1])
    ms = []
    for mode in (0, 1):
        ctx.set_long_rows(mode)
        times = []
        for _ in range(6):
            r = ctx.louvain(g)
            times.append(r["levels"][0]["contract_ms"])
            assert np.array_equal(r["labels"], o["labels"]) and r["iter_q"] == o["iter_q"]
        ms.append(min(times))
    ctx.close()
    assert ms[0] <= 1.5 * ms[1], ms
