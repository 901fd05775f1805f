"""Degree-bin tuning on levels that run in one launch: the limits of bins 4 and 5
and the bin-5 block, tuned for the one-bin launches, neither change the partition
nor slow such a level down."""
import time

import numpy as np
import pytest

from test_batch import torch_cuda  # noqa: F401


def _planted(n, deg, size, seed):
    rng = np.random.default_rng(seed)
    m = n * deg // 2
    u = rng.integers(0, n, m)
    v = np.where(rng.random(m) < 0.3, rng.integers(0, n, m), np.minimum(n - 1, u // size * size + rng.integers(0, size, m)))
    key = np.unique(np.minimum(u, v) * n + np.maximum(u, v))
    lo, hi = key // n, key % n
    lo, hi = lo[lo != hi], hi[lo != hi]
    a, b = np.concatenate([lo, hi]), np.concatenate([hi, lo])
    order = np.argsort(a * n + b)
    return np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n))]).astype(np.int64), b[order].astype(np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["int", "float"])
def test_limits_on_a_small_level(ffi, oracle, torch_cuda, kind):  # noqa: F811
    offs, nbr = _planted(30000, 100, 300, 4)
    assert 1 << 21 < offs[-1] <= 1 << 23
    if kind == "int":
        g, o = ffi.Graph.from_csr(offs, nbr, None), oracle.louvain(offs, nbr, None, nthreads=8)
    else:
        w = np.full(nbr.shape[0], 0.5, dtype=np.float32)
        g, o = ffi.Graph.from_csr_f32(offs, nbr, w), oracle.louvain_f32(offs, nbr, w, nthreads=8)
    ctx = ffi.Context(30000, offs[-1])
    best = []
    for tuning in (None, {"bin_max": [64, 1024, 4096], "bin5_block": 512}, {"bin_max": [32, 32, 100], "bin5_block": 256},
                   {"bin_max": [128, 200, 2000], "bin5_block": 256}):
        times = []
        for _ in range(5):
            t = time.perf_counter()
            r = ctx.louvain(g, tuning=tuning)
            times.append(time.perf_counter() - t)
        best.append(min(times))
        assert np.array_equal(r["labels"], o["labels"]) and r["iter_q"] == o["iter_q"]
    ctx.close()
    assert best[1] <= 1.4 * best[0], best
