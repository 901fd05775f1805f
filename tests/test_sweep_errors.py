"""Error bits of a sweep inside the one-launch phase 1: every block takes the
same decision from them, so an overflow ends the call at once, never by a grid
barrier that ran out."""
import numpy as np
import pytest

from test_batch import torch_cuda  # noqa: F401


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["int", "float"])
def test_overflow_of_many_hubs(ffi, torch_cuda, kind):  # noqa: F811
    rng = np.random.default_rng(8)
    n, hubs = 30000, 24
    u = np.repeat(np.arange(hubs), 8192 + 1 + 300 * np.arange(hubs))
    v = np.concatenate([hubs + rng.permutation(n - hubs)[:8193 + 300 * i] for i in range(hubs)])
    a, b = np.concatenate([u, v]).astype(np.int64), np.concatenate([v, u]).astype(np.int64)
    k = np.argsort(a * n + b)
    offs = np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n))]).astype(np.int64)
    nbr = b[k].astype(np.int32)
    g = (ffi.Graph.from_csr(offs, nbr, None) if kind == "int" else
         ffi.Graph.from_csr_f32(offs, nbr, np.full(nbr.shape[0], 0.5, dtype=np.float32)))
    assert offs[-1] <= 1 << 23
    ctx = ffi.Context(n, offs[-1])
    want = ctx.louvain(g)
    for _ in range(5):
        ctx.set_hub_table_cap(1024)
        with pytest.raises(ffi.GalaError) as e:
            ctx.louvain(g)
        assert e.value.status == 7 and str(e.value).endswith("error bits 1")
        ctx.set_hub_table_cap(0)
        r = ctx.louvain(g)
        assert np.array_equal(r["labels"], want["labels"]) and r["iter_q"] == want["iter_q"]
    ctx.close()
