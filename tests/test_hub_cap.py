"""The cap on hub tables (gala_context_set_hub_table_cap) is for rows of more than
8192 entries (or the caller's bin_max[2]).  Small levels sum shorter rows in
global tables too, above 4096 entries and, with float weights, above 2048:
those keep tables sized by degree, and the run succeeds."""
import numpy as np
import pytest

from test_batch import torch_cuda  # noqa: F401


def _stars(degs, n):
    """Vertex i joined to degs[i] others."""
    rng = np.random.default_rng(4)
    k = len(degs)
    u = np.repeat(np.arange(k), degs)
    v = np.concatenate([k + rng.permutation(n - k)[:d] for d in degs])
    a, b = np.concatenate([u, v]).astype(np.int64), np.concatenate([v, u]).astype(np.int64)
    o = np.argsort(a * n + b)
    offs = np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n))]).astype(np.int64)
    return offs, b[o].astype(np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,degs", [("int", [4097, 8192]), ("float", [2049, 4097, 8192])])
@pytest.mark.parametrize("mode", [0, 2])  # one launch, launches of their own
def test_cap_spares_rows_up_to_8192(ffi, oracle, torch_cuda, kind, degs, mode):  # noqa: F811
    offs, nbr = _stars(degs, 20000)
    if kind == "float":
        w = np.full(nbr.shape[0], 0.5, dtype=np.float32)
        g, o = ffi.Graph.from_csr_f32(offs, nbr, w), oracle.louvain_f32(offs, nbr, w, nthreads=4)
    else:
        g, o = ffi.Graph.from_csr(offs, nbr, None), oracle.louvain(offs, nbr, None)
    ctx = ffi.Context(20000, offs[-1])
    ctx.set_update_mode(mode)
    ctx.set_hub_table_cap(32)
    r = ctx.louvain(g)
    assert np.array_equal(r["labels"], o["labels"]) and r["iter_q"] == o["iter_q"]
    # one entry more is a hub at any level size
    offs, nbr = _stars([8193], 20000)
    big = (ffi.Graph.from_csr(offs, nbr, None) if kind == "int" else
           ffi.Graph.from_csr_f32(offs, nbr, np.full(nbr.shape[0], 0.5, dtype=np.float32)))
    with pytest.raises(ffi.GalaError) as e:
        ctx.louvain(big)
    assert e.value.status == 7
    # the caller's own limit counts as the hubs' start
    if kind == "int":
        with pytest.raises(ffi.GalaError) as e:
            ctx.louvain(g, tuning={"bin_max": [256, 2048, 8191], "bin5_block": 256})
        assert e.value.status == 7
    ctx.close()
