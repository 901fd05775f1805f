"""Rows that the contraction returns sorted, at the lengths where the sort
changes hands: warp registers (32 ... 512 pairs), shared memory (4096 and 16384)
and the bitmap over the communities; against the same contraction in numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = [0, 1, 2, 31, 32, 33, 64, 65, 128, 129, 256, 257, 511, 512, 513, 1024, 1025, 2049, 4095, 4096, 4097, 8193, 16383,
        16384, 16385, 20011]


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.cuda.init()
    return torch


def _expected(n, offs, nbr, w, comm):
    ids, lab = np.unique(comm, return_inverse=True)
    C = len(ids)
    row = np.repeat(np.arange(n), np.diff(offs))
    key, inv = np.unique(lab[row] * np.int64(C) + lab[nbr], return_inverse=True)
    wsum = np.bincount(inv, weights=w, minlength=len(key)).astype(np.int64)
    noffs = np.concatenate([[0], np.cumsum(np.bincount(key // C, minlength=C))])
    return lab, noffs, key % C, wsum


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("merge", [1, 2])
@pytest.mark.parametrize("weighted", [False, True])
def test_sorted_row_lengths(ffi, torch_cuda, weighted, merge, mode):
    """merge = 2: two vertices per community, so keys repeat in the rows."""
    torch = torch_cuda
    rng = np.random.default_rng(7 + merge)
    n = 30000 * merge
    deg = np.zeros(n, np.int64)
    deg[: len(ROWS) * merge] = np.repeat(ROWS, merge)
    offs = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    perm = rng.permutation(n // merge)
    comm = np.repeat(perm, merge).astype(np.int32)  # vertices of one community are neighbours in id
    nbr = np.concatenate([rng.permutation(n // merge)[:d] * merge + rng.integers(0, merge, d) for d in deg if d]).astype(np.int32)
    w = rng.integers(1, 50, offs[-1]).astype(np.int32) if weighted else None
    want = _expected(n, offs, nbr, np.ones(offs[-1], np.int64) if w is None else w, comm)
    d = [torch.from_numpy(a).cuda() for a in (offs, nbr)]
    dw = torch.from_numpy(w).cuda() if weighted else None
    dc = torch.from_numpy(comm).cuda()
    out = (torch.zeros(n + 1, dtype=torch.int64, device="cuda"), torch.zeros(offs[-1], dtype=torch.int32, device="cuda"),
           torch.zeros(offs[-1], dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    ctx = ffi.Context(n, offs[-1])
    ctx.set_long_rows(mode)
    C, E = ctx.contract_device(n, d[0].data_ptr(), d[1].data_ptr(), dw.data_ptr() if weighted else None, dc.data_ptr(),
                               *(x.data_ptr() for x in out))
    ctx.close()
    lab, noffs, nnbr, nw = want
    assert (C, E) == (len(noffs) - 1, len(nnbr))
    assert np.array_equal(dc.cpu().numpy(), lab)
    assert np.array_equal(out[0].cpu().numpy()[: C + 1], noffs)
    assert np.array_equal(out[1].cpu().numpy()[:E], nnbr)
    assert np.array_equal(out[2].cpu().numpy()[:E], nw)


@pytest.mark.parametrize("kind", ["unit", "float"])
def test_sorted_levels_give_the_same_run(ffi, torch_cuda, kind):
    if kind == "unit":
        g = ffi.Graph.rmat(15, 400000, seed=3)
    else:
        g = ffi.Graph.lfr(30000, dmin=6, dmax=3000, cmax=4000, seed=4)
    n, e, _ = g.info()
    ctx = ffi.Context(n, e)
    a, b = ctx.louvain(g), ctx.louvain(g, sorted_levels=True)
    ctx.close()
    assert a["iter_q"] == b["iter_q"] and np.array_equal(a["labels"], b["labels"])
