"""Static device modularity over row lengths around the kernel's limits (lane
groups of 8, batches of 4, rows over 512 entries go to a whole warp): exact
against the same sums on the host."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n", [1, 2, 5, 33, 4001])
def test_static_modularity_row_lengths(ffi, weighted, n):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(n)
    deg = rng.choice([0, 1, 7, 8, 9, 31, 32, 33, 511, 512, 513, 2000], n) if n > 2 else np.full(n, 3)
    offs = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    nbr = rng.integers(0, n, offs[-1]).astype(np.int32)  # directed entries: the sums need no symmetry
    w = rng.integers(1, 1000, offs[-1]).astype(np.int32) if weighted else np.ones(offs[-1], np.int32)
    comm = rng.integers(0, max(1, n // 7), n).astype(np.int32)
    row = np.repeat(np.arange(n), deg)
    inside = int(w[comm[row] == comm[nbr]].sum())
    m2 = int(w.sum(dtype=np.int64))
    tot = np.zeros(n, dtype=object)
    np.add.at(tot, comm[row], w.astype(object))
    t2 = int(sum(int(t) * int(t) for t in tot))
    c = 1.0 / m2
    q = inside * c - (float(t2 >> 64) * 18446744073709551616.0 + float(t2 & (2 ** 64 - 1))) * c * c
    d = [torch.from_numpy(a).cuda() for a in (offs, nbr, w, comm)]
    torch.cuda.synchronize()
    got = ffi.modularity_device_static(n, d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr() if weighted else None,
                                       d[3].data_ptr())
    assert got == q
