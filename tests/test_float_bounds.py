"""Float-weight decisions settled by FP32 bounds must equal the FP64 ones.

The decide and prune kernels of 64-bit fixed-point graphs take a decision from
FP32 bounds when these exclude every other outcome and from the FP64
expressions otherwise.  The graphs here put candidates at or next to equality
(equal weights, weights one FP32 step apart) and over a wide range, in every
degree bin up to hub rows: labels and every iteration's modularity must equal
the oracle's (FP64 throughout), bit for bit.
"""
import numpy as np
import pytest

from test_gpu_parity import _sym_graph

WEIGHTS = {
    "equal": lambda h: np.ones(h.size),
    "one_step_apart": lambda h: 1.0 + (h % 3) * 2.0 ** -23,
    "few_values": lambda h: np.array([0.5, 1.0, 3.0])[h % 3],
    "wide_range": lambda h: 2.0 ** ((h % 25).astype(np.float64) - 10),
}


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.cuda.init()
    return torch


@pytest.mark.gpu
@pytest.mark.parametrize("kind", sorted(WEIGHTS))
@pytest.mark.parametrize("n,m", [(600, 1500), (20000, 110000)])
def test_gpu_float_decisions_match_oracle(ffi, oracle, torch_cuda, kind, n, m):
    hubs = [(3, 13000), (77, 9000), (500, 5000), (501, 1500), (502, 600), (503, 200), (504, 100)] if n > 600 else ()
    rng = np.random.default_rng(n + m)
    offs, nbr, _ = _sym_graph(rng, n, m, False, hubs=hubs)
    row = np.repeat(np.arange(n, dtype=np.int64), np.diff(offs))
    lo, hi = np.minimum(row, nbr), np.maximum(row, nbr)
    h = ((lo * 2654435761 + hi * 40503) >> 7) & 0xFFFFFF  # the same for an entry and its mirror
    wf = WEIGHTS[kind](h).astype(np.float32)
    ctx = ffi.Context(n, offs[-1])
    r = ctx.louvain(ffi.Graph.from_csr_f32(offs, nbr, wf))
    ctx.close()
    o = oracle.louvain_f32(offs, nbr, wf, nthreads=4)
    assert np.array_equal(r["labels"], o["labels"])
    assert r["iter_q"] == o["iter_q"]
