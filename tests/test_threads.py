"""Contexts on several host threads at once.  Their small levels launch cooperative
grids that each fill the GPU; the grids take turns, and every run gives what it
gives alone.  One thread runs on a stream of higher priority, one runs batches."""
import threading

import numpy as np
import pytest

from test_batch import torch_cuda  # noqa: F401
from test_small_tuning import _planted


@pytest.mark.gpu
@pytest.mark.parametrize("refine", [False, True])
def test_runs_on_several_threads(ffi, torch_cuda, refine):  # noqa: F811
    graphs = []
    for k, (n, deg) in enumerate([(30000, 100), (60000, 24), (4000, 12), (9000, 300)]):
        offs, nbr = _planted(n, deg, 300, 20 + k)
        if k == 1:
            graphs.append(ffi.Graph.from_csr_f32(offs, nbr, np.full(nbr.shape[0], 0.5, dtype=np.float32)))
        else:
            graphs.append(ffi.Graph.from_csr(offs, nbr, None))
    ctxs = [ffi.Context(*g.info()[:2]) for g in graphs]
    small = ffi.Graph.sbm_batch(60, n_min=100, n_max=3000, seed=3)
    bctx = ffi.Context(sum(g.info()[0] for g in small), sum(g.info()[1] for g in small))
    stream = torch_cuda.cuda.Stream(priority=-5)
    ctxs[2].set_stream(stream.cuda_stream)
    want = [c.louvain(g, refine=refine) for c, g in zip(ctxs, graphs)]
    bwant = bctx.louvain_batch(small)
    bad = []
    start = threading.Barrier(5)

    def run(i):
        try:
            start.wait()
            for _ in range(25):
                r = ctxs[i].louvain(graphs[i], refine=refine)
                if not np.array_equal(r["labels"], want[i]["labels"]) or r["iter_q"] != want[i]["iter_q"]:
                    bad.append(i)
        except Exception as e:  # noqa: BLE001
            bad.append((i, e))

    def batches():
        try:
            start.wait()
            for k in range(25):
                r = bctx.louvain_batch(small, batch_mode=k & 1)
                if any(not np.array_equal(a, b) for a, b in zip(r["labels"], bwant["labels"])):
                    bad.append("batch")
        except Exception as e:  # noqa: BLE001
            bad.append(("batch", e))

    threads = [threading.Thread(target=run, args=(i,)) for i in range(4)] + [threading.Thread(target=batches)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
    for c in ctxs + [bctx]:
        c.close()
