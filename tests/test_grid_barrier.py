"""Grid barriers that give up.

A cooperative launch runs whole steps of a level with grid barriers in between;
a barrier that waits too long sets an error bit and the blocks leave the kernel.
With a limit of one look the barriers of a grid of over a hundred blocks give
up at once; each of the three kernels (phase 1, contraction, refinement) must
end the call with the status, and the same context must give the oracle's
partition on the next run.
"""
import numpy as np
import pytest

from test_batch import torch_cuda  # noqa: F401


def test_rejects_bad_limits(ffi):
    L = ffi.load()
    assert L.gala_context_set_barrier_polls(None, 0) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", ["phase 1", "contraction", "refinement"])
@pytest.mark.parametrize("kind", ["int", "float"])
def test_barrier_limit_ends_the_call(ffi, oracle, torch_cuda, kernel, kind):  # noqa: F811
    offs, nbr, _ = ffi.Graph.sbm(16000, 100, 0.08, 0.0001, 3).arrays()
    rows = np.repeat(np.arange(16000), np.diff(offs))
    w = 1 + (rows + nbr) % 5
    refine = kernel == "refinement"
    if kind == "float":
        w = (w * 0.3).astype(np.float32)
        g = ffi.Graph.from_csr_f32(offs, nbr, w)
        o = oracle.louvain_f32(offs, nbr, w, nthreads=4, refine=refine)
    else:
        w = w.astype(np.int32)
        g = ffi.Graph.from_csr(offs, nbr, w)
        o = oracle.louvain(offs, nbr, w, refine=refine)
    assert 200000 < offs[-1] <= 1 << 18  # the contraction's limit for one launch
    ctx = ffi.Context(16000, offs[-1])
    if kernel != "phase 1":
        ctx.set_update_mode(2)  # phase 1 in launches of its own
    for bad in (-1, 1 << 31):
        with pytest.raises(ffi.GalaError) as e:
            ctx.set_barrier_polls(bad)
        assert e.value.status == 1
    ctx.set_barrier_polls(1)
    for _ in range(2):
        with pytest.raises(ffi.GalaError) as e:
            ctx.louvain(g, refine=refine)
        assert e.value.status == 7
        assert kernel + ": a grid barrier gave up" in str(e.value)
    ctx.set_barrier_polls(0)
    for mode in (2, 0):
        ctx.set_update_mode(mode)
        r = ctx.louvain(g, refine=refine)
        assert np.array_equal(r["labels"], o["labels"])
        assert r["iter_q"] == o["iter_q"] and r["level_c"] == o["level_c"]
    ctx.close()
