"""A caller's stream with part of the GPU (a green context's): the one-launch phase 1,
contraction and refinement fit their grids to it and give the same results."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_batch import torch_cuda  # noqa: F401
from test_small_tuning import _planted

SOURCE = r"""
#include <cuda.h>
void *partition_stream(int sms)
{
    CUdevice d;
    CUdevResource all, part;
    CUdevResourceDesc desc;
    CUgreenCtx g;
    CUstream s;
    unsigned groups = 1;
    if (cuInit(0) || cuDeviceGet(&d, 0) || cuDeviceGetDevResource(d, &all, CU_DEV_RESOURCE_TYPE_SM) ||
        cuDevSmResourceSplitByCount(&part, &groups, &all, 0, 0, sms) || cuDevResourceGenerateDesc(&desc, &part, 1) ||
        cuGreenCtxCreate(&g, desc, d, CU_GREEN_CTX_DEFAULT_STREAM) ||
        cuGreenCtxStreamCreate(&s, g, CU_STREAM_NON_BLOCKING, 0))
        return 0;
    return s;
}
"""


@pytest.fixture(scope="module")
def stream(torch_cuda, tmp_path_factory):  # noqa: F811
    d = tmp_path_factory.mktemp("green")
    src, lib = d / "green.c", d / "green.so"
    src.write_text(SOURCE)
    home = os.path.dirname(os.path.dirname(os.path.realpath(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")))
    r = subprocess.run(["gcc", "-shared", "-fPIC", "-I", home + "/include", "-o", str(lib), str(src), "-L",
                        home + "/lib64/stubs", "-lcuda"], capture_output=True, text=True)
    if r.returncode:
        pytest.skip("no green contexts in this toolkit: " + r.stderr[-200:])
    f = ctypes.CDLL(str(lib)).partition_stream
    f.restype = ctypes.c_void_p
    s = f(16)
    if not s:
        pytest.skip("no green contexts on this device")
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["int", "float"])
@pytest.mark.parametrize("refine", [False, True])
def test_runs_on_part_of_the_gpu(ffi, torch_cuda, stream, kind, refine):  # noqa: F811
    for n, deg in ((40000, 40), (16000, 14)):
        offs, nbr = _planted(n, deg, 300, deg)
        g = (ffi.Graph.from_csr(offs, nbr, None) if kind == "int" else
             ffi.Graph.from_csr_f32(offs, nbr, np.full(nbr.shape[0], 0.5, dtype=np.float32)))
        ctx = ffi.Context(n, offs[-1])
        want = ctx.louvain(g, refine=refine)
        for mode in (0, 2):  # 2: phase 1 in launches of its own, the contraction in one
            ctx.set_update_mode(mode)
            ctx.set_stream(stream)
            r = ctx.louvain(g, refine=refine)
            ctx.set_stream(None)
            assert np.array_equal(r["labels"], want["labels"]) and r["iter_q"] == want["iter_q"]
        ctx.close()
