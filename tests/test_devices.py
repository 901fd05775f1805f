"""State that belongs to a device: the opt-in of a kernel for more than 48 KB of
shared memory and its count of resident blocks.  A context finds its own when it
is created, so that one process can use several GPUs."""
import glob
import os
import re

import numpy as np
import pytest

from conftest import PKG

CSRC = os.path.join(PKG, "csrc")


def _functions(text):
    """(name, body) of the functions that start in column 0."""
    for m in re.finditer(r"^[^\s#/}][^;{}]*?(\w+)\([^;{}]*\)\s*\n\{\n(.*?)^\}", text, re.M | re.S):
        yield m.group(1), m.group(2)


def test_opt_ins_are_made_at_context_creation():
    with open(os.path.join(CSRC, "engine.cu")) as f:
        create = dict(_functions(f.read()))["gala_context_create"]
    seen = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        with open(path) as f:
            text = f.read()
        bodies = list(_functions(text))
        users = [(n, b) for n, b in bodies if "cudaFuncSetAttribute" in b or "coop_grid(" in b]
        assert sum(b.count("cudaFuncSetAttribute") for _, b in users) == text.count("cudaFuncSetAttribute"), path
        for name, body in users:
            callers = {name} | {n for n, b in bodies if re.search(r"\b%s\s*(<[^>]*>)?\(" % name, b)}
            assert any(re.search(r"\b%s\(" % c, create) for c in callers), (path, name)
            assert "static" not in body, (path, name)
            seen += 1
    assert seen >= 6


@pytest.mark.gpu
def test_two_devices_in_one_process(ffi):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available() or torch.cuda.device_count() < 2:
        pytest.skip("needs two CUDA devices")
    g = ffi.Graph.sbm(4000, 40, 0.1, 0.002, 2)
    n, e, _ = g.info()
    out = []
    for dev in (0, 1, 0):
        for refine in (False, True):
            ctx = ffi.Context(n, e, device=dev)
            out.append(ctx.louvain(g, refine=refine))
            ctx.close()
    for k in range(2, 6):
        assert np.array_equal(out[k]["labels"], out[k % 2]["labels"])
