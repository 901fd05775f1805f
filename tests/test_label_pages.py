"""Labels written to a caller's buffer whose pages are mapped while the run goes
on: sizes around the line (2^18 vertices, 1 MB) from which a thread does it,
buffers that don't begin on a page, and memory around the buffer left alone."""
import ctypes
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1 << 18) - 1, 1 << 18, 300007])
@pytest.mark.parametrize("shift", [0, 1, 1021])
def test_labels_in_a_fresh_unaligned_buffer(ffi, n, shift):
    """Pairs, the last vertex alone if n is odd: labels equal those of a buffer
    that was written before."""
    nbr = (np.arange(n & ~1) ^ 1).astype(np.int32)
    offs = np.minimum(np.arange(n + 1, dtype=np.int64), nbr.shape[0])
    g = ffi.Graph.from_csr(offs, nbr)
    ctx = ffi.Context(n, int(offs[-1]))
    want = ctx.louvain(g)["labels"]
    buf = np.frombuffer(mmap.mmap(-1, (n + shift + 64) * 4), dtype=np.int32)  # pages not there yet
    out = buf[shift:shift + n]
    o = ffi.default_options()
    r = ffi.Result()
    ptr = out.ctypes.data_as(ctypes.POINTER(ctypes.c_int32))
    assert ffi.load().gala_louvain(ctx.h, g.h, ctypes.byref(o), ptr, ctypes.byref(r)) == 0
    assert np.array_equal(out, want)
    assert not buf[:shift].any() and not buf[shift + n:].any()
    ctx.close()
