"""Device memory of a context per graph entry: two level graphs (4 bytes of ids and
8 of weights each), the contraction's two streams (12 each), 32 bytes of table
pool, and chunk lists of under 0.1 byte."""
import pytest

from test_batch import torch_cuda  # noqa: F401


@pytest.mark.gpu
def test_bytes_per_entry(ffi, torch_cuda):  # noqa: F811
    cuda = torch_cuda.cuda
    ffi.Context(1000, 1000).close()  # one-time allocations of the library
    used = []
    for entries in (1 << 26, 1 << 27):
        free = cuda.mem_get_info()[0]
        ctx = ffi.Context(1000, entries)
        used.append(free - cuda.mem_get_info()[0])
        ctx.close()
    # allocations are rounded up to 2 MB, some ten of them
    assert used[1] - used[0] <= 80.1 * (1 << 26) + (64 << 20), used
