"""The symmetry hash that allows the incremental weight update, summed over
chunks of 1024 entries that begin and end inside rows: one entry without a
mirror, at the edge of a chunk, in a hub's row or next to rows without
entries, has to be seen (no incremental sweep), and without it the graph has to
pass."""
import numpy as np
import pytest

from test_gpu_parity import _sym_graph

pytestmark = pytest.mark.gpu


def _graph(weighted):
    """Rows without entries at the start, between and at the end; one hub row
    over several chunks."""
    offs, nbr, w = _sym_graph(np.random.default_rng(5), 1500, 4000, weighted, hubs=[(700, 6000)])
    n = offs.shape[0] - 1
    new = np.arange(n) + 40 + np.where(np.arange(n) >= 600, 300, 0)  # ids with gaps
    N = n + 40 + 300 + 70
    out = np.zeros(N + 1, dtype=np.int64)
    out[new + 1] = np.diff(offs)
    return np.cumsum(out), new[nbr].astype(np.int32), w


@pytest.mark.parametrize("weighted", [False, True])
def test_symmetric_graph_passes(ffi, weighted):
    offs, nbr, w = _graph(weighted)
    ctx = ffi.Context(offs.shape[0] - 1, offs[-1])
    ctx.set_update_mode(2)
    assert ctx.louvain(ffi.Graph.from_csr(offs, nbr, w))["incremental_sweeps"] > 0
    ctx.close()


@pytest.mark.parametrize("where", ["first", 1023, 1024, 2047, "hub", "last"])
def test_one_entry_without_mirror_is_seen(ffi, where):
    offs, nbr, w = _graph(True)
    hub = int(np.argmax(np.diff(offs)))
    at = {"first": 0, "hub": int(offs[hub]) + 1500, "last": nbr.shape[0] - 1}.get(where, where)
    assert 0 <= at < nbr.shape[0] and offs[hub + 1] - offs[hub] > 1024
    row = int(np.searchsorted(offs, at, side="right")) - 1
    assert row != nbr[at]
    w = w.copy()
    w[at] += 1
    ctx = ffi.Context(offs.shape[0] - 1, offs[-1])
    ctx.set_update_mode(2)
    assert ctx.louvain(ffi.Graph.from_csr(offs, nbr, w))["incremental_sweeps"] == 0
    ctx.close()
