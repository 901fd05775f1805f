"""The refinement of a level in one launch and in launches of its own: the line
between them is 2^20 vertices.  The same graph padded with vertices without
entries up to both sides of the line: labels of the graph's vertices equal those
without padding, which equal the oracle's (test_refine.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weights", ["none", "int", "float"])
def test_both_sides_of_the_line_agree(ffi, weights):
    g = ffi.Graph.sbm(3000, 40, 0.15, 0.004, 11)
    offs, nbr, _ = g.arrays()
    n0, e = offs.shape[0] - 1, int(offs[-1])
    rows = np.repeat(np.arange(n0), np.diff(offs))
    w = 1 + (rows + nbr) % 5  # symmetric

    def run(n):
        padded = np.concatenate([offs, np.full(n - n0, e, dtype=np.int64)])
        if weights == "float":
            h = ffi.Graph.from_csr_f32(padded, nbr, (w * 0.75).astype(np.float32))
        else:
            h = ffi.Graph.from_csr(padded, nbr, w.astype(np.int32) if weights == "int" else None)
        ctx = ffi.Context(n, e)
        r = ctx.louvain(h, refine=True)
        ctx.close()
        return r

    base = run(n0)
    assert base["rounds"] > 1
    for n in (1 << 20, (1 << 20) + 1):
        r = run(n)
        assert np.array_equal(r["labels"][:n0], base["labels"]), n
        assert np.array_equal(r["labels"][n0:], base["num_communities"] + np.arange(n - n0)), n
        assert r["iter_q"] == base["iter_q"], n
