"""Equal best gains in a batch with one CTA per graph.

A vertex with more than 32 entries keeps one best candidate per lane, so a tie
between different weights can sit inside one lane (ids 1 and 33, which share a
lane in every table) while the first winning lane (id 0) has no tie of its own.
All three have the same exact gain numerator; FP64 puts 33 above 0, and the
vertex must go there, as in its single run and the oracle's.
"""
import numpy as np
import pytest

from test_batch import torch_cuda  # noqa: F401


def _tied(deg, ta, tb, n):
    """Vertex n-1 with neighbours 0..deg-1 (weights 2, 2, 1, ..., 3 at id 33),
    whose totals are ta, ta, ..., tb at id 33 (each joined to a vertex of its
    own), in a graph of total weight K (tb - ta): w m2 - K Tot is equal for
    (2, ta) and (3, tb)."""
    k, v = deg + 4, n - 1
    edge = {(u, v): 3 if u == 33 else (2 if u < 2 else 1) for u in range(deg)}
    for u in range(deg):
        edge[(u, deg + u)] = (tb if u == 33 else ta) - edge[(u, v)]
    rest = k * (tb - ta) - 2 * sum(edge.values())
    assert rest > 0 and rest % 2 == 0
    edge[(2 * deg, 2 * deg + 1)] = rest // 2
    a, b = np.array(list(edge), dtype=np.int64).T
    a, b, w = np.concatenate([a, b]), np.concatenate([b, a]), np.array(list(edge.values()) * 2)
    order = np.argsort(a * n + b)
    offs = np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n))]).astype(np.int64)
    return offs, b[order].astype(np.int32), w[order].astype(np.int32)


# vertices over and under 512 (the warps' dense tables), rows of at most and of
# more than 128 entries (hash tables, global tables)
CASES = [(40, 5, 22, 400), (100, 5, 53, 700), (200, 5, 16, 1200)]


@pytest.mark.gpu
@pytest.mark.parametrize("deg,ta,tb,n", CASES)
def test_tie_inside_a_lane_goes_to_fp64(ffi, oracle, torch_cuda, deg, ta, tb, n):  # noqa: F811
    offs, nbr, w = _tied(deg, ta, tb, n)
    k, m2 = deg + 4, int(w.sum())
    assert 2 * m2 - k * ta == 3 * m2 - k * tb > 0
    assert 6.0 - (2.0 * k * tb) * (1.0 / m2) > 4.0 - (2.0 * k * ta) * (1.0 / m2)
    # a threshold between the gains of the first and the second sweep: the
    # partition is the first sweep's
    o = oracle.louvain(offs, nbr, w, min_mod=0.3, max_levels=1)
    assert o["labels"][n - 1] == o["labels"][33] != o["labels"][0]
    g = ffi.Graph.from_csr(offs, nbr, w)
    ctx = ffi.Context(2 * n, 2 * offs[-1])
    single = ctx.louvain(g, min_mod=0.3, max_levels=1)
    r = ctx.louvain_batch([g, g], min_mod=0.3, max_levels=1)
    u = ctx.louvain_batch([g, g], min_mod=0.3, max_levels=1, batch_mode=1)
    full = ctx.louvain_batch([g, g])
    ctx.close()
    assert np.array_equal(single["labels"], o["labels"])
    ofull = oracle.louvain(offs, nbr, w)
    for i in range(2):
        assert np.array_equal(u["labels"][i], o["labels"])
        assert np.array_equal(r["labels"][i], o["labels"])
        assert np.array_equal(full["labels"][i], ofull["labels"])
