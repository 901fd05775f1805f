"""The first sweep of a level over hub rows (more than 8192 entries) without
their tables: row lengths at the edges of the 4096-entry chunks, hubs that are
neighbours of hubs, a hub with a self-loop, and rows of equal weights (ties go to
the lowest id), against the oracle.  Update mode 2 keeps these sizes on the
separate launches; FP64 gains evaluate the rows' candidates a second time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hubs(degrees, weighted, seed):
    """One hub per degree (the hubs are linked with one another) over a ring of
    leaves; hub 0 lists itself when there is more than one."""
    rng = np.random.default_rng(seed)
    H, leaves = len(degrees), max(degrees) + 10
    n = H + leaves
    pairs = {(a, b) for a in range(H) for b in range(a + 1, H)}
    for h, d in enumerate(degrees):
        own = H - 1 + (1 if h == 0 and H > 1 else 0)  # links to hubs and itself
        for x in rng.choice(leaves, d - own, replace=False):
            pairs.add((h, H + int(x)))
    pairs |= {tuple(sorted((H + i, H + (i + 1) % leaves))) for i in range(leaves)}
    p = np.array(sorted(pairs), dtype=np.int64)
    wt = rng.integers(1, 9, p.shape[0])
    src, dst, w = np.concatenate([p[:, 0], p[:, 1]]), np.concatenate([p[:, 1], p[:, 0]]), np.concatenate([wt, wt])
    if H > 1:
        src, dst, w = np.append(src, 0), np.append(dst, 0), np.append(w, 3)
    order = np.lexsort((dst, src))
    offs = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int64)
    assert list(np.diff(offs)[:H]) == list(degrees)
    return offs, dst[order].astype(np.int32), w[order].astype(np.int32) if weighted else None


@pytest.mark.parametrize("fp64_gains", [False, True])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("degrees", [[8193], [12288, 12289, 8200], [16384, 16385, 20000]])
def test_hub_rows_equal_the_oracle(ffi, oracle, degrees, weighted, fp64_gains):
    """With rows said to be distinct (no tables in the first sweep) and not."""
    import torch
    offs, nbr, w = _hubs(degrees, weighted, len(degrees))
    n = offs.shape[0] - 1
    o = oracle.louvain(offs, nbr, w)
    d = [torch.from_numpy(x).cuda() if x is not None else None for x in (offs, nbr, w)]
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    ctx = ffi.Context(n, offs[-1])
    ctx.set_update_mode(2)
    for distinct in (True, False):
        r = ctx.louvain_device(n, d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr() if weighted else None,
                               out.data_ptr(), fp64_gains=fp64_gains, distinct_rows=distinct)
        assert np.array_equal(out.cpu().numpy(), o["labels"]), distinct
        assert r["iter_q"] == o["iter_q"], distinct
        assert r["level_c"] == o["level_c"], distinct
    ctx.close()


def test_hub_rows_with_float_weights_equal_the_oracle(ffi, oracle):
    """Rows of an LFR graph whose largest are hubs, 64-bit fixed-point weights."""
    g = ffi.Graph.lfr(60000, dmin=24, dmax=20000, cmin=20, cmax=30000, seed=5)
    offs, nbr, _ = g.arrays()
    assert np.diff(offs).max() > 8192
    n, e, _ = g.info()
    ctx = ffi.Context(n, e)
    ctx.set_update_mode(2)
    r = ctx.louvain(g)
    ctx.close()
    o = oracle.louvain_f32(offs, nbr, g.weights_f32(), nthreads=4)
    assert np.array_equal(r["labels"], o["labels"]) and r["iter_q"] == o["iter_q"]
