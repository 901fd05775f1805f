"""The first sweep of a level over rows of up to 32 distinct neighbours without
the search for equal labels: every row length from 0 to 36 (the bins end at 4, 8,
16 and 32), self-loops, fewer and more rows than a warp takes, equal weights
(ties go to the lowest id), against the oracle.  Update mode 2 keeps these sizes
on the separate launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(n, weighted, seed):
    """Vertex v has about v mod 37 neighbours, every seventh a self-loop too."""
    rng = np.random.default_rng(seed)
    pairs = set()
    for v in range(n):
        for x in rng.choice(n, min(v % 37, n - 1) // 2, replace=False):
            if x != v:
                pairs.add((min(v, int(x)), max(v, int(x))))
    p = np.array(sorted(pairs), dtype=np.int64).reshape(-1, 2)
    wt = rng.integers(1, 9, p.shape[0])
    loops = np.arange(0, n, 7)
    src = np.concatenate([p[:, 0], p[:, 1], loops])
    dst = np.concatenate([p[:, 1], p[:, 0], loops])
    w = np.concatenate([wt, wt, np.full(loops.shape[0], 5)])
    order = np.lexsort((dst, src))
    offs = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int64)
    return offs, dst[order].astype(np.int32), w[order].astype(np.int32) if weighted else None


@pytest.mark.parametrize("fp64_gains", [False, True])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n", [2, 9, 38, 259, 5003])
def test_first_sweep_equals_the_oracle(ffi, oracle, n, weighted, fp64_gains):
    import torch
    offs, nbr, w = _rows(n, weighted, n)
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
    ctx.close()
