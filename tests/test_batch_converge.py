"""Per-graph convergence of a union run on the device: graph counts at the
edges of its 256-thread blocks, graphs that stop after different numbers of
sweeps, and graphs without entries, against single runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graphs", [False, True])
@pytest.mark.parametrize("count", [1, 31, 255, 256, 257])
def test_union_run_equals_single_runs(ffi, count, use_graphs):
    kinds = [ffi.Graph.sbm(n, k, 0.4, 0.02, 7 + n) for n, k in ((40, 2), (150, 5), (400, 8), (900, 30))]
    kinds.append(ffi.Graph.from_csr(np.zeros(6, dtype=np.int64), np.zeros(0, dtype=np.int32)))
    ctx = ffi.Context(900 * count, max(k.info()[1] for k in kinds) * count)
    one = [ctx.louvain(g) if g.info()[1] else None for g in kinds]
    assert len({len(o["iter_q"]) for o in one if o}) > 1
    pick = np.random.default_rng(count).integers(0, len(kinds), count)
    pick[-1] = 2
    r = ctx.louvain_batch([kinds[k] for k in pick], batch_mode=1, use_graphs=use_graphs)
    for i, k in enumerate(pick):
        if one[k] is None:
            assert r["modularity"][i] == 0.0
            continue
        assert np.array_equal(r["labels"][i], one[k]["labels"]), (i, k)
        assert r["modularity"][i] == one[k]["modularity"]
    ctx.close()
