"""Batched queries over fact columns that do not start on a 16-byte boundary:
each of the columns shifted alone, and all of them, against the plain
star-join of each query, directly and through a recorded graph."""
import numpy as np
import pytest

from memory_database_b200 import batch, olapcore

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def shifted(x, by):
    t = torch.empty(len(x) + by, dtype=torch.int32, device="cuda")
    t[by:] = torch.from_numpy(x).cuda()
    return t[by:]


@pytest.mark.parametrize("agg", [olapcore.AGG_M1_PLUS_M2, olapcore.AGG_M2])
@pytest.mark.parametrize("probe", [0, 1])
@pytest.mark.parametrize("n_queries", [1, 2, 3, 16])
@pytest.mark.parametrize("rows", [1, 4, 5, 131, 70_003])
def test_shifted_columns(ctx, rows, probe, agg, n_queries):
    rng = np.random.default_rng(rows)
    sizes, groups = (3000, 500, 800, 60), (5, 5, 4, 7)
    dims = batch.make_dim_tables(ctx, sizes, groups)
    fk = [rng.integers(0, n, rows).astype(np.int32) for n in sizes]
    m1, m2 = (rng.integers(-2**31, 2**31, rows).astype(np.int32) for _ in range(2))
    qs = batch.random_queries(rng, n_queries, rows, groups, sel_range=(0.3, 1.0))
    eng = batch.BatchEngine(ctx, dims)
    try:
        eng.tune(512, 4096, probe)
        for which in ((0,), (3,), (4,), (5,), range(6)):
            off = [(1 + i % 3) if i in which else 0 for i in range(6)]
            f = [shifted(c, o) for c, o in zip(fk, off)]
            a, b = shifted(m1, off[4]), shifted(m2, off[5])
            for use_graph in (False, True):
                out, totals, offs = eng.run(qs, f, a, b, agg=agg, use_graph=use_graph)
                for q, o, t in zip(qs, offs, totals.tolist()):
                    gs, tot = batch.run_plain(ctx, dims, q, f, a, b, agg=agg)
                    assert torch.equal(out[o: o + q.group_nums], gs[0]) and t == int(tot[0])
        assert ctx.take_range_errors() == 0
    finally:
        eng.close()
