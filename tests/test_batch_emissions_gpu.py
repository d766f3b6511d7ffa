"""The batched scan's emissions: lists that overflow (every query passes every
row), factors that 16 bits cannot hold, smallest tables on both sides of the
staging line, group attributes that are no codes, filters at the int32 ends."""
import numpy as np
import pytest

from memory_database_b200 import batch, olapcore

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("probe", [0, 1])
@pytest.mark.parametrize("wide_factor", [False, True])
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("smallest,rows", [(40, 1), (4096, 5003), (4097, 20_001)])
def test_batch_equals_plain(ctx, smallest, rows, dense, wide_factor, probe):
    rng = np.random.default_rng(smallest + rows)
    sizes, groups = (9000, smallest, 5000, 6000), (3, 5, 4, 7)
    d = batch.DimTables(sizes, groups)
    for n, g in zip(sizes, groups):
        f = rng.integers(-2**31, 2**31, n).astype(np.int32)
        f[: n // 8] = rng.choice([-2**31, 2**31 - 1], n // 8)
        c = rng.integers(0, g, n).astype(np.int32)
        c[rng.random(n) < 0.02] = rng.choice([-1, 127, 2**31 - 1])
        d.filt.append(torch.from_numpy(f).cuda())
        d.grp.append(torch.from_numpy(c).cuda())
    fk = [torch.from_numpy(rng.integers(0, n, rows).astype(np.int32)).cuda() for n in sizes]
    m1, m2 = (torch.from_numpy(rng.integers(-2**31, 2**31, rows).astype(np.int32)).cuda() for _ in range(2))
    qs = []
    for q in range(64):
        lo = [-2**31] * 4 if dense else [int(x) for x in rng.integers(-2**31, 0, 4)]
        hi = [2**31 - 1] * 4 if dense else [int(x) for x in rng.integers(0, 2**31, 4)]
        grouped = sorted(rng.choice(4, 2, replace=False).tolist())
        factor = [0, 0, 0, 0]
        factor[grouped[1]] = 1
        factor[grouped[0]] = 70_000 if wide_factor and q % 2 else groups[grouped[1]]
        n_groups = factor[grouped[0]] * (groups[grouped[0]] - 1) + groups[grouped[1]]
        b = int(rng.integers(0, rows))
        qs.append(batch.Query(0 if dense else b, rows, lo, hi, grouped, [0, 1, 2, 3], factor, n_groups))
    eng = batch.BatchEngine(ctx, d, max_queries=64)
    try:
        eng.tune(512, 4096, probe)
        for use_graph in (False, True):
            out, totals, offs = eng.run(qs, fk, m1, m2, use_graph=use_graph)
            ctx.take_range_errors()
            for q, o, t in zip(qs, offs, totals.tolist()):
                gs, tot = batch.run_plain(ctx, d, q, fk, m1, m2)
                assert torch.equal(out[o: o + q.group_nums], gs[0]) and t == int(tot[0])
            ctx.take_range_errors()
    finally:
        eng.close()


def test_largest_accumulators(ctx):
    """The largest shared accumulators the engine accepts still launch."""
    dims = batch.make_dim_tables(ctx, (1000, 500, 800, 60), (5, 5, 4, 7))
    fk = [torch.zeros(1001, dtype=torch.int32, device="cuda") for _ in range(4)]
    m = torch.ones(1001, dtype=torch.int32, device="cuda")
    qs = batch.random_queries(np.random.default_rng(1), 8, 1001, (5, 5, 4, 7), sel_range=(0.5, 1.0))
    eng = batch.BatchEngine(ctx, dims)
    try:
        for block, probe in ((1024, 0), (512, 1)):
            eng.tune(block, 24576, probe)
            out, totals, offs = eng.run(qs, fk, m, m)
            for q, o in zip(qs, offs):
                gs, _ = batch.run_plain(ctx, dims, q, fk, m, m)
                assert torch.equal(out[o: o + q.group_nums], gs[0])
    finally:
        eng.close()
