"""The star-join scan where the share of surviving rows changes along the table,
so that warps go back and forth between reading the measures with the keys and
reading them late, with ragged ends, keys out of range and both accumulators."""
import numpy as np
import pytest

from memory_database_b200 import olapcore
from memory_database_b200.olapcore import AGG_COUNT, AGG_M1, AGG_M1_PLUS_M2, AGG_M1_TIMES_M2, AGG_M2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("aggs", [(AGG_M1_PLUS_M2,), (AGG_M1, AGG_M1_TIMES_M2), (AGG_M2, AGG_COUNT)])
@pytest.mark.parametrize("groups", [(3, 4), (120, 110)])
@pytest.mark.parametrize("n", [1, 130, 40_003, 3_000_001])
def test_changing_selectivity(ctx, n, groups, aggs):
    rng = np.random.default_rng(n)
    lens = (60_000, 900)
    vec = [rng.integers(0, g, m).astype(np.int8) for g, m in zip(groups, lens)]
    vec[0][: lens[0] // 2] = 127  # keys of the lower half are filtered
    vec[1][rng.random(lens[1]) < 0.3] = 127
    # phases of rows: nearly all filtered, nearly none, a few per warp
    phase = (np.arange(n) // 20_011) % 3
    upper = np.where(phase == 0, rng.random(n) < 0.002, np.where(phase == 1, True, rng.random(n) < 0.05))
    fk = [(rng.integers(0, lens[0] // 2, n) + upper * (lens[0] // 2)).astype(np.int32),
          rng.integers(0, lens[1], n).astype(np.int32)]
    at = rng.random(n) < 0.001
    fk[1][at] = rng.choice([-1, lens[1]], at.sum())
    m1, m2 = (rng.integers(-2**31, 2**31, n).astype(np.int32) for _ in range(2))
    G = groups[0] * groups[1]
    ok = [(k >= 0) & (k < m) for k, m in zip(fk, lens)]
    code = [v[np.where(o, k, 0)].astype(np.int64) for v, k, o in zip(vec, fk, ok)]
    live = ok[0] & ok[1] & (code[0] != 127) & (code[1] != 127)
    null = (ok[0] & (code[0] == 127)) | (ok[1] & (code[1] == 127))
    g = code[0] * groups[1] + code[1]
    val = {AGG_M1_PLUS_M2: m1.astype(np.int64) + m2, AGG_M1: m1.astype(np.int64), AGG_M2: m2.astype(np.int64),
           AGG_M1_TIMES_M2: m1.astype(np.int64) * m2, AGG_COUNT: np.ones(n, np.int64)}
    d = lambda x: torch.from_numpy(x).cuda()  # noqa: E731
    for first in (0, min(5, n)):  # from the column's start and off the 16-byte phase
        gs, tot = olapcore.starjoin_groupsum([d(v) for v in vec], [d(k) for k in fk], [groups[1], 1], d(m1), d(m2), G,
                                             aggs=aggs, row_range=(first, n), ctx=ctx)
        sel = live & (np.arange(n) >= first)
        for a, agg in enumerate(aggs):
            want = np.zeros(G, np.int64)
            np.add.at(want, g[sel], val[agg][sel])
            assert np.array_equal(gs[a].cpu().numpy(), want)
            assert int(tot[a]) == int(want.sum())
        assert ctx.take_range_errors() == (~(ok[0] & ok[1]) & ~null & (np.arange(n) >= first)).sum()
