"""The column-wise probes: staged (int8 and 4-bit) and L2 dimensions, codes that
4 bits cannot hold, unaligned columns, keys out of range, chunked lists."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NULL, GROUP_NULL = 127, 32767


def schema(rng, n, lens, sele, codes, bad_keys):
    vec, fk = [], []
    for m, p, hi in zip(lens, sele, codes):
        v = rng.integers(-3 if hi > 14 else 0, hi, m).astype(np.int8)
        v[rng.random(m) >= p] = NULL
        vec.append(v)
        k = rng.integers(0, m, n).astype(np.int32)
        if bad_keys:
            at = rng.random(n) < 0.01
            k[at] = rng.choice([-1, m, 2**31 - 1], at.sum())
        fk.append(k)
    return vec, fk


def expected(vec, fk, order, factor, n):
    ok, g = np.ones(n, bool), np.zeros(n, np.int64)
    for t in order:
        ok &= (fk[t] >= 0) & (fk[t] < len(vec[t]))
    live = ok.copy()
    for t, f in zip(order, factor):
        c = vec[t][np.where(ok, fk[t], 0)].astype(np.int64)
        live &= c != NULL
        g += c * f
    return live, g, int((~ok).sum())


@pytest.mark.parametrize("bad_keys", [False, True])
@pytest.mark.parametrize("shape", ["small", "staged", "wide_codes", "late"])
@pytest.mark.parametrize("n", [1, 127, 129, 4099, 2_000_003])
def test_join_cwm(ctx, n, shape, bad_keys):
    import torch
    from memory_database_b200 import olapcore
    rng = np.random.default_rng(n)
    lens = (70_001, 33_000, 40, 3_000_000) if shape != "small" else (50, 7, 40, 900)
    sele = (0.6, 0.5, 1.0 if shape == "late" else 0.7, 0.8)
    codes = (15, 90, 5, 8) if shape == "wide_codes" else (15, 8, 5, 8)
    vec, fk = schema(rng, n, lens, sele, codes, bad_keys)
    order, factor = [3, 0, 2, 1], [1, 11, 170, 850]
    live, g, bad = expected(vec, fk, order, factor, n)
    dv = [torch.from_numpy(v).cuda() for v in vec]
    for shift in (0, 1):  # 16-byte aligned columns and not
        dfk = []
        for k in fk:
            t = torch.empty(n + shift, dtype=torch.int32, device="cuda")
            t[shift:] = torch.from_numpy(k).cuda()
            dfk.append(t[shift:])
        gid = torch.zeros(n, dtype=torch.int16, device="cuda")
        oid = torch.zeros(n, dtype=torch.int64, device="cuda")
        olapcore.join_cwm_sv(dv, dfk, order, 4, gid, factor, n, ctx=ctx)
        assert np.array_equal(gid.cpu().numpy(), np.where(live, g, GROUP_NULL).astype(np.int16))
        assert ctx.take_range_errors() == bad
        k = olapcore.join_cwm_dv(dv, dfk, order, 4, oid, gid, factor, n, ctx=ctx)
        assert k == live.sum() and ctx.take_range_errors() == bad
        assert np.array_equal(oid[:k].cpu().numpy(), np.flatnonzero(live))
        assert np.array_equal(gid[:k].cpu().numpy(), g[live].astype(np.int16))


@pytest.mark.parametrize("nd", [0, 1, 3])
def test_join_cwm_dv_in_chunks(nd):
    """Marks and ids of 1.2M rows in a 1 MB arena: several chunks."""
    import torch
    from memory_database_b200 import olapcore
    n = 1_200_007
    rng = np.random.default_rng(nd)
    vec, fk = schema(rng, n, (500, 40_000, 90, 7), (0.5, 0.9, 0.9, 1.0), (8, 8, 8, 8), False)
    order, factor = [2, 0, 1][:nd], [1, 8, 64][:nd]
    live, g, _ = expected(vec, fk, order, factor, n)
    with olapcore.Context(0, scratch_bytes=1 << 20) as c:
        oid = torch.zeros(n, dtype=torch.int64, device="cuda")
        gid = torch.zeros(n, dtype=torch.int16, device="cuda")
        k = olapcore.join_cwm_dv([torch.from_numpy(v).cuda() for v in vec], [torch.from_numpy(x).cuda() for x in fk],
                                 order, nd, oid, gid, factor, n, ctx=c)
        assert k == live.sum()
        assert np.array_equal(oid[:k].cpu().numpy(), np.flatnonzero(live))
        assert np.array_equal(gid[:k].cpu().numpy(), g[live].astype(np.int16))


@pytest.mark.parametrize("dense", [0.03, 0.5, 1.0])
@pytest.mark.parametrize("n", [1, 9, 2047, 100_003])
def test_agg_cwm(ctx, n, dense):
    """Both aggregations, group ids out of range and OIDs out of range among the entries."""
    import torch
    from memory_database_b200 import olapcore
    rng = np.random.default_rng(n)
    G = 900
    m1, m2 = (rng.integers(-2**31, 2**31, n).astype(np.int32) for _ in range(2))
    gid = np.where(rng.random(n) < dense, rng.integers(0, G, n), GROUP_NULL).astype(np.int16)
    wrong = rng.random(n) < 0.01
    gid[wrong] = rng.choice([-1, G, 32766], wrong.sum())
    ok = (gid >= 0) & (gid < G)
    val = m1.astype(np.int64) + m2
    t = lambda x: torch.from_numpy(x).cuda()  # noqa: E731
    gv = torch.zeros(G, dtype=torch.int64, device="cuda")
    want = np.zeros(G, np.int64)
    np.add.at(want, gid[ok], val[ok])
    assert olapcore.agg_cwm_sv(t(gid), n, t(m1), t(m2), G, group_vector=gv, ctx=ctx) == want.sum()
    assert np.array_equal(gv.cpu().numpy(), want) and ctx.take_range_errors() == wrong.sum()
    rows = np.flatnonzero(gid != GROUP_NULL).astype(np.int64)
    g2 = gid[rows].copy()
    if len(rows) == 0:
        return
    off = rng.random(len(rows)) < 0.02
    rows[off] = rng.choice([-1, n], off.sum())
    ok = (g2 >= 0) & (g2 < G) & ~off
    want = np.zeros(G, np.int64)
    np.add.at(want, g2[ok], val[rows[ok]])
    got = olapcore.agg_cwm_dv(t(rows), t(g2), len(rows), t(m1), t(m2), n, G, group_vector=gv, ctx=ctx)
    assert got == want.sum() and np.array_equal(gv.cpu().numpy(), want)
    assert ctx.take_range_errors() == len(rows) - ok.sum()
