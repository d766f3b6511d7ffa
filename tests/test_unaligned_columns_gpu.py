"""Columns 4 bytes past a 16-byte boundary take loads of their own; their results
equal those of the aligned columns (numpy), at the edges of a step (32, 128) and
of a tile."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def shifted(x):
    import torch
    t = torch.empty(len(x) + 1, dtype=torch.int32, device="cuda")
    t[1:] = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    return t[1:]


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 4095, 1_000_003, 6_000_001])
def test_select_unaligned(ctx, n):
    from memory_database_b200 import operators as ops
    rng = np.random.default_rng(n)
    col = rng.integers(-2**31, 2**31, n).astype(np.int32)
    for t in (-2**31, 0, 2**31 - 1):
        want = col <= t
        assert np.array_equal(ops.select_rowids(shifted(col), t, ctx=ctx).cpu().numpy(), np.flatnonzero(want))
        bits = ops.select_bitmap(shifted(col), t, ctx=ctx).cpu().numpy().view(np.uint8)
        full = np.zeros(32 * ((n + 31) // 32), bool)
        full[:n] = want
        assert np.array_equal(np.unpackbits(bits, bitorder="little").astype(bool), full)


@pytest.mark.parametrize("moved", ["one key column", "output"])
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 1025, 700_001])
def test_column_wise_probes_unaligned(ctx, n, moved):
    import torch
    from memory_database_b200 import olapcore, operators as ops
    rng = np.random.default_rng(n)
    lens, fk = (900, 40, 70_001, 7), []
    vec = [rng.integers(0, 15, m).astype(np.int8) for m in lens]
    for v in vec:
        v[rng.random(len(v)) < 0.3] = 127
    for m in lens:
        k = rng.integers(0, m, n).astype(np.int32)
        bad = rng.random(n) < 0.01
        k[bad] = rng.choice([-1, m], bad.sum())
        fk.append(k)
    ok = np.all([(k >= 0) & (k < m) for k, m in zip(fk, lens)], axis=0)
    codes = [v[np.where(ok, k, 0)].astype(np.int64) for v, k in zip(vec, fk)]
    live = ok & np.all([c != 127 for c in codes], axis=0)
    g = sum(c << s for c, s in zip(codes, (12, 8, 4, 0)))
    dv = [torch.from_numpy(v).cuda() for v in vec]
    dk = [shifted(k) if moved == "one key column" and j == 2 else torch.from_numpy(k).cuda() for j, k in enumerate(fk)]
    pad = 1 if moved == "output" else 0
    out = torch.empty(n + pad, dtype=torch.int32, device="cuda")[pad:]
    assert ops.starjoinalgo_cwm_sv(n, *dv, *dk, out, ctx=ctx) == live.sum()
    assert np.array_equal(out.cpu().numpy(), np.where(live, g, 32767))
    k, pos, grp = ops.starjoinalgo_cwm_dv(n, *dv, *dk, ctx=ctx)
    assert k == live.sum() and np.array_equal(pos.cpu().numpy(), np.flatnonzero(live))
    assert np.array_equal(grp.cpu().numpy(), g[live])
    gid = torch.empty(n + pad, dtype=torch.int16, device="cuda")[pad:]
    olapcore.join_cwm_sv(dv, dk, [0, 1, 2, 3], 4, gid, [1, 2, 3, 4], n, ctx=ctx)
    want = sum(c * f for c, f in zip(codes, (1, 2, 3, 4)))
    assert np.array_equal(gid.cpu().numpy(), np.where(live, want, 32767).astype(np.int16))
    assert ctx.take_range_errors() == 3 * (~ok).sum()


@pytest.mark.parametrize("nd", [0, 1, 3])
@pytest.mark.parametrize("n", [1, 255, 257, (1 << 20) - 1, 1 << 20, (1 << 20) + 1])
def test_vector_of_few_rows(ctx, n, nd):
    """Both sides of the size up to which the vector takes a thread per row."""
    import torch
    from memory_database_b200 import olapcore
    rng = np.random.default_rng(n + nd)
    lens, factor = (900, 40, 70_001)[:nd], [1, 7, 50][:nd]
    vec = [np.where(rng.random(m) < 0.3, 127, rng.integers(-3, 15, m)).astype(np.int8) for m in lens]
    fk = [np.where(rng.random(n) < 0.01, rng.choice([-1, m], n), rng.integers(0, m, n)).astype(np.int32) for m in lens]
    ok, live, g = np.ones(n, bool), np.ones(n, bool), np.zeros(n, np.int64)
    for v, k, f in zip(vec, fk, factor):
        ok &= (k >= 0) & (k < len(v))
    for v, k, f in zip(vec, fk, factor):
        c = v[np.where(ok, k, 0)].astype(np.int64)
        live &= c != 127
        g += c * f
    gid = torch.empty(n, dtype=torch.int16, device="cuda")
    olapcore.join_cwm_sv([torch.from_numpy(v).cuda() for v in vec], [torch.from_numpy(k).cuda() for k in fk],
                         list(range(nd)), nd, gid, factor, n, ctx=ctx)
    assert np.array_equal(gid.cpu().numpy(), np.where(live & ok, g, 32767).astype(np.int16))
    assert ctx.take_range_errors() == (~ok).sum()
