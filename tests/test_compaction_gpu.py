"""Compaction by marks and expansion, at the edges of its steps (32, 128, 1,024
items), its tiles and its chunks (a 1 MB scratch arena), against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = (1, 31, 33, 127, 128, 129, 1023, 1025, 4097, 300_007)


@pytest.fixture(scope="module")
def small_ctx():
    from memory_database_b200 import olapcore
    c = olapcore.Context(0, scratch_bytes=1 << 20)
    yield c
    c.close()


def dev(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def unaligned(x):
    """The same values 4 bytes past a 16-byte boundary."""
    import torch
    t = torch.empty(len(x) + 1, dtype=torch.int32, device="cuda")
    t[1:] = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    return t[1:]


@pytest.mark.parametrize("share", [0.0, 0.002, 0.2, 0.6, 1.0])
@pytest.mark.parametrize("n", SIZES)
def test_select_edges(ctx, n, share):
    from memory_database_b200 import operators as ops
    rng = np.random.default_rng(n)
    col = rng.integers(-1000, 1000, n).astype(np.int32)
    t = int(-1000 + 2000 * share)
    want = np.flatnonzero(col < t)
    rid = rng.permutation(n)[: max(1, n // 2)].astype(np.int32)
    for put in (dev, unaligned):
        d = put(col)
        assert np.array_equal(ops.select_rowids(d, t, ops.CMP_LT, ctx=ctx).cpu().numpy(), want)
        assert np.array_equal(ops.select_rowids(d, t, ops.CMP_LT, in_rowids=put(rid), ctx=ctx).cpu().numpy(),
                              rid[col[rid] < t])
        bits = ops.select_bitmap(d, t, ops.CMP_LT, ctx=ctx).cpu().numpy().view(np.uint8)
        full = np.zeros(32 * ((n + 31) // 32), np.uint8)
        full[want] = 1
        assert np.array_equal(np.unpackbits(bits, bitorder="little"), full)


@pytest.mark.parametrize("cmp_lt", [False, True])
@pytest.mark.parametrize("val", [-2**31, -2**31 + 1, 0, 2**31 - 1])
def test_select_extreme_thresholds(ctx, val, cmp_lt):
    from memory_database_b200 import operators as ops
    col = np.array([-2**31, -2**31 + 1, -1, 0, 1, 2**31 - 1] * 50, np.int32)
    want = np.flatnonzero(col < val if cmp_lt else col <= val)
    got = ops.select_rowids(dev(col), val, ops.CMP_LT if cmp_lt else ops.CMP_LE, ctx=ctx)
    assert np.array_equal(got.cpu().numpy(), want)


def test_select_in_chunks(small_ctx):
    """The marks of 12M rows need more than a 1 MB arena: several chunks."""
    from memory_database_b200 import operators as ops
    rng = np.random.default_rng(3)
    col = rng.integers(0, 1000, 12_000_003).astype(np.int32)
    d = dev(col)
    for t in (0, 30, 999):
        assert np.array_equal(ops.select_rowids(d, t, ctx=small_ctx).cpu().numpy(), np.flatnonzero(col <= t))


@pytest.mark.parametrize("apart", [1, 5, 7, 40])
@pytest.mark.parametrize("k", [1, 5, 1023, 1025, 70_001])
def test_gather_densities(ctx, k, apart):
    """Both gathers (up to 6 rows apart, and farther), ids out of range among them."""
    from memory_database_b200 import operators as ops
    rng = np.random.default_rng(k)
    n = k * apart
    cols = [rng.integers(-2**31, 2**31, n).astype(np.int32) for _ in range(3)]
    ids = np.sort(rng.integers(0, n, k)).astype(np.int32)
    bad = rng.random(k) < 0.1
    ids[bad] = rng.choice([-1, n, 2**31 - 1], bad.sum())
    for put in (dev, unaligned):
        got = ops.gather(put(ids), [dev(c) for c in cols], ctx=ctx)
        for c, g in zip(cols, got):
            assert np.array_equal(g.cpu().numpy(), np.where(bad, 0, c[np.where(bad, 0, ids)]))
        assert ctx.take_range_errors() == bad.sum()
