"""Hash group-by at the edges of its partitioned plan: both table sizes, the
three scatters (long tile, short tile, none), rows around a tile, runs that end
inside a sector, skew, values at the int32 extremes, the reserved key."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(ctx, keys, vals, vals2, max_groups, offset=0):
    import torch
    from memory_database_b200 import operators as ops
    d = lambda x: None if x is None else torch.from_numpy(x).cuda()  # noqa: E731
    k, s, c = ops.group_hash(d(keys), d(vals), d(vals2), key_offset=offset, max_groups=max_groups, ctx=ctx)
    shifted = (keys.astype(np.int64) + offset + 2**31) % 2**32 - 2**31
    ok = shifted != -2**31
    uk, inv, cnt = np.unique(shifted[ok], return_inverse=True, return_counts=True)
    v = vals.astype(np.int64) + (0 if vals2 is None else vals2)
    want = np.zeros(len(uk), np.int64)
    np.add.at(want, inv, v[ok])
    k, s, c = (x.cpu().numpy() for x in (k, s, c))
    order = np.argsort(k)
    assert np.array_equal(k[order], uk)
    assert np.array_equal(s[order], want)
    assert np.array_equal(c[order], cnt)
    assert ctx.take_range_errors() == (~ok).sum()


@pytest.mark.parametrize("two", [False, True])
@pytest.mark.parametrize("max_groups", [400, 300_000, 700_000, 6_000_000, 16_000_000, 30_000_000])
@pytest.mark.parametrize("n", [1, 8191, 8193, 700_003])
def test_partitioned_plans(ctx, n, max_groups, two):
    from memory_database_b200 import _lib
    rng = np.random.default_rng(n + max_groups)
    keys = rng.integers(-2**31 + 1, 2**31, max(1, min(n // 3, max_groups))).astype(np.int32)
    keys = rng.choice(keys, n)
    vals = rng.integers(-2**31, 2**31, n).astype(np.int32)
    vals2 = rng.integers(-2**31, 2**31, n).astype(np.int32) if two else None
    if n > 1:
        keys[n // 2] = -2**31 + 5  # the reserved key once the offset is added
        vals[: n // 4] = 2**31 - 1
        vals[n // 4: n // 2] = -2**31
    ctx.set_tuning(_lib.TUNE_GROUP_PLAN, 2)
    try:
        check(ctx, keys, vals, vals2, max_groups, offset=-5 if n > 1 else 0)
    finally:
        ctx.set_tuning(_lib.TUNE_GROUP_PLAN, 0)


@pytest.mark.parametrize("two", [False, True])
@pytest.mark.parametrize("max_groups", [60_000, 900_000])
def test_split_partitions(ctx, max_groups, two):
    """Four fifths of the rows on three keys: their partitions are split and merged."""
    rng = np.random.default_rng(max_groups)
    n = 3_000_017
    keys = np.where(rng.random(n) < 0.8, rng.integers(0, 3, n), rng.integers(0, max_groups, n)).astype(np.int32)
    vals = rng.integers(-2**31, 2**31, n).astype(np.int32)
    check(ctx, keys, vals, vals[::-1].copy() if two else None, max_groups)


@pytest.mark.parametrize("sign", [-1, 1])
@pytest.mark.parametrize("groups", [3, 4000])
def test_block_tables_at_extremes(ctx, groups, sign):
    """The per-block tables: sums that pass +-2^31 many times over."""
    rng = np.random.default_rng(groups)
    n = 1_000_003
    keys = rng.integers(0, groups, n).astype(np.int32)
    vals = np.full(n, 2**31 - 1 if sign > 0 else -2**31, np.int32)
    vals[::7] = -sign * 12345
    check(ctx, keys, vals, None, groups)
    check(ctx, keys, vals, vals, groups)
