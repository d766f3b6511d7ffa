"""Merging the slices of a split partition: all rows in one partition whose shared
tables are nearly full, so that runs of full buckets cross the ends of the merging
blocks' shares, and one or two keys with most of the rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def mix32(x):
    x = x.astype(np.uint32)
    x ^= x >> np.uint32(16)
    x *= np.uint32(0x7feb352d)
    x ^= x >> np.uint32(15)
    x *= np.uint32(0x846ca68b)
    return x ^ (x >> np.uint32(16))


def check(ctx, keys, vals, vals2, max_groups):
    import torch
    from memory_database_b200 import operators as ops
    d = lambda x: None if x is None else torch.from_numpy(x).cuda()  # noqa: E731
    k, s, c = (x.cpu().numpy() for x in ops.group_hash(d(keys), d(vals), d(vals2), max_groups=max_groups, ctx=ctx))
    uk, inv, cnt = np.unique(keys, return_inverse=True, return_counts=True)
    want = np.zeros(len(uk), np.int64)
    np.add.at(want, inv, vals.astype(np.int64) + (0 if vals2 is None else vals2))
    order = np.argsort(k)
    assert np.array_equal(k[order], uk) and np.array_equal(s[order], want) and np.array_equal(c[order], cnt)


@pytest.mark.parametrize("two", [False, True])
@pytest.mark.parametrize("distinct", [3000, 9000, 13_000])
def test_full_tables(ctx, distinct, two):
    import torch
    rng = np.random.default_rng(distinct)
    parts = 3 * torch.cuda.get_device_properties(0).multi_processor_count  # of 14,336-slot tables at 2^21 slots
    cand = np.unique(rng.integers(-2**31 + 1, 2**31, 8_000_000).astype(np.int32))
    cand = cand[(mix32(cand).astype(np.uint64) * np.uint64(parts)) >> np.uint64(32) == 5]
    assert len(cand) > 13_000
    n = 400_003
    keys = rng.choice(cand[:distinct], n)
    vals = rng.integers(-2**31, 2**31, n).astype(np.int32)
    check(ctx, keys, vals, vals[::-1].copy() if two else None, 900_000)


@pytest.mark.parametrize("hot", [1, 2])
@pytest.mark.parametrize("max_groups", [60_000, 900_000])
def test_hot_keys(ctx, max_groups, hot):
    rng = np.random.default_rng(max_groups + hot)
    n = 6_000_001
    keys = np.where(rng.random(n) < 0.97, rng.integers(0, hot, n), rng.integers(0, max_groups, n)).astype(np.int32)
    vals = rng.integers(-2**31, 2**31, n).astype(np.int32)
    check(ctx, keys, vals, None, max_groups)


@pytest.mark.parametrize("share", [0.5, 1.0])
def test_large_capacity_filled(ctx, share):
    """More partitions than the tiled scatter keeps: as many distinct keys as asked for, and as the outputs hold."""
    import torch
    from memory_database_b200 import operators as ops
    n = int((1 << 26) * share)
    keys = torch.arange(n, dtype=torch.int32, device="cuda") * 63  # distinct modulo 2^32
    keys = torch.where(keys == -2**31, torch.full_like(keys, -63), keys)  # the reserved key
    k, s, c = ops.group_hash(keys, keys, max_groups=1 << 25, ctx=ctx)
    want = torch.sort(torch.unique(keys))[0]
    order = torch.argsort(k)
    assert torch.equal(k[order], want)
    assert int(c.sum()) == n and int(s.sum()) == int(keys.sum(dtype=torch.int64))
    once = c[order] == 1
    assert torch.equal(s[order][once], want[once].long())
