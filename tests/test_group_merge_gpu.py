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
