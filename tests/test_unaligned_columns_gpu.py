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
