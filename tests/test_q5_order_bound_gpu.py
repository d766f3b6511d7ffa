"""Q5 where the largest int32 order key is the first one past the orders (2^31 - 1
of them: a range error) and where it is the last order (2^31)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_orders", [2**31 - 1, 2**31])
def test_largest_order_key(n_orders):
    import torch
    from memory_database_b200 import olapcore, q5
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    ones = torch.ones(n_orders, dtype=torch.int32, device="cuda")  # every order: customer 1, day 1
    keys = [2**31 - 1, 2**31 - 2, 0, 2**31 - 1, -1, 5, 2**31 - 3, 2**31 - 1, 2**31 - 1, 7, -2**31]
    price = np.arange(1, len(keys) + 1) * 1000
    cols = {"r_regionkey": i32([0]), "n_regionkey": i32([0]), "s_nationkey": i32([0]), "c_nationkey": i32([0]),
            "o_custkey": ones, "o_orderdate": ones, "l_orderkey": i32(keys),
            "l_suppkey": i32([1] * len(keys)), "l_price": i32(price), "l_discount": i32([0] * len(keys))}
    ok = np.array([0 <= k < n_orders for k in keys])
    with olapcore.Context(0, scratch_bytes=n_orders + (1 << 20)) as c:
        got = q5.q5(c, q5.Q5Data(cols), 0, 1, 2)
        assert got.cpu().tolist() == [int(price[ok].sum()) * 100]
        assert c.take_range_errors() == (~ok).sum()
