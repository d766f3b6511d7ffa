"""Q5 line pass: nation codes for regions of 0 to 64 nations (4-bit ranks up
to 15, nations themselves beyond), supplier vectors in and out of shared
memory, odd sizes and columns that start off a 16-byte boundary, against the
oracle restatement of Q5.cpp:913-978.  Integer sums: equal, not close."""
import numpy as np
import pytest

import oracle
from memory_database_b200 import q5 as Q5

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _tables(rng, supp, lines, nations, in_region, offset=0):
    orders, cust = 40_001, 5_003
    regionkey = np.where(np.arange(nations) % nations < in_region, 1, 0)
    rng.shuffle(regionkey)

    def uni(n, lo, hi):
        return rng.integers(lo, hi + 1, n, dtype=np.int32)

    t = {"r_regionkey": np.arange(2, dtype=np.int32), "n_regionkey": regionkey.astype(np.int32),
         "s_nationkey": uni(supp, -1, nations), "c_nationkey": uni(cust, -2, 70),
         "o_custkey": uni(orders, 0, cust + 1), "o_orderdate": uni(orders, 0, 99),
         "l_orderkey": uni(lines, -1, orders), "l_suppkey": uni(lines, 0, supp + 1),
         "l_price": uni(lines, -5, 10_500_000), "l_discount": uni(lines, 0, 10)}
    for k, v in t.items():
        pad = offset if k.startswith("l_") else 0
        d = torch.empty(len(v) + pad, dtype=torch.int32, device="cuda")[pad:]
        d.copy_(torch.from_numpy(v))
        yield k, v, d


@pytest.mark.parametrize("supp,lines,nations,in_region,offset", [
    (1, 1, 1, 1, 0), (1, 7, 3, 0, 0), (2, 4_099, 25, 5, 0), (777, 100_001, 25, 15, 1), (777, 100_003, 25, 16, 0),
    (1_001, 100_000, 64, 64, 3), (98_303, 60_002, 25, 5, 0), (327_680, 300_001, 25, 5, 0),
    (327_681, 300_001, 25, 5, 0), (400_001, 300_002, 64, 40, 2)])
def test_q5_codes(ctx, supp, lines, nations, in_region, offset):
    rng = np.random.default_rng(supp + lines + in_region)
    rows = list(_tables(rng, supp, lines, nations, in_region, offset))
    host, data = {k: v for k, v, _ in rows}, Q5.Q5Data({k: d for k, _, d in rows})
    exp, errs = oracle.q5(host, 1, 20, 70)
    got = Q5.q5(ctx, data, 1, 20, 70).cpu().numpy()
    assert np.array_equal(got, exp)
    assert ctx.take_range_errors() == errs
    both = Q5.q5_batch(ctx, data, [(1, 20, 70), (0, 0, 50)]).cpu().numpy()
    assert np.array_equal(both[0], exp)
    assert np.array_equal(both[1], oracle.q5(host, 0, 0, 50)[0])
    ctx.take_range_errors()
