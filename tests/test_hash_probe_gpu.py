"""Hash lookups: 32-byte buckets from tables aligned to 32 and to 16 bytes, full
tables (runs over many buckets and past the end), the reserved key among the
probe keys, match lists in chunks, tables on both sides of the filter's line."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dev(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


@pytest.mark.parametrize("scratch", [0, 1 << 20])
@pytest.mark.parametrize("shift", [0, 2])  # 64-bit words past a 32-byte boundary
@pytest.mark.parametrize("nb,cap", [(1, 8), (7, 8), (1000, 1008), (1000, 2000), (30_000, 60_000), (2_200_000, 4_400_000)])
def test_lookups(nb, cap, shift, scratch):
    import torch
    from memory_database_b200 import _lib, olapcore
    L = _lib.lib
    rng = np.random.default_rng(nb + shift)
    space = np.unique(rng.integers(-2**31 + 1, 2**31, 3 * nb + 50).astype(np.int32))
    rng.shuffle(space)
    bk = np.concatenate([space[:nb], space[: nb // 10]])[: cap - 1]  # duplicates: the last row wins
    bp = rng.integers(-2**31, 2**31, len(bk)).astype(np.int32)
    want = dict(zip(bk.tolist(), bp.tolist()))
    pk = rng.choice(np.concatenate([space[: 2 * nb], [-2**31]]), 100_003 if scratch else 20_001).astype(np.int32)
    hit = np.array([int(k) in want for k in pk])
    pay = np.array([want.get(int(k), 0) for k in pk], np.int64)
    with olapcore.Context(0, scratch_bytes=scratch) as c:
        h = c.handle
        c.follow_torch_stream()
        table = torch.empty(cap + 4, dtype=torch.int64, device="cuda")[shift: shift + cap]
        words = int(L.olap_hashjoin_filter_words(len(bk)))
        filt = torch.empty(words, dtype=torch.int64, device="cuda")
        k, p, q = dev(bk), dev(bp), dev(pk)
        _lib.check(L.olap_hashjoin_build_filtered(h, k.data_ptr(), p.data_ptr(), len(bk), table.data_ptr(), cap,
                                                  filt.data_ptr(), words), h)
        for f in (filt.data_ptr(), None):
            s, m = (torch.zeros(1, dtype=torch.int64, device="cuda") for _ in range(2))
            rows, out = (torch.zeros(len(pk), dtype=torch.int32, device="cuda") for _ in range(2))
            _lib.check(L.olap_hashjoin_probe_filtered(h, table.data_ptr(), cap, f, words, q.data_ptr(), len(pk),
                                                      s.data_ptr(), m.data_ptr(), None, None), h)
            assert int(s) == pay.sum() and int(m) == hit.sum()
            _lib.check(L.olap_hashjoin_probe_filtered(h, table.data_ptr(), cap, f, words, q.data_ptr(), len(pk),
                                                      None, m.data_ptr(), rows.data_ptr(), out.data_ptr()), h)
            n = int(m)
            assert np.array_equal(rows[:n].cpu().numpy(), np.flatnonzero(hit))
            assert np.array_equal(out[:n].cpu().numpy(), pay[hit].astype(np.int32))
