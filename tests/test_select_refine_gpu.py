"""Refining a selection vector in place (out_rowids == in_rowids): no entry may be
overwritten before it is read, whatever the order the blocks run in."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entry", ["c", "mirror"])
@pytest.mark.parametrize("scratch", [0, 1 << 20])  # one chunk, several
@pytest.mark.parametrize("n", [129, 1025, 1_000_003])
def test_refine_in_place(n, scratch, entry):
    import torch
    from memory_database_b200 import olapcore, operators as ops
    from memory_database_b200._lib import CMP_LE, check, lib
    rng = np.random.default_rng(n)
    a, b = (rng.integers(0, 1000, 2 * n).astype(np.int32) for _ in range(2))
    ids = np.sort(rng.choice(2 * n, n, replace=False)).astype(np.int32)
    want = ids[a[ids] <= 900]
    want = want[b[want] <= 700]
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    with olapcore.Context(0, scratch_bytes=scratch) as c:
        for off in (0, 1):  # 16-byte aligned and not
            sv = torch.empty(n + off, dtype=torch.int32, device="cuda")[off:]
            sv.copy_(torch.from_numpy(ids))
            k = n
            for col, t in ((da, 900), (db, 700)):
                if entry == "mirror":
                    k = ops.sel_lt_T_fsel_independent_val_branching(k, sv, col, t, if_sv=sv, ctx=c)
                    continue
                cnt = torch.empty(1, dtype=torch.int64, device="cuda")
                c.follow_torch_stream()
                check(lib.olap_select_rowids(c.handle, col.data_ptr(), 2 * n, t, CMP_LE, sv.data_ptr(), k,
                                             sv.data_ptr(), cnt.data_ptr()), c.handle)
                k = int(cnt.item())
            assert np.array_equal(sv[:k].cpu().numpy(), want)
