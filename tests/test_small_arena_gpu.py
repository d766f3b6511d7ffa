"""Row lists far longer than a small arena holds marks for: the context's growing
buffer is used, but not by a graph, which a later growth must not pull it from."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1_100_001, 20_000_003])
def test_lists_in_a_small_arena(n):
    from memory_database_b200 import olapcore, operators as ops
    rng = np.random.default_rng(n)
    col = rng.integers(0, 1000, n).astype(np.int32)
    keys = rng.choice(4000, 1000, replace=False).astype(np.int32)
    pay = rng.integers(-2**31, 2**31, 1000).astype(np.int32)
    table = np.full(4000, -1, np.int64)
    table[keys] = np.arange(1000)
    probe = rng.integers(0, 4000, n).astype(np.int32)
    hit = np.flatnonzero(table[probe] >= 0)
    d = lambda x: torch.from_numpy(x).cuda()  # noqa: E731
    with olapcore.Context(0, scratch_bytes=1 << 20) as c:
        ids = ops.select_rowids(d(col), 500, ctx=c)
        assert np.array_equal(ids.cpu().numpy(), np.flatnonzero(col <= 500))
        assert ops.sel_lt_T_fsel_independent_val_branching(ids.numel(), ids, d(probe), 2000, if_sv=ids, ctx=c) == \
            (both := np.flatnonzero((col <= 500) & (probe <= 2000))).size
        assert np.array_equal(ids[:both.size].cpu().numpy(), both)
        rows, vals = ops.HashTable(1000, ctx=c).build(d(keys), d(pay)).probe_pairs(d(probe))
        assert np.array_equal(rows.cpu().numpy(), hit)
        assert np.array_equal(vals.cpu().numpy(), pay[table[probe[hit]]])


def test_graph_keeps_to_the_arena():
    from memory_database_b200 import olapcore, operators as ops
    from memory_database_b200._lib import CMP_LE, check, lib
    rng = np.random.default_rng(2)
    n = 3_000_001
    ids = rng.permutation(n).astype(np.int32)
    col = rng.integers(0, 1000, n).astype(np.int32)
    want = ids[col[ids] <= 300]
    d_ids, d_col = torch.from_numpy(ids).cuda(), torch.from_numpy(col).cuda()
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    cnt = torch.empty(1, dtype=torch.int64, device="cuda")
    with olapcore.Context(0, scratch_bytes=1 << 20) as c:
        def run():
            c.follow_torch_stream()
            check(lib.olap_select_rowids(c.handle, C.c_void_p(d_col.data_ptr()), n, 300, CMP_LE,
                                         C.c_void_p(d_ids.data_ptr()), n, C.c_void_p(out.data_ptr()),
                                         C.c_void_p(cnt.data_ptr())), c.handle)
        run()  # the buffer exists from here on
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run()
        big = torch.randint(0, 1 << 20, (30_000_000,), dtype=torch.int32, device="cuda")
        ops.group_hash(big, big, max_groups=1 << 20, ctx=c)  # grows the buffer: the old one is freed
        out.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert int(cnt) == want.size and np.array_equal(out[:want.size].cpu().numpy(), want)
        del graph
