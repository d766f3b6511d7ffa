"""olap_starjoin_launch_count against the kernels that the call launches: empty
columns, unaligned columns and the plans with prepasses."""
import numpy as np
import pytest

from memory_database_b200 import _lib, olapcore

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [0, 1, 5001])
@pytest.mark.parametrize("knobs", [{}, {_lib.TUNE_SMEM_DIM_BYTES: 1, _lib.TUNE_SMEM_NIB_BYTES: 200 * 1024},
                                   {_lib.TUNE_SMEM_DIM_BYTES: 1, _lib.TUNE_PROBE_BITS: 1}])
@pytest.mark.parametrize("shift", [0, 1])
def test_counts_the_launches(ctx, n, knobs, shift):
    from torch.profiler import ProfilerActivity, profile
    rng = np.random.default_rng(1)
    dims = [torch.from_numpy(rng.integers(0, 8, m).astype(np.int8)).cuda() for m in (500, 3000)]
    col = lambda hi: torch.from_numpy(rng.integers(0, hi, n + 4).astype(np.int32)).cuda()[shift:shift + n]  # noqa: E731
    fks, m1, m2 = [col(500), col(3000)], col(100), col(100)
    out = torch.empty((1, 64), dtype=torch.int64, device="cuda")
    tot = torch.empty(1, dtype=torch.int64, device="cuda")
    args = (dims, fks, [8, 1], m1, m2, 64)
    try:
        for k, v in knobs.items():
            ctx.set_tuning(k, v)
        said = olapcore.launch_count(*args, ctx=ctx)
        run = lambda: olapcore.starjoin_groupsum(*args, ctx=ctx, out=out, totals_out=tot)  # noqa: E731
        run()
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            run()
            torch.cuda.synchronize()
        seen = sum(e.count for e in p.key_averages() if "olap::" in e.key)
        assert said == seen == (2 + (2 if knobs else 0) if n else 1)
    finally:
        for k in knobs:
            ctx.set_tuning(k, 0)
