"""One context used from several streams without waiting in between: the calls
share the context's scratch, so each stream's work must follow the last one's."""
import numpy as np
import pytest

import oracle
from memory_database_b200 import q5 as Q5

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

QUERIES = [(0, 0, 1500), (3, 700, 2500), (1, 100, 465)]


@pytest.fixture(scope="module")
def data(ctx):
    d = Q5.make_q5_data(ctx, n_supp=50_000, n_cust=500_000, n_orders=8_000_000, n_lines=40_000_000)
    h = {k: v.cpu().numpy() for k, v in d.cols.items()}
    torch.cuda.synchronize()
    return d, [oracle.q5(h, *q)[0] for q in QUERIES]


def outputs(n):
    return [torch.empty(25, dtype=torch.int64, device="cuda") for _ in range(n)]


def test_streams_in_turn(data):
    from memory_database_b200 import olapcore
    d, want = data
    streams = [torch.cuda.Stream() for _ in range(2)] + [torch.cuda.default_stream()]
    with olapcore.Context(0) as c:
        got = outputs(24)
        torch.cuda.synchronize()
        for i, out in enumerate(got):
            with torch.cuda.stream(streams[i % len(streams)]):
                Q5.q5(c, d, *QUERIES[(i // 2) % 3], out=out)
        torch.cuda.synchronize()
        for i, out in enumerate(got):
            assert np.array_equal(out.cpu().numpy(), want[(i // 2) % 3]), i


def test_capture_between_streams(data):
    """A capture in between runs nothing, so the stream after it follows the one before it."""
    from memory_database_b200 import olapcore
    d, want = data
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with olapcore.Context(0) as c:
        got = outputs(3)
        with torch.cuda.stream(b):
            Q5.q5(c, d, *QUERIES[2], out=got[2])
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            Q5.q5(c, d, *QUERIES[2], out=got[2])
        for _ in range(4):
            with torch.cuda.stream(a):
                Q5.q5(c, d, *QUERIES[0], out=got[0])
            with torch.cuda.stream(b):
                Q5.q5(c, d, *QUERIES[1], out=got[1])
        torch.cuda.synchronize()
        for out, w in zip(got, want):
            assert np.array_equal(out.cpu().numpy(), w)
        for out in got:
            out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(got[2].cpu().numpy(), want[2])
        del graph
