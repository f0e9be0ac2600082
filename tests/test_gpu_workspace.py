"""Workspaces of eager and captured launches: whose memory a launch uses, and for how long it stays right."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SPLIT = (512, 14336, 3072, 8)  # K split over CTA pairs: counters and partial sums in the workspace


@pytest.fixture(scope="module")
def d(b200_lib):
    import dexter_labs_b200

    assert b200_lib.dxb_scratch_bytes(SPLIT[0], SPLIT[2], SPLIT[1], SPLIT[3], 0) > 0
    return dexter_labs_b200


def problem(d, m, k, n, bits, seed=0):
    torch.manual_seed(seed)
    x = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    w = (torch.randn(n, k, device="cuda") * 0.02).to(torch.bfloat16)
    return x, d.quantize(w, bits=bits, symmetric=True)


def call(d, x, q):
    return (d.w4a16 if q.bits == 4 else d.w8a16)(x, q.qweight, q.scales, q.zeros, None, q.group_size)


def capture(d, x, q, stream):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        y = call(d, x, q)
    return graph, y


@pytest.mark.parametrize("warm", [True, False])
def test_graphs_captured_on_one_stream_run_side_by_side(warm, d):
    x, q = problem(d, *SPLIT)
    xs = [x, x.roll(1, 0), x.roll(2, 0)]
    want = [call(d, v, q) for v in xs]
    stream, others = torch.cuda.Stream(), [torch.cuda.Stream() for _ in range(3)]
    if warm:
        with torch.cuda.stream(stream):
            call(d, x, q)
    graphs = [capture(d, v, q, stream) for v in xs]
    for _ in range(20):
        for _, y in graphs:
            y.zero_()
        torch.cuda.synchronize()
        for (graph, _), s in zip(graphs, others):
            with torch.cuda.stream(s):
                graph.replay()
        with torch.cuda.stream(stream):
            eager = call(d, x, q)
        torch.cuda.synchronize()
        assert all(torch.equal(y, w) for (_, y), w in zip(graphs, want)) and torch.equal(eager, want[0])
    with torch.cuda.stream(stream):
        assert d.ops.last_status() == 0


@pytest.mark.parametrize("shape", [SPLIT, (83, 3072, 3072, 8)])
def test_a_graph_keeps_its_scratch_when_a_larger_call_comes(shape, d):
    x, q = problem(d, *shape)
    big = problem(d, 512, 14336, 3200, 8, seed=1)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        want = call(d, x, q)
        graph, y = capture(d, x, q, stream)
        call(d, *big)  # wants more scratch than the stream has
        # whatever was given back is taken again
        fill = [torch.full((size,), 0x5A, dtype=torch.uint8, device="cuda")
                for size in (1 << 20, 66 << 10, 16 << 20, 19 << 20, 24 << 20, 32 << 20) for _ in range(8)]
        for _ in range(3):
            y.zero_()
            graph.replay()
            assert torch.equal(y, want)
        assert all(bool((f == 0x5A).all()) for f in fill)
        assert d.ops.last_status() == 0


def test_eager_calls_after_a_capture_that_never_ran(d):
    x, q = problem(d, *SPLIT)
    want = call(d, x, q)
    stream = torch.cuda.Stream()
    dirty = torch.full((64 << 20,), 0xA5, dtype=torch.uint8, device="cuda")
    graph, y = capture(d, x, q, stream)  # nothing has run on this stream before
    del dirty
    with torch.cuda.stream(stream):
        assert torch.equal(call(d, x, q), want)
        graph.replay()
        assert torch.equal(y, want)
        assert d.ops.last_status() == 0


def test_a_capture_on_a_fresh_stream_adds_nothing_to_a_small_graph(d):
    # no scratch, no block yet: the library's own block serves, without a node that makes one ready
    x, q = problem(d, 83, 1024, 1024, 8)
    want = call(d, x, q)
    stream = torch.cuda.ExternalStream(torch.cuda.Stream().cuda_stream)
    key = (torch.cuda.current_device(), stream.cuda_stream)
    block, _ = d.ops._blocks.pop(key, None), d.ops._captured.pop(key, None)
    try:
        graph, y = capture(d, x, q, stream)
        assert key not in d.ops._captured and key not in d.ops._blocks
        with torch.cuda.stream(stream):
            graph.replay()
            assert torch.equal(y, want) and d.ops.last_status() == 0
    finally:
        if block is not None:  # (streams come from a pool: an earlier test may have used this one)
            d.ops._blocks[key] = block


def test_status_of_scratch_reaches_the_streams_status_word(d):
    x, q = problem(d, *SPLIT)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        want = call(d, x, q)
        key = (torch.cuda.current_device(), stream.cuda_stream)
        d.ops._scratch[key][0][256:260].view(torch.int32).fill_(0x8000)  # the finisher's wait runs out
        if d.ops._CHECK:  # every call reads the word and clears it
            with pytest.raises(RuntimeError, match="TIMEOUT"):
                call(d, x, q)
        else:
            call(d, x, q)
            assert d.ops.last_status() == -8
            d.ops._blocks[key][0].zero_()
        assert torch.equal(call(d, x, q), want) and d.ops.last_status() == 0
