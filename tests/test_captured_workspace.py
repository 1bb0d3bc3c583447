"""Products whose tiles are cut into K ranges, captured into CUDA graphs: each graph owns the buffers it sums in."""
import pytest
import torch

from codegendemo_b200.kcg.matmul_op import matmul

# fp32 with a remainder cut into ranges, fp32 with a fused bias (every tile goes through the workspace), 16-bit with a
# remainder cut into ranges
CASES = [(3456, 768, 1408, torch.float32, False), (512, 768, 512, torch.float32, True),
         (2688, 2560, 10240, torch.bfloat16, False)]


def _operands(case, seed=1):
    m, n, k, dtype, fused = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    a, b = [torch.rand(s, generator=gen, device="cuda").sub_(0.5).to(dtype) for s in ((m, k), (k, n))]
    return a, b, torch.rand(n, generator=gen, device="cuda").to(dtype) if fused else None


def _capture(ops, c, stream):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        matmul(ops[0], ops[1], c, bias=ops[2])
    return graph


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[:3])))
def test_the_first_call_on_a_stream_may_be_captured(case):
    ops = _operands(case)
    want = matmul(ops[0], ops[1], bias=ops[2])  # (compiles and loads the kernel: another stream's call)
    c = torch.full_like(want, float("nan"))
    graph = _capture(ops, c, torch.cuda.Stream())
    for _ in range(3):
        c.fill_(float("nan"))
        graph.replay()
        assert torch.equal(c, want)


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[:3])))
def test_a_larger_call_later_leaves_a_graph_alone(case):
    ops = _operands(case)
    want = matmul(ops[0], ops[1], bias=ops[2])
    stream = torch.cuda.Stream()
    c = torch.empty_like(want)
    graph = _capture(ops, c, stream)
    big = _operands((4096, 8192, 1024, torch.float32, True))
    with torch.cuda.stream(stream):
        matmul(big[0], big[1], bias=big[2])  # 128 MB of workspace on the stream of the capture
    torch.cuda.synchronize()
    junk = [torch.full((1 << 22,), 7.0, device="cuda") for _ in range(16)]  # what is free now belongs to others
    c.fill_(float("nan"))
    graph.replay()
    assert torch.equal(c, want) and all(bool((j == 7.0).all()) for j in junk)


@pytest.mark.gpu
def test_graphs_of_one_capture_stream_run_side_by_side():
    stream, streams = torch.cuda.Stream(), [torch.cuda.Stream() for _ in CASES]
    ops = [_operands(case, seed=i) for i, case in enumerate(CASES)]
    want = [matmul(a, b, bias=bias) for a, b, bias in ops]
    out = [torch.empty_like(w) for w in want]
    graphs = [_capture(o, c, stream) for o, c in zip(ops, out)]
    for _ in range(20):
        for c in out:
            c.fill_(float("nan"))
        torch.cuda.synchronize()
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(c, w) for c, w in zip(out, want))


@pytest.mark.gpu
def test_buffers_of_graphs_that_are_gone_serve_the_next():
    ops = _operands(CASES[2])
    want = matmul(ops[0], ops[1])
    c = torch.empty_like(want)
    stream = torch.cuda.Stream()
    used = []
    for _ in range(12):
        graph = _capture(ops, c, stream)
        graph.replay()
        torch.cuda.synchronize()
        graph.reset()
        torch.cuda.synchronize()
        used.append(torch.cuda.mem_get_info()[1] - torch.cuda.mem_get_info()[0])
    # A buffer of this product is 18 MB. It comes back when the driver has run the graph's destructor, which may be after
    # the next capture has begun: two or three take turns then, but not one for each of twelve graphs.
    assert used[-1] - used[0] <= 60 << 20, used
    assert torch.equal(c, want)
