"""A captured call keeps its scratch to itself: eager calls, other captures and other streams may come and go between the
capture and its replays, and graphs may be replayed beside one another."""
import gc

import pytest

from boostr_b200 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ops():
    from boostr_b200 import ops as o

    return o


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _steps(ops, gen):
    """Calls whose scratch is some tens of KB: few rows, a prompt cut along K, a feed-forward block."""
    w = synth.device_weight("Q4_K", 512, 1024, gen)
    q2 = synth.device_weight("Q2_K", 256, 512, gen)
    g, u, d = (synth.device_weight("Q4_K", 512, 256, gen), synth.device_weight("Q4_K", 512, 256, gen), synth.device_weight("Q6_K", 256, 512, gen))
    x5, x20, x70 = (torch.randn(m, k, device="cuda", generator=gen) for m, k in ((5, 1024), (20, 512), (70, 256)))
    nw = torch.ones(1024, device="cuda")
    return [lambda: ops.quant_matmul(x5, w), lambda: ops.quant_matmul(x20, q2), lambda: ops.quant_mlp(x70, g, u, d),
            lambda: ops.rmsnorm_quant_matmul_batch(x5, nw, 1e-5, [w, w])[1],
            # a misaligned activation takes the Python form of the operator
            lambda: ops.quant_matmul(torch.cat([x5.view(-1)[:1], x5.view(-1)])[1:].view(5, 1024), w)]


def test_replay_after_the_stream_s_scratch_has_grown(ops):
    gen = _gen(1)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    big_x, big_w = torch.randn(300, 4096, device="cuda", generator=gen), synth.device_weight("Q4_K", 256, 4096, gen)
    big_cat = torch.randn(300 * 4096 + 1, device="cuda", generator=gen)[1:].view(300, 4096)
    for step in _steps(ops, gen):
        with torch.cuda.stream(stream):
            want = step().clone()  # makes the stream's eager scratch
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            got = step()
        with torch.cuda.stream(stream):
            ops.quant_matmul(big_x, big_w)  # a larger one takes its place ...
            ops.quant_matmul(big_cat, big_w)
            others = [torch.full((1 << 20,), 7, dtype=torch.uint8, device="cuda") for _ in range(4)]  # ... and its memory goes to these
        torch.cuda.synchronize()
        got.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)
        assert all(bool((o == 7).all()) for o in others), "a replay wrote over other tensors"
        ops.check_device_status()


def test_graphs_replayed_beside_one_another(ops):
    gen = _gen(2)
    w = synth.device_weight("Q4_K", 512, 1024, gen)  # a few CTAs a launch: the graphs really run side by side
    graphs, got, want = [], [], []
    for _ in range(3):
        x = torch.randn(12, 1024, device="cuda", generator=gen)
        want.append(ops.quant_matmul(x, w))
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for _ in range(60):
                y = ops.quant_matmul(x, w)
        graphs.append((g, x))
        got.append(y)
    streams = [torch.cuda.Stream() for _ in graphs]
    torch.cuda.synchronize()
    for _ in range(30):
        for y in got:
            y.zero_()
        torch.cuda.synchronize()
        for (g, _), s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    ops.check_device_status()


def test_graph_outlives_the_graphs_captured_before_it(ops):
    gen = _gen(3)
    w = synth.device_weight("Q4_K", 1024, 1024, gen)

    def capture(rows):
        x = torch.randn(rows, 1024, device="cuda", generator=gen)
        want = ops.quant_matmul(x, w)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            y = ops.quant_matmul(x, w)
        return g, x, y, want

    first, second = capture(10), capture(12)
    del first
    gc.collect()
    torch.cuda.empty_cache()
    third = capture(700)
    for g, _, y, want in (second, third):
        y.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)
    ops.check_device_status()
