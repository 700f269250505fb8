"""The number of rows that an AUTO call recomputes lives on the device from one call to the next: batches that grow (the list of rows moves),
calls recorded into a CUDA graph whose replays come between direct ones.  Every result is that of a net that has seen nothing else."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NETS = [([64, 128, 10], [1, 5]), ([64, 256, 256, 10], [1, 1, 5])]      # layer by layer, and the three-layer kernel


@pytest.fixture(autouse=True)
def margin(spg):
    spg.set_math_mode(spg.abi.MATH_AUTO)
    spg.lib().spingalett_set_auto_margin(0.1)
    yield
    spg.lib().spingalett_set_auto_margin(0.0)


def build(spg, topo, acts):
    net = spg.Network.build(topo, acts, spg.abi.WEIGHT_INITIALIZATION_NONE)
    rng = np.random.default_rng(len(topo))
    net.weights[:] = rng.standard_normal(net.weights.size, dtype=np.float32) / 8
    net.sync_weights()
    return net


def call(spg, net, x, y):
    net.forward_batch_ptr(x.data_ptr(), x.shape[0], y.data_ptr())
    net.synchronize()
    return y[:x.shape[0]].clone(), spg.lib().spingalett_last_repaired(net._h)


@pytest.mark.parametrize("topo,acts", NETS)
def test_batches_that_grow(spg, topo, acts):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(1)
    data = torch.randn(600000, 64, generator=gen, device="cuda")      # a list of 2.4 MB
    y = torch.empty(600000, 10, device="cuda")
    net = build(spg, topo, acts)
    for rows in (600, 5000, 700, 70000, 600000, 5000):
        got, count = call(spg, net, data[:rows], y)
        fresh = build(spg, topo, acts)
        want, expected = call(spg, fresh, data[:rows], y)
        fresh.free()
        assert count == expected > 0 and torch.equal(got, want), (rows, count, expected)
    net.free()


@pytest.mark.parametrize("topo,acts", NETS)
def test_replays_between_direct_calls(spg, topo, acts):
    import torch
    net = build(spg, topo, acts)
    stream = torch.cuda.Stream()
    net.set_stream(stream.cuda_stream)
    x, other = torch.randn(3000, 64, device="cuda"), torch.randn(2000, 64, device="cuda")
    y, z = torch.empty(3000, 10, device="cuda"), torch.empty(3000, 10, device="cuda")
    torch.cuda.synchronize()
    want, expected = call(spg, net, x, y)
    want_other, expected_other = call(spg, net, other, z)
    assert expected != expected_other
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        net.forward_batch_ptr(x.data_ptr(), 3000, y.data_ptr())
    for replays in (0, 1, 2, 0, 3):
        for _ in range(replays):
            y.zero_()
            torch.cuda.synchronize()
            with torch.cuda.stream(stream):
                graph.replay()
            net.synchronize()
            assert torch.equal(y, want)
        got, count = call(spg, net, other, z)
        assert count == expected_other and torch.equal(got, want_other)
    del graph
    net.free()


@pytest.mark.parametrize("topo,acts", NETS)
def test_replays_after_calls_that_list_more_rows(spg, topo, acts):
    """A call is captured when few rows are listed; direct ones of as many rows then list all of them.  What the graph refers to is still there."""
    import torch
    net = build(spg, topo, acts)
    stream = torch.cuda.Stream()
    net.set_stream(stream.cuda_stream)
    x, ties = torch.randn(3000, 64, device="cuda") * 40, torch.zeros(3000, 64, device="cuda")
    y, z = torch.empty(3000, 10, device="cuda"), torch.empty(3000, 10, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):                                         # (the second goes by the first one's count)
        want, few = call(spg, net, x, y)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        net.forward_batch_ptr(x.data_ptr(), 3000, y.data_ptr())
    for _ in range(3):
        _, many = call(spg, net, ties, z)
        assert few < 600 and many == 3000, (few, many)
        keep = [torch.randn(1 << 18, device="cuda") for _ in range(8)]      # (what would lie in memory that was given back)
        y.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            graph.replay()
        net.synchronize()
        assert torch.equal(y, want)
        del keep
    del graph
    net.free()
