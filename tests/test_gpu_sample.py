"""forward() of small nets: launches replayed as a graph from the third call on, answers taken from page-locked memory as they arrive.  Whatever comes between
the calls, every one of them answers its own input, in every layer."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def layers(net):
    """All layers' outputs of the last forward(), from the net's own array."""
    total = sum(net.topology)
    return np.ctypeslib.as_array(net._h.contents.neurons, shape=(total,)).copy()[net.topology[0]:]


def want(net, x, acts):
    out, w_at, b_at, a = [], 0, 0, x.astype(np.float64)
    for i, o, act in zip(net.topology, net.topology[1:], acts):
        z = net.weights[w_at:w_at + i * o].reshape(o, i).astype(np.float64) @ a + net.biases[b_at:b_at + o]
        a = np.maximum(z, 0) if act == "relu" else np.exp(z - z.max()) / np.exp(z - z.max()).sum()
        out.append(a)
        w_at += i * o
        b_at += o
    return np.concatenate(out)


@pytest.mark.parametrize("topology", [[784, 512, 1000, 10], [33, 100, 7], [5, 3]])
def test_every_call_answers_its_own_input(spg, has_gpu, topology):
    import torch
    a = spg.abi
    acts = ["relu"] * (len(topology) - 2) + ["softmax"]
    net = spg.Network.build(topology, [a.ACT_RELU] * (len(topology) - 2) + [a.ACT_SOFTMAX], a.WEIGHT_INITIALIZATION_NONE)
    rng = np.random.default_rng(len(topology))
    net.weights[:] = rng.standard_normal(net.weights.size).astype(np.float32) / np.sqrt(topology[0])
    net.biases[:] = rng.standard_normal(net.biases.size).astype(np.float32) * 0.1
    other = torch.cuda.Stream()
    for step in range(24):
        x = rng.standard_normal(topology[0]).astype(np.float32)
        if step == 5:
            net.forward_batch(rng.standard_normal((8, topology[0])).astype(np.float32))        # the workspace grows
        if step == 9:
            net.weights[:] *= 0.5                                                               # other weights, another device image
            net.sync_weights()
        if step == 14:
            net.set_stream(other.cuda_stream)
        if step == 19:
            net.profile(True)
        y = net.forward(x)
        exp = want(net, x, acts)
        assert np.abs(layers(net) - exp).max() <= 2e-5 * max(1, np.abs(exp).max()), step
        assert np.array_equal(y, layers(net)[-topology[-1]:])
    net.profile(False)
    net.set_stream(None)
    # a NaN goes through to the answer (as whatever NaN the device makes of it), and the next call is right
    for bits in (0x7FC00000, 0xFFF1DEAD):
        bad = np.full(topology[0], 1, np.float32)
        bad.view(np.uint32)[0] = bits
        net.forward(bad)
        x = rng.standard_normal(topology[0]).astype(np.float32)
        net.forward(x)
        assert np.abs(layers(net) - want(net, x, acts)).max() <= 2e-5 * max(1, np.abs(want(net, x, acts)).max())
    net.free()


def test_many_nets_side_by_side(spg, has_gpu):
    import threading
    a = spg.abi
    failed = []

    def work(seed):
        rng = np.random.default_rng(seed)
        net = spg.Network.build([64, 48, 10], [a.ACT_RELU, a.ACT_SOFTMAX], a.WEIGHT_INITIALIZATION_NONE)
        net.weights[:] = rng.standard_normal(net.weights.size).astype(np.float32) / 8
        for _ in range(50):
            x = rng.standard_normal(64).astype(np.float32)
            if np.abs(net.forward(x) - want(net, x, ["relu", "softmax"])[-10:]).max() > 2e-5:
                failed.append(seed)
        net.free()

    threads = [threading.Thread(target=work, args=(s,)) for s in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


@pytest.mark.parametrize("topology,acts", [([784, 512, 1000, 10], [1, 1, 5]), ([33, 100, 7], [1, 2]), ([4096, 24], [0])])
def test_last_outputs_go_to_the_host_alone(spg, has_gpu, topology, acts):
    """Whoever has seen every output may go on before the stream is idle: no store to device memory may be under way then."""
    import torch
    lib = spg.lib()
    lib.spgk_rows_sample.argtypes = [C.c_void_p, C.c_uint32, C.c_void_p, C.c_void_p, C.c_void_p]
    pairs = list(zip(topology, topology[1:]))
    gen = torch.Generator().manual_seed(1)
    w = [(torch.randn(b, a, generator=gen) / a ** 0.5).cuda() for a, b in pairs]
    bias = [torch.randn(b, generator=gen).cuda() for _, b in pairs]
    layers = (spg.abi.KLayer * len(pairs))(*[spg.abi.KLayer(m.data_ptr(), v.data_ptr(), 1.0, a, b, 0, act) for (a, b), m, v, act in zip(pairs, w, bias, acts)])
    host = torch.full((sum(topology),), -7.0).pin_memory()
    host[:topology[0]] = torch.randn(topology[0], generator=gen)
    dev = torch.full((sum(topology),), -7.0, device="cuda")
    torch.cuda.synchronize()
    assert lib.spgk_rows_sample(layers, len(pairs), host.data_ptr(), dev.data_ptr(), None) == 0
    torch.cuda.synchronize()
    last = topology[-1]
    assert torch.equal(dev[:-last].cpu(), host[:-last]) and bool((dev[-last:] == -7.0).all())
    a = host[:topology[0]].double()
    for m, v, act in zip(w, bias, acts):
        z = m.double().cpu() @ a + v.double().cpu()
        a = {0: torch.sigmoid, 1: torch.relu, 2: torch.tanh, 5: lambda t: torch.softmax(t, 0)}[act](z)
    assert float((host[-last:].double() - a).abs().max()) <= 2e-5
