"""Arrays that go to and from the device through page-locked pieces of 8 MB (spg_stage.c): lengths around a piece, saved files byte for byte against
the host encoder, trained nets bit for bit against copies of page-locked arrays."""
import ctypes as C
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("topo", [[2048, 1024], [2048, 1025, 2], [4097, 1024, 5], [2047, 512]])      # 8 MB, a little more, two pieces and a little, one that is not full
@pytest.mark.parametrize("precision", ["fp32", "fp16", "int8", "int4", "int2"])
def test_saved_files_are_what_the_host_encoder_writes(spg, tmp_path, monkeypatch, topo, precision):
    net = spg.Network.build(topo, [spg.abi.ACT_RELU] * (len(topo) - 1), spg.abi.WEIGHT_INITIALIZATION_NONE)
    rng = np.random.default_rng(len(topo))
    net.weights[:] = rng.standard_normal(net.weights.size, dtype=np.float32)
    net.biases[:] = rng.standard_normal(net.biases.size, dtype=np.float32)
    files = [str(tmp_path / n) for n in ("device.nn", "host.nn")]
    p = spg.abi.PRECISION_NAMES[precision]
    net.save(files[0], p)
    net.save(files[0], p)                                   # over the file that is there
    monkeypatch.setenv("SPINGALETT_HOST_ENCODE", "1")
    net.save(files[1], p)
    a, b = (open(f, "rb").read() for f in files)
    assert a == b
    net.free()


def test_a_full_disk_is_an_error(spg, tmp_path):
    net = spg.Network.build([2048, 1024], [spg.abi.ACT_RELU], spg.abi.WEIGHT_INITIALIZATION_NONE)
    net.weights[:] = 1.0
    os.symlink("/dev/full", tmp_path / "full.nn")
    with pytest.raises(spg.SpingalettError):
        net.save(str(tmp_path / "full.nn"), spg.abi.PRECISION_INT8)
    net.free()


@pytest.mark.parametrize("samples", [2674, 5350])           # inputs of 8 MB (784 wide: 2675 rows) and of two pieces
def test_training_from_pageable_and_page_locked_arrays_is_the_same(spg, samples):
    import torch
    rng = np.random.default_rng(samples)
    x, t = rng.random((samples, 784), dtype=np.float32), np.eye(10, dtype=np.float32)[rng.integers(0, 10, samples)]
    px, pt = torch.from_numpy(x).pin_memory(), torch.from_numpy(t).pin_memory()
    got = []
    for a, b in ((x, t), (px.numpy(), pt.numpy())):
        net = spg.Network.build([784, 1400, 10], [spg.abi.ACT_RELU, spg.abi.ACT_SOFTMAX], spg.abi.WEIGHT_INITIALIZATION_NONE)
        net.weights[:] = np.random.default_rng(1).standard_normal(net.weights.size, dtype=np.float32) / 28
        spg.lib().spingalett_seed(3)
        net.train(a, b, epochs=4, batch_size=191, optimizer=spg.abi.OPTIMIZER_ADAM, learning_rate=1e-3)
        arrays = [np.ctypeslib.as_array(getattr(net.c, n), (net.weights.size,)).copy() for n in ("grad_weights", "opt_m_weights", "opt_v_weights")]
        got.append([net.weights.copy(), net.biases.copy()] + arrays)
        net.free()
    for a, b in zip(*got):
        assert np.any(a != 0) and np.array_equal(a, b)


def test_a_failed_allocation_is_not_the_next_launchs_error(spg):
    """Room for pieces, orders and encoders is asked for and done without where there is none: the failure must not be left for a launch to find."""
    lib = spg.lib()
    lib.spgk_malloc.argtypes = [C.POINTER(C.c_void_p), C.c_size_t]
    net = spg.Network.build([40, 30, 10], [spg.abi.ACT_RELU, spg.abi.ACT_SOFTMAX], spg.abi.WEIGHT_INITIALIZATION_NONE)
    net.weights[:] = 1.0
    x = np.ones((3, 40), np.float32)
    want = net.forward_batch(x)
    p = C.c_void_p()
    assert lib.spgk_malloc(C.byref(p), 1 << 50) != 0
    assert np.array_equal(net.forward_batch(x), want)
    net.free()
