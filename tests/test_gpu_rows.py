"""One to eight rows of a small net (spg_rows.cu): every precision, widths around a lane's eight values and a warp's 1024, rows that
start in the middle of a byte, rows that several warps share, softmax rows finished in the kernel (up to 128 outputs) and behind it; which
nets go there."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# payload bytes of a random matrix and the values they stand for
def matrix(rng, out, inn, prec):
    count = out * inn
    if prec == 0:
        w = rng.standard_normal(count).astype(np.float32)
        return w.view(np.uint8), w
    if prec in (1, 2):
        w = rng.standard_normal(count).astype(np.float32)
        if prec == 1:
            h = w.astype(np.float16)
            return h.view(np.uint8), h.astype(np.float64)
        h = (w.view(np.uint32) >> 16).astype(np.uint16)
        return h.view(np.uint8), (h.astype(np.uint32) << 16).view(np.float32)
    bits = {3: 8, 4: 4, 5: 2}[prec]
    q = rng.integers(-(1 << (bits - 1)), 1 << (bits - 1), count)
    per = 8 // bits
    padded = np.zeros(-(-count // per) * per, np.int64)
    padded[:count] = q & ((1 << bits) - 1)
    return (padded.reshape(-1, per) << (np.arange(per) * bits)).sum(1).astype(np.uint8), q


@pytest.mark.parametrize("prec", range(6))
@pytest.mark.parametrize("widths", [(1, 1, 2), (7, 9, 3), (8, 16, 128), (301, 77, 129), (1023, 33, 10), (1024, 40, 64), (1032, 8, 5), (2049, 17, 1), (2048, 2056, 70), (4096, 9, 100), (9001, 3, 128)])
def test_small_net_against_float64(spg, prec, widths):
    import torch
    lib = spg.lib()
    lib.spgk_rows_forward.argtypes = [C.POINTER(spg.abi.KLayer), C.c_uint32, C.c_void_p, C.c_uint32, C.POINTER(C.c_void_p), C.c_uint32, C.c_void_p]
    lib.spgk_error_string.restype = C.c_char_p
    rng = np.random.default_rng(prec * 100 + widths[0])
    keep, layers, values = [], (spg.abi.KLayer * 2)(), []
    for l, act in enumerate((2, 5)):
        inn, out = widths[l], widths[l + 1]
        raw, w = matrix(rng, out, inn, prec)
        scale = float(np.float32(1 / (np.abs(w).max() * np.sqrt(inn))))
        bias = rng.standard_normal(out).astype(np.float32)
        dw, db = torch.from_numpy(np.concatenate([raw, np.zeros(64, np.uint8)])).cuda(), torch.from_numpy(bias).cuda()
        keep += [dw, db]
        layers[l] = spg.abi.KLayer(dw.data_ptr(), db.data_ptr(), scale, inn, out, prec, act)
        values.append((np.asarray(w, np.float64).reshape(out, inn) * scale, bias.astype(np.float64)))
    for n in (1, 2, 3, 4, 5, 7, 8):                     # (one row of the batch a warp up to four, two beyond, the last of an odd number alone)
        for pad in (0, 1):                              # rows of the input that lie on 16 bytes, and rows that do not
            ldx = widths[0] + pad
            x = rng.standard_normal((n, ldx)).astype(np.float32)
            dx = torch.from_numpy(x).cuda()
            ys = [torch.full((n + 1, w), -3.0, device="cuda") for w in widths[1:]]
            ptrs = (C.c_void_p * 2)(*[y.data_ptr() for y in ys])
            assert lib.spgk_rows_forward(layers, 2, dx.data_ptr(), ldx, ptrs, n, None) == 0, lib.spgk_error_string()
            torch.cuda.synchronize()
            a = x[:, :widths[0]].astype(np.float64)
            hidden = np.tanh(a @ values[0][0].T + values[0][1])
            got = [y.cpu().numpy() for y in ys]
            # four products are added in fp32 (four roundings of at most the sum of their sizes), the rest in 64 bits; tanh adds two units in the last place
            off = 2.0 ** -22 * (np.abs(a) @ np.abs(values[0][0]).T)
            assert np.all(np.abs(got[0][:n] - hidden) <= off + 4 * 2.0 ** -24 * np.maximum(1.0, np.abs(a @ values[0][0].T)))
            z = hidden @ values[1][0].T + values[1][1]
            e = np.exp(z - z.max(1, keepdims=True))
            want = e / e.sum(1, keepdims=True)
            # logits of a few units, off by their own sums' roundings and by those of the hidden values
            dz = (np.abs(values[1][0]).sum(1).max()) * (off.max() + 2.0 ** -21) + 2.0 ** -22 * (np.abs(hidden) @ np.abs(values[1][0]).T).max() + 2.0 ** -23 * np.abs(z).max()
            assert np.all(np.abs(got[1][:n] - want) <= want * (2 * dz + 16 * 2.0 ** -24) + 1e-9)
            assert np.all(got[0][n] == -3.0) and np.all(got[1][n] == -3.0)


@pytest.mark.parametrize("prec", [3, 4, 5])
@pytest.mark.parametrize("n", [1, 4, 7])
@pytest.mark.parametrize("inn", [1100, 3000, 9000])
def test_integer_weights_times_large_inputs(spg, prec, n, inn):
    """Inputs up to 1e38: a stored weight times an input is out of fp32's range, a weight times an input is not.  Rows with values that are not
    finite keep them to themselves."""
    import torch
    lib = spg.lib()
    lib.spgk_rows_forward.argtypes = [C.POINTER(spg.abi.KLayer), C.c_uint32, C.c_void_p, C.c_uint32, C.POINTER(C.c_void_p), C.c_uint32, C.c_void_p]
    rng = np.random.default_rng(prec * 10 + n)
    out = 41
    raw, q = matrix(rng, out, inn, prec)
    scale = float(np.float32(1 / (np.abs(q).max() * inn)))          # no sum is larger than its largest input
    bias = rng.standard_normal(out).astype(np.float32)
    dw, db = torch.from_numpy(np.concatenate([raw, np.zeros(64, np.uint8)])).cuda(), torch.from_numpy(bias).cuda()
    layer = spg.abi.KLayer(dw.data_ptr(), db.data_ptr(), scale, inn, out, prec, 6)
    x = (rng.standard_normal((n, inn)) * 2e37).astype(np.float32)
    x[n // 2] *= np.float32(1e-37)
    x[n - 1, :2] = np.float32(1e38), np.float32(-1e38)
    if n == 7:
        x[2, 5], x[4, 6] = np.inf, np.nan
    w = np.asarray(q, np.float64).reshape(out, inn) * scale
    dx, y = torch.from_numpy(x).cuda(), torch.full((n + 1, out), -3.0, device="cuda")
    assert lib.spgk_rows_forward(C.byref(layer), 1, dx.data_ptr(), inn, (C.c_void_p * 1)(y.data_ptr()), n, None) == 0
    torch.cuda.synchronize()
    got, a = y.cpu().numpy(), x.astype(np.float64)
    good = np.isfinite(x).all(1)
    want = a[good] @ w.T + bias
    assert np.all(np.abs(got[:n][good] - want) <= 2.0 ** -22 * (np.abs(a[good]) @ np.abs(w).T) + 2.0 ** -23 * np.abs(want))
    assert not np.isfinite(got[:n][~good]).any() and np.all(got[n] == -3.0)


@pytest.mark.parametrize("topo,last", [([784, 512, 10], 5), ([301, 77, 128], 5), ([40, 4100, 100], 5), ([4100, 97], 5), ([33, 40, 129], 5), ([7, 1], 0)])
def test_a_sample_from_host_memory_gives_what_a_batch_of_one_gives(spg, topo, last):
    """forward() (input and outputs of every layer through page-locked memory; wider softmax rows by copies) against forward_batch."""
    net = spg.Network.build(topo, [1] * (len(topo) - 2) + [last], spg.abi.WEIGHT_INITIALIZATION_NONE)
    rng = np.random.default_rng(topo[0])
    net.weights[:] = rng.standard_normal(net.weights.size) / 8
    net.biases[:] = rng.standard_normal(net.biases.size)
    for _ in range(2):
        x = rng.standard_normal((1, topo[0])).astype(np.float32)
        assert np.array_equal(net.forward_batch(x)[0], net.forward(x[0])) and spg.last_path() == "rows"
        neurons = np.ctypeslib.as_array(net.c.neurons, (sum(topo),))
        assert np.array_equal(neurons[:topo[0]], x[0])
        if len(topo) > 2:
            w, b = net.weights[:topo[0] * topo[1]].reshape(topo[1], topo[0]).astype(np.float64), net.biases[:topo[1]].astype(np.float64)
            hidden = np.maximum(w @ x[0].astype(np.float64) + b, 0)
            assert np.all(np.abs(neurons[topo[0]:topo[0] + topo[1]] - hidden) <= 2.0 ** -24 * hidden + 2.0 ** -22 * (np.abs(w) @ np.abs(x[0]) + np.abs(b)))
    net.free()


# on either side of the lines: weights a layer (integers at two rows and more, rows of odd lengths), weights in all, outputs of a layer of streamed rows.  64-65536-34
# goes to two other kernels by turns.
@pytest.mark.parametrize("topo,precision,n,rows", [([4096, 1024], "int4", 8, False), ([4096, 1024], "int4", 6, True), ([4096, 1032], "int8", 1, True), ([4096, 1032], "int8", 2, False),
                                                   ([4096, 1032], "fp16", 8, True), ([1001, 3142], "int2", 2, True), ([1001, 3143], "int2", 2, False),
                                                   ([1001, 2095], "fp32", 5, True), ([1001, 2096], "fp32", 5, False), ([1001, 2096], "fp32", 8, True), ([2048, 2048, 2048], "bf16", 3, True),
                                                   ([2048, 2048, 2056], "bf16", 3, False), ([64, 65535, 32], "int4", 2, True), ([64, 65536, 34], "int4", 2, False), ([48, 65536, 34], "int4", 2, True),
                                                   ([64, 65536, 32], "fp32", 2, True)])
def test_which_nets_go_there(spg, tmp_path, topo, precision, n, rows):
    net = spg.Network.build(topo, [2] * (len(topo) - 2) + [6], spg.abi.WEIGHT_INITIALIZATION_NONE)
    rng = np.random.default_rng(sum(topo))
    net.weights[:] = rng.standard_normal(net.weights.size, dtype=np.float32) / 32
    net.biases[:] = rng.standard_normal(net.biases.size, dtype=np.float32) / 8
    net.save(str(tmp_path / "net.nn"), spg.abi.PRECISION_NAMES[precision])
    net.free()
    net = spg.Network.load(str(tmp_path / "net.nn"))
    x = rng.standard_normal((n, topo[0])).astype(np.float32)
    got = net.forward_batch(x)
    assert (spg.last_path() == "rows") == rows
    a, off, at, bt = x.astype(np.float64), 0.0, 0, 0
    for l, (i, o) in enumerate(zip(topo, topo[1:])):
        w, b = net.weights[at:at + i * o].reshape(o, i).astype(np.float64), net.biases[bt:bt + o]
        # every kernel: values to 16 bits at least, weights exact, tanh no steeper than 1
        off = off @ np.abs(w).T if l else 0.0
        off = off + 2.0 ** -15 * (np.abs(a) @ np.abs(w).T) + 2.0 ** -20
        a = a @ w.T + b
        if l + 2 < len(topo):
            a = np.tanh(a)
        at, bt = at + i * o, bt + o
    assert np.all(np.abs(got - a) <= off)
    net.free()
