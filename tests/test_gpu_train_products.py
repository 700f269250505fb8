"""The products of a training step on the tensor cores and the output end of a step (spg_train_mma.cu) at the edges of their tiles, slices and
strides, against float64."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -23
vp, u32, f32 = C.c_void_p, C.c_uint32, C.c_float


def dev(*arrays):
    import torch
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


# rows, inputs, outputs: tiles of 32, slices of 16, 32 tiles or fewer (eight warps a tile) and more (four), whole and ragged, rows on 16 bytes or not
@pytest.mark.parametrize("rows,fi,fo", [(1, 1, 17), (1, 16, 32), (31, 15, 33), (33, 17, 20), (32, 128, 32), (33, 129, 36), (1023, 65, 33), (1056, 64, 34),
                                        (47, 260, 1024), (64, 1001, 44)])
def test_products_against_float64(spg, rows, fi, fo):
    import torch
    lib = spg.lib()
    lib.spgk_train_gemm.argtypes = [C.c_int, vp, u32, vp, u32, vp, u32, u32, u32, u32, f32, vp, vp, u32, C.c_int, vp]
    lib.spgk_train_grad.argtypes = [vp, u32, vp, u32, vp, u32, vp, u32, u32, u32, f32, vp]
    rng = np.random.default_rng(rows + 7 * fi)
    x, w, d = (rng.standard_normal(s).astype(np.float32) for s in ((rows, fi), (fo, fi), (rows, fo)))
    b, a = rng.standard_normal(fo).astype(np.float32), rng.uniform(-1, 1, (rows, fi)).astype(np.float32)
    dx, dw, dd, db, da = dev(x, w, d, b, a)
    X, W, D = x.astype(np.float64), w.astype(np.float64), d.astype(np.float64)
    # a term is off by 2^-22 of itself, each of the 3K + 8 additions by at most a unit of the sum of the terms' sizes
    off = lambda K, p, q: (3 * K + 12) * EPS * (np.abs(p) @ np.abs(q))
    y = torch.full((rows + 1, fo), -7.0, device="cuda")
    assert lib.spgk_train_gemm(0, dx.data_ptr(), fi, dw.data_ptr(), fi, y.data_ptr(), fo, rows, fo, fi, 1.0, db.data_ptr(), None, 0, spg.abi.ACT_LEAKY_RELU, None) == 0
    z = X @ W.T + b
    got = y.cpu().numpy()
    assert np.all(np.abs(got[:rows] - np.where(z > 0, z, 0.01 * z)) <= off(fi, X, W.T) + 2 * EPS * np.abs(z) + EPS) and np.all(got[rows] == -7.0)
    back = torch.full((rows + 1, fi), -7.0, device="cuda")
    assert lib.spgk_train_gemm(1, dd.data_ptr(), fo, dw.data_ptr(), fi, back.data_ptr(), fi, rows, fi, fo, 1.0, None, da.data_ptr(), fi, spg.abi.ACT_TANH, None) == 0
    got, slope = back.cpu().numpy(), 1.0 - a.astype(np.float64) ** 2
    assert np.all(np.abs(got[:rows] - (D @ W) * slope) <= off(fo, D, W) + 4 * EPS * np.abs(D @ W)) and np.all(got[rows] == -7.0)
    gw, gb, gs = torch.full((fo + 1, fi), -7.0, device="cuda"), torch.full((fo + 1,), -7.0, device="cuda"), 1.0 / rows
    assert lib.spgk_train_grad(dd.data_ptr(), fo, dx.data_ptr(), fi, gw.data_ptr(), fi, gb.data_ptr(), fo, fi, rows, gs, None) == 0
    got, sums = gw.cpu().numpy(), gb.cpu().numpy()
    assert np.all(np.abs(got[:fo] - gs * (D.T @ X)) <= gs * off(rows, D.T, X) + 2 * EPS * gs * np.abs(D.T @ X)) and np.all(got[fo] == -7.0)
    assert np.all(np.abs(sums[:fo] - gs * D.sum(0)) <= gs * (rows + 2) * EPS * np.abs(D).sum(0)) and sums[fo] == -7.0


@pytest.mark.parametrize("rows,w0,w1,w2", [(256, 784, 512, 1000), (100, 301, 333, 129), (32, 24, 50, 10), (7, 36, 1024, 40), (300, 1024, 1024, 20)])
def test_two_layers_gradients_in_one_launch(spg, rows, w0, w1, w2):
    """The same bits as one launch each, for products that are cut alike and for those that are not."""
    import torch
    lib = spg.lib()

    class Gradients(C.Structure):
        _fields_ = [("delta", vp), ("a", vp), ("gw", vp), ("gb", vp), ("out", u32), ("in_", u32)]
    lib.spgk_train_grad2.argtypes = [C.POINTER(Gradients), C.POINTER(Gradients), u32, f32, vp]
    lib.spgk_train_grad.argtypes = [vp, u32, vp, u32, vp, u32, vp, u32, u32, u32, f32, vp]
    rng = np.random.default_rng(rows)
    d1, d2, x, h = dev(*(rng.standard_normal((rows, w)).astype(np.float32) for w in (w1, w2, w0, w1)))
    one, two = ([torch.full(s, -7.0, device="cuda") for s in ((w2, w1), (w2,), (w1, w0), (w1,))] for _ in range(2))
    a = Gradients(d2.data_ptr(), h.data_ptr(), one[0].data_ptr(), one[1].data_ptr(), w2, w1)
    b = Gradients(d1.data_ptr(), x.data_ptr(), one[2].data_ptr(), one[3].data_ptr(), w1, w0)
    assert lib.spgk_train_grad2(C.byref(a), C.byref(b), rows, 0.25, None) == 0
    assert lib.spgk_train_grad(d2.data_ptr(), w2, h.data_ptr(), w1, two[0].data_ptr(), w1, two[1].data_ptr(), w2, w1, rows, 0.25, None) == 0
    assert lib.spgk_train_grad(d1.data_ptr(), w1, x.data_ptr(), w0, two[2].data_ptr(), w0, two[3].data_ptr(), w1, w0, rows, 0.25, None) == 0
    for p, q in zip(one, two):
        assert torch.equal(p, q) and not torch.any(p == -7.0)


# inputs around a lane's four, a warp's 128 and the 1024 of a round; one and two outputs a warp; an odd number of rows
@pytest.mark.parametrize("sigmoid", [0, 1])
@pytest.mark.parametrize("rows,fi,fo", [(1, 1, 1), (2, 4, 8), (3, 127, 9), (5, 128, 16), (255, 1000, 10), (4, 1023, 3), (2, 1024, 16), (3, 1028, 10), (3, 2049, 10)])
def test_output_end_against_float64(spg, rows, fi, fo, sigmoid):
    import torch
    lib = spg.lib()
    lib.spgk_train_output.argtypes = [vp, u32, vp, u32, vp, vp, vp, vp, vp, u32, u32, u32, C.c_int, vp]
    rng = np.random.default_rng(rows + 3 * fi)
    x, w, b = (rng.standard_normal(s).astype(np.float32) for s in ((rows, fi), (fo, fi), (fo,)))
    w /= np.float32(np.sqrt(fi))
    t = np.eye(fo, dtype=np.float32)[rng.integers(0, fo, rows)]
    dx, dw, db, dt = dev(x, w, b, t)
    y, delta = (torch.full((rows + 1, fo), -7.0, device="cuda") for _ in range(2))
    loss = torch.zeros(1, device="cuda")
    assert lib.spgk_train_output(dx.data_ptr(), fi, dw.data_ptr(), fi, db.data_ptr(), y.data_ptr(), dt.data_ptr(), delta.data_ptr(), loss.data_ptr(), rows, fo, fi,
                                 sigmoid, None) == 0
    X, W = x.astype(np.float64), w.astype(np.float64)
    z = X @ W.T + b
    dz = (fi / 32 + 12) * EPS * (np.abs(X) @ np.abs(W).T + np.abs(b)).max()      # a lane adds K/32 terms, the tree five levels
    want = 1 / (1 + np.exp(-z)) if sigmoid else np.exp(z - z.max(1, keepdims=True)) / np.exp(z - z.max(1, keepdims=True)).sum(1, keepdims=True)
    got, d = y.cpu().numpy(), delta.cpu().numpy()
    rel = 2 * dz + 24 * EPS                                                      # exp (2 ulp), a sum of 16, a quotient
    assert np.all(np.abs(got[:rows] - want) <= rel * want) and np.all(got[rows] == -7.0)
    assert np.array_equal(d[:rows], got[:rows] - t) and np.all(d[rows] == -7.0)
    c = np.clip(want, 1e-9, 1 - 1e-9) if sigmoid else np.maximum(want, 1e-9)
    cost = -(t * np.log(c) + (1 - t) * np.log(1 - c)).sum() if sigmoid else -(t * np.log(c)).sum()
    assert abs(float(loss[0]) - cost) <= (rel * 4 + (rows + 8) * EPS) * (rows * fo + abs(cost))
