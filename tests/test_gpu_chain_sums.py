"""How long the sums of a net in one launch are: accumulators of a tile from one to eight, of several stages, one stage or one k-block, those of a cut last layer
among them; and what positive values lose to the tensor core's cutting off, which goes by the products that follow one another in an accumulator."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_chain import Net, inputs, lib  # noqa: F401  (lib: fixture)
from test_gpu_gemm_split import lib as split_lib, planes  # noqa: F401  (split_lib: fixture)

pytestmark = pytest.mark.gpu

FP16, SOFTMAX = 1, 5
NETS = [([192, 100, 64], [1, 6]), ([448, 256, 200], [2, 6]), ([512, 300, 130], [1, 0]), ([784, 512, 1000, 10], [1, 3, 6]), ([900, 1000, 90], [4, 2]),
        ([300, 90, 70, 500, 7], [1, 1, 2, 6]), ([2048, 500, 100], [1, 6]), ([1000, 24, 24], [1, 6])]


@pytest.mark.parametrize("rows", [1, 40, 300, 2500])
@pytest.mark.parametrize("net", range(len(NETS)), ids=["-".join(map(str, t)) for t, _ in NETS])
@pytest.mark.parametrize("t16,a_parts,w_parts", [(0, 2, 1), (0, 1, 1), (1, 2, 2)])
def test_accumulators(spg, lib, net, rows, t16, a_parts, w_parts):  # noqa: F811
    topology, acts = NETS[net]
    n = Net(spg, lib, topology, acts, t16, a_parts, w_parts, seed=net)
    for layer in n.layers:
        layer.precision = FP16                                 # (its sums are asked to be the shortest)
    x, xd = inputs(rows, topology[0])
    y, plan = n.run(xd)
    want, err = n.want(x)
    assert np.all(np.abs(y - want) <= err), (plan.C, plan.R, np.max(np.abs(y - want) / err))


def layer_by_layer(n, x):
    import torch
    dt = torch.float16 if n.t16 == 0 else torch.bfloat16
    rows, a = len(x), planes(x, dt, n.a_parts)
    for l, layer in enumerate(n.layers):
        lda, ldo = a.shape[2], (layer.out + 7) & ~7
        o16, o32 = torch.zeros(2, rows, ldo, dtype=dt, device="cuda"), torch.zeros(rows, layer.out, device="cuda")
        assert n.lib.spgk_layer_gemm_tc(C.byref(layer), n.ptrs[l], n.ld[l], n.plane[l], n.w_parts, n.t16, a.data_ptr(), lda, rows * lda, n.a_parts, n.t16, o16.data_ptr(), ldo,
                                        rows * ldo, n.a_parts, o32.data_ptr(), layer.out, rows, 0, n.status.data_ptr(), None) == 0, n.lib.spgk_error_string()
        a = o16
    assert n.lib.spgk_gemm_tc_status(n.status.data_ptr(), None) == 0
    return o32.cpu().numpy()


@pytest.mark.parametrize("rows", [33, 200, 1000])
@pytest.mark.parametrize("t16", [0, 1])
@pytest.mark.parametrize("topology", [[784, 512, 64], [2048, 512, 64], [4096, 512, 64], [8192, 512, 64], [784, 512, 1000, 10], [4096, 1024, 1024, 300]], ids=lambda t: "-".join(map(str, t)))
def test_positive_values_lose_no_more_than_layer_by_layer(spg, lib, split_lib, topology, t16, rows):  # noqa: F811
    """... or the plan says that the layers one by one are the choice.  A tenth, and 2^-22 for the accumulators' own sum and its rounding."""
    n = Net(spg, lib, topology, [1] * (len(topology) - 2) + [6], t16, 2, 1, seed=1)
    for layer, w, b in zip(n.layers, n.w16, n.bias):
        layer.precision = FP16 if t16 == 0 else 2
        w[0].abs_()
        b.abs_()
    x, xd = inputs(rows, topology[0])
    x = np.abs(x)
    xd.abs_()
    y, plan = n.run(xd)
    want, _ = n.want(x)
    here, layers = [abs(float(((v - want) / want).mean())) for v in (y, layer_by_layer(n, x))]
    assert plan.layered_us == 0 or here <= 1.1 * layers + 2.0 ** -22, (here, layers)


@pytest.mark.parametrize("rows", [33, 90])
def test_short_products_stay_where_sums_hold_them(spg, rows, tmp_path):
    """INT4: the streaming kernel's sums of the first terms' products are whole, the layer kernels' are not.  16 bits of a value leave 2^-17 of it either way, at the mean of
    256 inputs and more 2^-21."""
    a = spg.abi
    topology = [256, 4096, 300]
    net = spg.Network.build(topology, [a.ACT_RELU, a.ACT_NONE], a.WEIGHT_INITIALIZATION_NONE)
    rng = np.random.default_rng(6)
    net.weights[:] = np.abs(rng.standard_normal(net.weights.size, dtype=np.float32)) / 256
    path = str(tmp_path / "net.nn")
    net.save(path, a.PRECISION_INT4)
    net.free()
    net = spg.Network.load(path)
    x = rng.random((rows, 256), dtype=np.float32)
    w = net.weights.astype(np.float64)
    want = x.astype(np.float64) @ w[:256 * 4096].reshape(4096, 256).T @ w[256 * 4096:].reshape(300, 4096).T
    spg.set_math_mode(a.MATH_EXACT)
    try:
        y = net.forward_batch(x)
    finally:
        spg.set_math_mode(a.MATH_AUTO)
    assert abs(((y - want) / want).mean()) <= 2.0 ** -21
    net.free()
