"""Where the integer streaming kernel keeps its operand tiles: in tensor memory beside one or two accumulators, or in shared memory for a wide layer of more
than 32 rows a group (spg_istream.cu).  Rows on either side of those lines, one segment a CTA and several, alone and in pairs, INT4 and INT2."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_istream import _bound, _is_wide, _layer, k  # noqa: F401  (k: fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("prec", [4, 5])
@pytest.mark.parametrize("out,inn,n", [(129, 1024, 8), (300, 512, 31), (1000, 2048, 32), (1000, 2048, 33), (640, 8192, 36), (5000, 4096, 64), (2600, 4096, 65), (300, 512, 130)])
def test_operand_tiles(spg, k, oracle, out, inn, n, prec, wide):  # noqa: F811
    import torch
    rng = np.random.default_rng(out + inn + n + prec)
    L, dec, bias, hold = _layer(spg, oracle, rng, out, inn, prec, 6, unused=inn // 2 if wide else None)
    x = rng.standard_normal((n, inn)).astype(np.float32)
    if wide:
        x[n // 2, inn // 2] = 1e6
    assert _is_wide(x)[0].any() == wide
    nbytes = k.spgk_istream_scratch_bytes(C.byref(L), 1, n)
    assert nbytes > 0
    scratch = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    xd, want = torch.from_numpy(x).cuda(), x.astype(np.float64) @ dec.T + bias
    for again in range(3):                             # the sums and counters are at zero again
        y = torch.full((n + 1, out), -9.0, device="cuda")
        ys = (C.c_void_p * 1)(y.data_ptr())
        assert k.spgk_istream_forward(C.byref(L), 1, xd.data_ptr(), inn, ys, n, scratch.data_ptr(), None) == 0, k.spgk_error_string()
        assert k.spgk_istream_status(scratch.data_ptr(), None) == 0, k.spgk_error_string()
        got = y.cpu().numpy()
        assert np.all(np.abs(got[:n] - want) <= _bound(x, dec, want)) and np.all(got[n] == -9.0), again
    del hold


def test_few_rows_and_many(spg, oracle, tmp_path):
    """The lines at 3 rows (nets that the small-net kernel does not take, not in EXACT) and at 448 rows of large nets: the same answers on either side, as
    the kernels that serve there in EXACT give them."""
    a = spg.abi
    for topo, prec, lines in [([4096, 4096, 500], a.PRECISION_INT4, {2: 0, 3: 1, 6: 1}), ([2048, 3072, 2048], a.PRECISION_INT8, {3: 1, 5: 1}),
                              ([512, 512, 10], a.PRECISION_INT8, {3: 0, 6: 0, 7: 1}),
                              ([8192, 10240], a.PRECISION_INT4, {257: 1, 448: 1, 449: 0}), ([8192, 10112], a.PRECISION_INT4, {256: 1, 257: 0})]:
        net = spg.Network.build(topo, [a.ACT_TANH] * (len(topo) - 1), a.WEIGHT_INITIALIZATION_NONE)
        rng = np.random.default_rng(len(topo))
        net.weights[:] = rng.standard_normal(net.weights.size, dtype=np.float32) / np.sqrt(topo[0])
        path = str(tmp_path / "net.nn")
        net.save(path, prec)
        net.free()
        net = spg.Network.load(path)
        for n, takes in lines.items():
            x = rng.standard_normal((n, topo[0]), dtype=np.float32)
            spg.set_math_mode(a.MATH_AUTO)
            y = net.forward_batch(x)
            assert (spg.last_path() == "istream") == bool(takes), (topo, n, spg.last_path())
            spg.set_math_mode(a.MATH_EXACT)
            try:
                other = net.forward_batch(x)
            finally:
                spg.set_math_mode(a.MATH_AUTO)
            assert np.abs(other - y).max() <= 1e-4, (topo, n)          # two bf16 terms: 2^-17 of a value, sums of a few units
            if takes and n < 7:
                assert spg.last_path() != "istream"
        net.free()
