"""Device outputs that start on any float: every kernel that writes a net's last layer, against the same call into aligned memory, bit for bit; and inputs
that start on any float, within the mode's error."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# rows: the small-batch kernels, products of few tiles, of one wave and more, on pairs of CTAs, with a head in the epilogue; outputs: a multiple of four (and of a
# tile) or not, with and without a softmax in an epilogue
@pytest.mark.parametrize("topo,last", [([96, 256, 64], 6), ([96, 256, 64], 5), ([96, 520, 1024], 0), ([96, 520, 1024], 5), ([96, 256, 512, 12], 0),
                                       ([96, 256, 512, 12], 5), ([528, 4096], 2), ([96, 30], 6)])
@pytest.mark.parametrize("precision", ["fp32", "int8"])
def test_outputs_and_inputs_on_any_float(spg, tmp_path, topo, last, precision):
    import torch
    net = spg.Network.build(topo, [1] * (len(topo) - 2) + [last], spg.abi.WEIGHT_INITIALIZATION_NONE)
    net.weights[:] = np.random.default_rng(len(topo)).standard_normal(net.weights.size, dtype=np.float32) / 16
    net.save(str(tmp_path / "n.nn"), spg.abi.PRECISION_NAMES[precision])
    net.free()
    net = spg.Network.load(str(tmp_path / "n.nn"))
    seen = set()
    try:
        for mode in (spg.abi.MATH_EXACT, spg.abi.MATH_AUTO, spg.abi.MATH_FAST):
            spg.set_math_mode(mode)
            for rows in (1, 5, 8, 40, 300, 1500, 5000, 20000):
                x = torch.randn(rows * topo[0] + 4, device="cuda")
                y = torch.zeros(rows * topo[-1] + 8, device="cuda")
                net.forward_batch_ptr(x.data_ptr(), rows, y.data_ptr())          # (AUTO measures its margin on a first call)
                net.forward_batch_ptr(x.data_ptr(), rows, y.data_ptr())
                net.synchronize()
                want = y[:rows * topo[-1]].clone()
                for at in (1, 2, 3):
                    y.fill_(-7.0)
                    net.forward_batch_ptr(x.data_ptr(), rows, y.data_ptr() + 4 * at)
                    net.synchronize()
                    assert torch.equal(y[at:at + rows * topo[-1]], want), (rows, mode, at, spg.last_path())
                    assert torch.all(y[:at] == -7.0) and torch.all(y[at + rows * topo[-1]:] == -7.0)
                seen.add(spg.last_path())
                moved = x[:rows * topo[0]].clone()
                x[1:1 + rows * topo[0]] = moved
                net.forward_batch_ptr(x.data_ptr() + 4, rows, y.data_ptr())
                net.synchronize()
                got = y[:rows * topo[-1]]
                assert torch.allclose(got, want, rtol=0, atol=float(want.abs().max()) * (2e-5 if mode == spg.abi.MATH_EXACT else 5e-3))
    finally:
        spg.set_math_mode(spg.abi.MATH_AUTO)
    assert len(seen) >= 2
    net.free()
