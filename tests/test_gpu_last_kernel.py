"""Calls of the three-layer net on either side of the line between its two kernels: the path has one name, the kernel another.  What the parity tests ask of
AUTO at 2048 and 4096 rows, where the net runs by clusters, is asked of the other kernel here."""
import ctypes as C

import numpy as np
import pytest

import nets

pytestmark = pytest.mark.gpu

FUSED, WHOLE = "spg_mlp3_fused_kernel", "spg_chain_kernel"


@pytest.fixture
def net(spg, tmp_path):
    path = nets.make_net_file(spg, str(tmp_path / "A_int8.nn"), nets.A_TOPO, nets.A_ACTS, 3, seed=1234, reference_rng=True)
    n = spg.Network.load(path)
    n.path = path
    spg.set_math_mode(spg.abi.MATH_AUTO)
    yield n
    spg.set_math_mode(spg.abi.MATH_AUTO)
    n.free()


@pytest.mark.parametrize("rows,kernel", [(1024, WHOLE), (4096, WHOLE), (12288, FUSED), (16384, FUSED)])
@pytest.mark.parametrize("mode", ["auto", "fast"])
def test_the_kernel_that_ran(spg, net, rows, kernel, mode):
    spg.set_math_mode({"auto": spg.abi.MATH_AUTO, "fast": spg.abi.MATH_FAST}[mode])
    x = nets.uniform_inputs(rows, 784, seed=rows)
    for _ in range(2):                                         # (AUTO: the margin is measured, and known)
        net.forward_batch(x)
        assert (spg.last_path(), spg.last_kernel()) == ("tcgen05-fused", kernel)
    net.forward_batch(x[:3])
    assert spg.last_kernel() == spg.last_path() == "rows"


@pytest.mark.parametrize("n", [12288, 16384])
def test_rows_that_leave_the_fp16_range(spg, oracle, net, n):
    onet = oracle.OracleNet.from_file(net.path)
    x = nets.uniform_inputs(n, 784, seed=99)
    big = [3, n // 2, n - 1]
    x[big[0]] *= 1.0e6
    x[big[1], 17] = 3.0e5
    x[big[2]] *= 4.0e3
    got = net.forward_batch(x)
    assert spg.last_kernel() == FUSED and np.all(np.isfinite(got))
    assert np.abs(got[big] - onet.forward_batch(x[big])).max() <= 5e-5
    assert spg.lib().spingalett_last_repaired(net._h) >= 2
    x[big] = 0.5
    other = net.forward_batch(x)
    keep = np.ones(n, bool)
    keep[big] = False
    assert np.abs(other[keep] - got[keep]).max() <= 2e-6


def test_the_margin_is_measured_again(spg, oracle, net):
    import torch
    lib, n = spg.lib(), 12288
    lib.spingalett_net_margin.restype = C.c_float
    onet = oracle.OracleNet.from_file(net.path)
    rng = np.random.default_rng(21)
    x = torch.from_numpy(rng.random((n, 784), dtype=np.float32)).cuda()
    harsh = (rng.standard_normal((n, 784)) * 6.0).astype(np.float32)
    harsh_d, y = torch.from_numpy(harsh).cuda(), torch.empty(n, 10, device="cuda")
    net.forward_batch_ptr(x.data_ptr(), n, y.data_ptr())
    first = float(lib.spingalett_net_margin(net._h))
    assert spg.last_kernel() == FUSED and first > 0.0
    for _ in range(1030):
        net.forward_batch_ptr(harsh_d.data_ptr(), n, y.data_ptr())
    net.synchronize()
    later = float(lib.spingalett_net_margin(net._h))
    assert spg.last_kernel() == FUSED and later >= first and np.isfinite(later), (first, later)
    agree, err = nets.parity(y.cpu().numpy(), onet.forward_batch(harsh))
    assert agree >= 0.999 and err <= 5e-3, (agree, err)
