"""A whole net in one launch (spg_chain.cu) through spgk_chain_plan and spgk_chain_forward: widths and rows at the edges of tiles, blocks and
clusters, both 16-bit types, one and two terms of either operand, rows gathered and scattered, row counts known on the device."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_gemm_split import ACT, TIMEOUT, planes

pytestmark = pytest.mark.gpu

SOFTMAX = 5


class Plan(C.Structure):
    _fields_ = [("C", C.c_uint32), ("R", C.c_uint32), ("clusters", C.c_uint32), ("exchange_bytes", C.c_uint32), ("scratch_bytes", C.c_uint64),
                ("us", C.c_float), ("layered_us", C.c_float)]


@pytest.fixture(scope="module")
def lib(spg):
    lib, vp, u32 = spg.lib(), C.c_void_p, C.c_uint32
    lib.spgk_chain_plan.argtypes = [vp, u32, u32, C.c_int, C.c_int, C.c_int, C.POINTER(Plan)]
    lib.spgk_chain_forward.argtypes = [C.POINTER(Plan), vp, u32, vp, vp, vp, C.c_int, C.c_int, C.c_int, vp, u32, vp, u32, vp, u32, C.c_int, C.c_int, vp, vp, vp]
    lib.spgk_gemm_tc_status.argtypes = [vp, vp]
    lib.spgk_set_dynamic_rows.argtypes = [vp, u32]
    lib.spgk_set_output_rows.argtypes = [vp]
    lib.spgk_set_margin_sink.argtypes = [C.c_float, vp, vp]
    lib.spgk_error_string.restype = C.c_char_p
    return lib


class Net:
    def __init__(self, spg, lib, topology, acts, t16, a_parts, w_parts, seed=0):
        import torch
        rng = np.random.default_rng(seed)
        self.lib, self.topology, self.acts, self.t16, self.a_parts, self.w_parts = lib, topology, acts, t16, a_parts, w_parts
        dt = torch.float16 if t16 == 0 else torch.bfloat16
        pairs = list(zip(topology, topology[1:]))
        self.w32 = [(rng.standard_normal((b, a)) / np.sqrt(a)).astype(np.float32) for a, b in pairs]
        self.w16 = [planes(w, dt, w_parts) for w in self.w32]
        self.bias = [torch.from_numpy(rng.standard_normal(b).astype(np.float32) * 0.3).cuda() for _, b in pairs]
        self.layers = (spg.abi.KLayer * len(pairs))(*[spg.abi.KLayer(w.data_ptr(), v.data_ptr(), 0.75, a, b, 0, act)
                                                      for (a, b), w, v, act in zip(pairs, self.w16, self.bias, acts)])
        self.status = torch.zeros(16, dtype=torch.int32, device="cuda")
        n = len(pairs)
        self.ptrs = (C.c_void_p * n)(*[w.data_ptr() for w in self.w16])
        self.ld = (C.c_uint32 * n)(*[w.shape[2] for w in self.w16])
        self.plane = (C.c_uint64 * n)(*[w.shape[1] * w.shape[2] for w in self.w16])

    def want(self, x):
        """Every layer in 64 bits on the operands as they are meant, and a bound on what 16-bit terms and fp32 sums may change: values of a
        terms keep (8 or 11) bits a term, sums of K products of P passes K P roundings, no activation stretches a difference."""
        bits = 11 if self.t16 == 0 else 8
        ea = 2.0 ** -(bits * self.a_parts) + (2.0 ** -24 if self.t16 == 0 else 0.0)
        a, err = x.astype(np.float64), np.zeros(x.shape)
        for w, b, act in zip(self.w16, self.bias, self.acts):
            w = w.double().cpu().numpy()[:, :, :a.shape[1]]
            ws, mag, K = w.sum(0), np.abs(w).sum(0), a.shape[1]
            z = 0.75 * (a @ ws.T) + b.double().cpu().numpy()
            tiny = 2.0 ** -25 if self.t16 == 0 else 0.0                      # what fp16's smallest spacing leaves of a value
            own = np.abs(a) * ea + tiny
            cross = 2.0 ** -(bits * 2) if self.w_parts > 1 else 0.0          # lo * lo is left out
            terms = self.a_parts + self.w_parts - 1
            err = 0.75 * ((err + own) @ mag.T + (np.abs(a) @ mag.T) * (cross + (terms * K + 24) * 2.0 ** -23)) + 2.0 ** -22 * (np.abs(z) + 1)
            a = z if act == SOFTMAX else ACT[act](z)
        return a, err

    def run(self, x, rows=None, ld=None, softmax=0, counted=None, x_rows=None, y_rows=None, out_rows=None, fails=False, ready=0):
        import torch
        rows = len(x) if rows is None else rows
        plan = Plan()
        assert self.lib.spgk_chain_plan(self.layers, len(self.layers), rows, self.w_parts, self.a_parts, softmax, C.byref(plan)) == 0
        scratch = torch.full((int(plan.scratch_bytes),), 0xFF, dtype=torch.uint8, device="cuda")      # (NaN where nothing is written)
        y = torch.full((out_rows or rows, self.topology[-1] + 1), -7.0, device="cuda")
        self.lib.spgk_set_output_rows(y_rows.data_ptr() if y_rows is not None else None)
        rc = self.lib.spgk_chain_forward(C.byref(plan), self.layers, len(self.layers), self.ptrs, self.ld, self.plane, self.w_parts, self.t16, self.a_parts,
                                         x.data_ptr(), ld or x.stride(0), x_rows.data_ptr() if x_rows is not None else None, rows, y.data_ptr(), y.stride(0), softmax,
                                         ready, scratch.data_ptr(), self.status.data_ptr(), None)
        self.lib.spgk_set_output_rows(None)
        assert rc == 0, self.lib.spgk_error_string()
        assert self.lib.spgk_gemm_tc_status(self.status.data_ptr(), None) == (TIMEOUT if fails else 0), self.lib.spgk_error_string()
        assert bool((y[:, -1] == -7.0).all())
        return y[:, :-1].cpu().numpy(), plan


def inputs(rows, width, seed=3):
    import torch
    x = np.random.default_rng(seed).standard_normal((rows, width)).astype(np.float32)
    return x, torch.from_numpy(x).cuda()


NETS = [([1, 1, 1], [1, 6]), ([8, 16, 8], [6, 6]), ([15, 17, 7], [1, 0]), ([64, 63, 128], [2, 1]), ([65, 64, 129], [3, 2]), ([127, 129, 33], [4, 0]),
        ([129, 1000, 9], [1, 6]), ([784, 512, 1000, 10], [1, 1, 6]), ([301, 777, 333, 129, 37], [2, 3, 1, 0]), ([20, 3, 200, 5, 130], [1, 3, 4, 2]),
        ([40, 24, 24, 24, 24, 24, 24, 24, 12], [1, 2, 3, 4, 0, 1, 6, 6]), ([2048, 96, 300], [1, 6]), ([100, 2040, 1], [0, 2])]


@pytest.mark.parametrize("rows", [1, 16, 17, 129, 530, 2113])
@pytest.mark.parametrize("net", range(len(NETS)), ids=["-".join(map(str, t)) for t, _ in NETS])
@pytest.mark.parametrize("t16,a_parts,w_parts", [(0, 1, 1), (0, 2, 1), (1, 2, 1), (1, 2, 2), (1, 1, 1)])
def test_nets(spg, lib, net, rows, t16, a_parts, w_parts):
    topology, acts = NETS[net]
    n = Net(spg, lib, topology, acts, t16, a_parts, w_parts, seed=net)
    x, xd = inputs(rows, topology[0])
    y, plan = n.run(xd, ready=rows % 2)
    want, err = n.want(x)
    assert 1 <= plan.C <= 8 and plan.R % 16 == 0
    assert np.all(np.abs(y - want) <= err), (plan.C, plan.R, np.max(np.abs(y - want) / err))


def test_the_sizes_meet_every_cluster(spg, lib):
    met = set()
    for topology, acts in NETS + [([512, 1500, 1500, 64], [1, 1, 6]), ([2000, 2000, 10], [1, 6])]:
        n = Net(spg, lib, topology, acts, 1, 2, 1)
        for rows in (1, 16, 17, 100, 129, 256, 400, 530, 1000, 2113, 4000):
            plan = Plan()
            if lib.spgk_chain_plan(n.layers, len(n.layers), rows, 1, 2, 0, C.byref(plan)) == 0:
                met.add(plan.C)
    assert {1, 2, 4, 8} <= met and met & {3, 5, 6, 7}, met


@pytest.mark.parametrize("width,shift,pad", [(64, 1, 0), (64, 2, 0), (64, 0, 3), (66, 0, 0), (63, 3, 1)])
def test_inputs_anywhere(spg, lib, width, shift, pad):
    """Rows that do not lie on 16 bytes, or are longer than the net's input."""
    import torch
    n = Net(spg, lib, [width, 80, 12], [1, 6], 1, 2, 1)
    rows = 77
    x = np.random.default_rng(1).standard_normal((rows, width + pad)).astype(np.float32)
    flat = torch.full((x.size + 8,), float("nan"), device="cuda")
    flat[shift:shift + x.size] = torch.from_numpy(x.reshape(-1)).cuda()
    y, _ = n.run(flat[shift:], rows=rows, ld=width + pad)
    want, err = n.want(x[:, :width])
    assert np.all(np.abs(y - want) <= err)


@pytest.mark.parametrize("width", [2, 10, 32, 33, 128])
def test_softmax_and_margin(spg, lib, width):
    import torch
    rows = 700
    n = Net(spg, lib, [100, 300, width], [1, SOFTMAX], 1, 2, 1, seed=width)
    x, xd = inputs(rows, 100)
    z, err = n.want(x)
    idx, count = torch.zeros(rows, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    lib.spgk_set_margin_sink(0.3, idx.data_ptr(), count.data_ptr())
    try:
        y, _ = n.run(xd, softmax=1)
    finally:
        lib.spgk_set_margin_sink(0.0, None, None)
    want = np.exp(z - z.max(1, keepdims=True))
    want /= want.sum(1, keepdims=True)
    # a change of the logits by e changes a probability by 2 e of itself at most; 1e-6: expf, the sum and the quotient
    assert np.all(np.abs(y - want) <= want * (4 * err.max(1, keepdims=True) + 1e-6) + 1e-30)
    top = np.sort(z, 1)
    gap, slack = top[:, -1] - top[:, -2], 2 * err.max(1)
    listed = set(idx[:int(count)].cpu().tolist())
    assert len(listed) == int(count)
    assert all(r in listed for r in np.nonzero(gap < 0.3 - slack)[0]) and all(gap[r] < 0.3 + slack[r] for r in listed)


@pytest.mark.parametrize("topology,acts", [([784, 512, 1000, 10], [1, 1, SOFTMAX]), ([50, 70, 300], [2, 6])])
def test_counted_and_listed_rows(spg, lib, topology, acts):
    """Rows of a list, as many as the device says, to their places: the same bits for any guess of the count, nothing beyond the count."""
    import torch
    cap = 5000
    n = Net(spg, lib, topology, acts, 1, 2, 1)
    x, xd = inputs(cap, topology[0])
    order = np.random.default_rng(0).permutation(cap).astype(np.int32)
    rows = torch.from_numpy(order).cuda()
    softmax = int(acts[-1] == SOFTMAX)
    z, err = n.want(x)
    want = z
    if softmax:
        want = np.exp(z - z.max(1, keepdims=True))
        want /= want.sum(1, keepdims=True)
        err = want * (4 * err.max(1, keepdims=True) + 1e-6)
    blocks = set()
    try:
        for count in (0, 1, 15, 16, 961, 4999):
            c = torch.tensor([count], dtype=torch.int32, device="cuda")
            results = []
            for guess in (0, 20, 950, 3000, 5000):
                lib.spgk_set_dynamic_rows(c.data_ptr(), guess)
                y, plan = n.run(xd, softmax=softmax, x_rows=rows, y_rows=rows)
                blocks.add(plan.R)
                results.append(y)
            for y in results[1:]:
                assert np.array_equal(results[0], y)
            live, rest = order[:count], order[count:]
            assert np.all(np.abs(results[0][live] - want[live]) <= err[live]) and np.all(results[0][rest] == -7.0)
    finally:
        lib.spgk_set_dynamic_rows(None, 0)
    assert len(blocks) >= 3, blocks


def test_a_wait_that_gives_up_is_reported(spg, lib):
    """Every CTA gives its first tile up with copies and products under way: the status says so, nothing is written, and the next call is right."""
    for topology, acts, rows in (([784, 512, 1000, 10], [1, 1, 6], 300), ([64, 80, 200], [1, 6], 3000)):
        n = Net(spg, lib, topology, acts, 1, 2, 1)
        x, xd = inputs(rows, topology[0])
        lib.spgk_selftest_impatient(1)
        try:
            y, _ = n.run(xd, fails=True)
        finally:
            lib.spgk_selftest_impatient(0)
        assert np.all(y == -7.0)
        y, _ = n.run(xd)
        want, err = n.want(x)
        assert np.all(np.abs(y - want) <= err)


@pytest.mark.parametrize("name,rows,auto_path", [("fp32", 60, "tcgen05"), ("bf16", 60, "tcgen05"), ("int4", 100, "tcgen05")])
def test_which_calls_come_here(spg, name, rows, auto_path, tmp_path):
    """Nets whose 16-bit operands are small, from 25 rows on, whatever the mode; in FAST they keep two terms up to 96 rows where the streaming
    kernel would have."""
    topology = [256, 256, 64]
    net = spg.Network.build(topology, [spg.abi.ACT_RELU, spg.abi.ACT_SIGMOID], spg.abi.WEIGHT_INITIALIZATION_NONE)
    rng = np.random.default_rng(2)
    net.weights[:] = rng.standard_normal(net.weights.size).astype(np.float32) / 16
    path = str(tmp_path / "net.nn")
    net.save(path, spg.abi.PRECISION_NAMES[name])
    net.free()
    net = spg.Network.load(path)
    x = rng.standard_normal((rows, 256)).astype(np.float32)
    w1, w2 = net.weights[:65536].reshape(256, 256).astype(np.float64), net.weights[65536:].reshape(64, 256).astype(np.float64)
    want = 1 / (1 + np.exp(-np.maximum(x @ w1.T, 0) @ w2.T))
    out = (C.c_uint32 * 2)()
    for mode in (spg.abi.MATH_EXACT, spg.abi.MATH_FAST, spg.abi.MATH_AUTO):
        spg.set_math_mode(mode)
        try:
            y = net.forward_batch(x)
        finally:
            spg.set_math_mode(spg.abi.MATH_AUTO)
        fast = mode == spg.abi.MATH_FAST and not (rows <= 96 and name == "bf16")
        assert np.abs(y - want).max() <= (2e-3 if fast else 4e-5)      # one term: 2^-11 of values of size 1 to 3, 256 of them at random
        if mode == spg.abi.MATH_EXACT:
            assert spg.last_path() == auto_path
            spg.lib().spgk_chain_arrangement(out)
            assert out[0] >= 1 and out[1] % 16 == 0 and out[1] > 0
    net.free()


@pytest.mark.parametrize("t16,a_parts,w_parts", [(0, 1, 1), (1, 1, 1), (0, 2, 1), (1, 2, 1), (1, 2, 2)])
@pytest.mark.parametrize("act", [0, 1, 2, 3, 4, 6])
@pytest.mark.parametrize("topology", [[70, 100, 91, 33], [70, 100, 91, 200], [129, 45, 6], [40, 7, 9, 11, 131]], ids=lambda t: "-".join(map(str, t)))
def test_infinities_stay_in_their_rows_and_columns(spg, lib, topology, act, t16, a_parts, w_parts):
    """Widths that are no multiple of 16, of positive weights: an infinity is an infinity in every sum, and what an activation makes of it behind.
    With one term that is the answer; an infinity has no second term (its row is NaN, in every output).  Other rows are as they were."""
    import torch
    acts = [act] * (len(topology) - 1)
    n = Net(spg, lib, topology, acts, t16, a_parts, w_parts, seed=act)
    for w in n.w16:
        w.abs_()
    x, xd = inputs(301, topology[0])
    bad = np.arange(0, 301, 9)
    x[bad, 3] = np.inf if t16 else 1e6                         # beyond fp16: an infinity as well
    xd.copy_(torch.from_numpy(x))
    y, _ = n.run(xd)
    good = np.setdiff1d(np.arange(301), bad)
    want, err = n.want(x[good])
    assert np.all(np.abs(y[good] - want) <= err)
    x[bad, 3] = np.inf
    with np.errstate(all="ignore"):
        far, _ = n.want(x[bad])
    if a_parts > 1:
        assert act == 1 or np.isnan(y[bad]).all()              # (a NaN is not above zero: ReLU makes 0 of it)
    elif act in (1, 3, 4, 6):
        assert np.isposinf(far).all() and np.array_equal(y[bad], far.astype(np.float32))
    else:
        assert np.isfinite(far).all() and np.abs(y[bad] - far).max() <= 0.02        # (hidden values of exactly 1 or a half, sums of 100 or fewer)


@pytest.mark.parametrize("a_parts", [1, 2])
@pytest.mark.parametrize("topology", [[784, 512, 1000, 10], [301, 777, 333, 129, 37], [64, 80, 200], [512, 1500, 1500, 64]])
def test_scratch_goes_by_the_rows_alone(spg, lib, topology, a_parts):
    """Whatever the guess of a count, and never less for more rows: a workspace that has served a call serves every later one of as many rows or fewer."""
    import torch
    n = Net(spg, lib, topology, [1] * (len(topology) - 1), 1, a_parts, 1)
    plan, c = Plan(), torch.zeros(1, dtype=torch.int32, device="cuda")

    def scratch(rows):
        if lib.spgk_chain_plan(n.layers, len(n.layers), rows, 1, a_parts, 0, C.byref(plan)) != 0:
            return None                                        # (more rows than this net's blocks hold)
        assert plan.scratch_bytes >= 2 * plan.clusters * plan.exchange_bytes
        return plan.scratch_bytes

    sizes = [size for size in (scratch(rows) for rows in [*range(1, 5000, 37), *range(5000, 66000, 611)]) if size]
    assert len(sizes) > 100 and sizes == sorted(sizes)
    try:
        last = 0
        for rows in (600, 1024, 1500, 8192, 65536):
            met = set()
            for guess in (0, 1, 20, 333, 950, 3000, 10000, rows):
                lib.spgk_set_dynamic_rows(c.data_ptr(), guess)
                met.add(scratch(rows))
            assert len(met) == 1 and max(met) >= last, (rows, met)
            last = max(met)
    finally:
        lib.spgk_set_dynamic_rows(None, 0)


@pytest.mark.parametrize("topology,rows", [([64, 128, 16], 20000), ([64, 128, 64], 3000), ([4096, 4096], 2)])
def test_outputs_in_the_place_of_inputs(spg, topology, rows):
    import torch
    a = spg.abi
    net = spg.Network.build(topology, [a.ACT_RELU] * (len(topology) - 2) + [a.ACT_SIGMOID], a.WEIGHT_INITIALIZATION_NONE)
    net.weights[:] = np.random.default_rng(1).standard_normal(net.weights.size, dtype=np.float32) / 8
    x = torch.randn(rows, topology[0], device="cuda")
    y, both = torch.empty(rows, topology[-1], device="cuda"), x.clone()
    spg.set_math_mode(a.MATH_EXACT)
    try:
        net.forward_batch_ptr(x.data_ptr(), rows, y.data_ptr())
        net.forward_batch_ptr(both.data_ptr(), rows, both.data_ptr())
        net.synchronize()
    finally:
        spg.set_math_mode(a.MATH_AUTO)
    got = both.reshape(-1)[:y.numel()].reshape(y.shape)
    assert float((got - y).abs().max()) <= 2e-4                # (logits of some units, two 16-bit terms of either operand)
    net.free()
