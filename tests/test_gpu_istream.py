"""The 8-bit integer streaming kernel (spgk_istream_forward): whole nets of INT8 / INT4 / INT2 layers against float64.

The bound per output is derived: an input value is rounded to a multiple of S / (2^27 - 1), S the row's largest magnitude,
so it is off by less than S * 2^-27.9; products and sums are exact; the result is rounded to fp32 once and the activation
function (2 ulp) is applied.  In a row of wide range (more than an eighth of its non-zero values below 2^-12 S) those values
are off by less than 2^-27.9 of the largest thing that the first rounding left of any of them."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
Q = {3: 127.0, 4: 7.0, 5: 1.0}


@pytest.fixture()
def k(spg, has_gpu):
    assert has_gpu
    lib, vp = spg.lib(), C.c_void_p
    lib.spgk_istream_scratch_bytes.argtypes = [C.POINTER(spg.abi.KLayer), C.c_uint32, C.c_uint32]
    lib.spgk_istream_scratch_bytes.restype = C.c_size_t
    lib.spgk_istream_forward.argtypes = [C.POINTER(spg.abi.KLayer), C.c_uint32, vp, C.c_uint32, C.POINTER(vp), C.c_uint32, vp, vp]
    lib.spgk_istream_status.argtypes = [vp, vp]
    lib.spgk_error_string.restype = C.c_char_p
    return lib


def _layer(spg, oracle, rng, out, inn, prec, act, unused=None):
    """A layer whose odd outputs take nothing from the inputs `unused`."""
    import torch
    vals = (rng.standard_normal((out, inn)) / np.sqrt(inn)).astype(np.float32)
    if unused is not None:
        vals[1::2, unused] = 0.0
    raw = oracle.Oracle.encode(vals.ravel(), prec)
    scale = float(np.float32(np.frombuffer(raw[:4].tobytes(), np.float32)[0] / Q[prec]))
    # the decoded weights before their own rounding to fp32, which the bounds below leave no room for
    dec = np.rint(oracle.Oracle.decode(raw, out * inn, prec).astype(np.float64).reshape(out, inn) / scale) * scale
    w = torch.from_numpy(np.concatenate([raw[4:], np.zeros(256, np.uint8)])).cuda()
    bias = rng.standard_normal(out).astype(np.float32) * 0.1
    b = torch.from_numpy(bias).cuda()
    return spg.abi.KLayer(w.data_ptr(), b.data_ptr(), scale, inn, out, prec, act), dec, bias, (w, b)


def _is_wide(x):
    """Rows of wide range, and which of their values are small ones (a value within a rounding of 2^-12 S may go either way)."""
    s = np.abs(x).max(1, keepdims=True)
    coarse = (x != 0) & (np.abs(x) < s * 2.0 ** -12)
    return 8 * coarse.sum(1) > (x != 0).sum(1), coarse


def _bound(x, dec, y):
    s = np.abs(x).max(1, keepdims=True) * 2.0 ** -27.9
    wide, coarse = _is_wide(x)
    left = np.where(coarse, np.minimum(np.abs(x), s), 0.0).max(1, keepdims=True)
    off = np.where(wide[:, None] & coarse, left * 2.0 ** -27.9, np.where(x != 0, s, 0.0))
    return off @ np.abs(dec).T + 4e-7 * np.abs(y) + 1e-30


# one row tile and ragged ones, a tile in pieces, one box and several, one group of rows and several, a padded group
@pytest.mark.parametrize("prec", [3, 4, 5])
@pytest.mark.parametrize("out,inn,n", [(128, 64, 1), (1, 128, 4), (100, 1024, 2), (1000, 8192, 3), (129, 576, 9), (257, 4096, 17),
                                       (640, 2048, 64), (300, 1280, 65), (130, 17408, 100), (2500, 1088, 512)])
def test_layer_against_float64(spg, k, oracle, prec, out, inn, n):
    import torch
    rng = np.random.default_rng(out * 31 + inn + n)
    L, dec, bias, hold = _layer(spg, oracle, rng, out, inn, prec, 6, unused=inn // 2)
    x = rng.standard_normal((n, inn)).astype(np.float32)
    x[0] *= 1e-30                                   # rows have scales of their own
    if n > 2:
        x[1] = 0.0
        x[2, inn // 2] = 1e6                        # one large value, which half of the outputs do not use
    buf = torch.zeros(n * inn + 1, device="cuda")
    y = torch.full((n + 1, out), -9.0, device="cuda")
    nbytes = k.spgk_istream_scratch_bytes(C.byref(L), 1, n)
    assert nbytes > 0
    scratch = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    ys = (C.c_void_p * 1)(y.data_ptr())
    want = x.astype(np.float64) @ dec.T + bias
    for off in (0, 1):                              # 16-byte aligned rows and rows that are not; the second call finds the counters at zero
        buf[off:off + n * inn] = torch.from_numpy(x.ravel()).cuda()
        y.fill_(-9.0)
        assert k.spgk_istream_forward(C.byref(L), 1, buf.data_ptr() + 4 * off, inn, ys, n, scratch.data_ptr(), None) == 0, k.spgk_error_string()
        assert k.spgk_istream_status(scratch.data_ptr(), None) == 0, k.spgk_error_string()
        got = y.cpu().numpy()
        assert np.all(got[n] == -9.0)
        assert np.all(np.abs(got[:n] - want) <= _bound(x.astype(np.float64), dec, want)), np.abs(got[:n] - want).max()


@pytest.mark.parametrize("precs", [(4, 4, 4), (3, 5, 4)])
def test_chain_and_rows_that_are_not_finite(spg, k, oracle, precs):
    import torch
    rng = np.random.default_rng(5)
    topo, acts, n = [576, 384, 640, 130], [3, 4, 6], 70      # leaky, foo52, none
    built = [_layer(spg, oracle, rng, o, i, p, a) for i, o, p, a in zip(topo, topo[1:], precs, acts)]
    Ls = (spg.abi.KLayer * 3)(*[b[0] for b in built])
    x = rng.standard_normal((n, topo[0])).astype(np.float32)
    x[3, 7], x[66, 9] = np.inf, np.nan
    ys_t = [torch.zeros(n, o, device="cuda") for o in topo[1:]]
    ys = (C.c_void_p * 3)(*[t.data_ptr() for t in ys_t])
    scratch = torch.zeros(k.spgk_istream_scratch_bytes(Ls, 3, n), dtype=torch.uint8, device="cuda")
    xd = torch.from_numpy(x).cuda()
    assert k.spgk_istream_forward(Ls, 3, xd.data_ptr(), topo[0], ys, n, scratch.data_ptr(), None) == 0, k.spgk_error_string()
    assert k.spgk_istream_status(scratch.data_ptr(), None) == 0, k.spgk_error_string()
    good = np.isfinite(x).all(1)
    a = x.astype(np.float64)
    for t, (_, dec, bias, _), act in zip(ys_t, built, acts):
        a = np.where(good[:, None], a, 0.0)
        z = a @ dec.T + bias
        want = {3: np.where(z > 0, z, 0.01 * z), 4: np.where(z > 1, 1 + 0.01 * (z - 1), np.where(z < 0, 0.01 * z, z)), 6: z}[act]
        got = t.cpu().numpy()
        assert not np.any(np.isfinite(got[~good]))
        # a layer is measured on the input that the device had, so that the bound is one layer's (the activations' slopes are at most 1)
        assert np.all(np.abs(got[good] - want[good]) <= _bound(a, dec, z)[good])
        a = got.astype(np.float64)


@pytest.mark.parametrize("n", [1, 70])
def test_outputs_after_a_failure_are_nan_until_its_status_is_read(spg, k, oracle, n):
    """The status word a failed launch leaves (set here by the host): what its sums and counters hold must not come out as a
    result, not even through a rectifier, in any layer."""
    import torch
    rng = np.random.default_rng(n)
    topo = [256, 4096, 300]
    built = [_layer(spg, oracle, rng, o, i, 4, 1) for i, o in zip(topo, topo[1:])]
    Ls = (spg.abi.KLayer * 2)(*[b[0] for b in built])
    x = torch.from_numpy(rng.standard_normal((n, topo[0])).astype(np.float32)).cuda()
    ys_t = [torch.zeros(n + 1, o, device="cuda") for o in topo[1:]]
    ys = (C.c_void_p * 2)(*[t.data_ptr() for t in ys_t])
    scratch = torch.zeros(k.spgk_istream_scratch_bytes(Ls, 2, n), dtype=torch.uint8, device="cuda")
    scratch[0] = 9
    for _ in range(2):
        assert k.spgk_istream_forward(Ls, 2, x.data_ptr(), topo[0], ys, n, scratch.data_ptr(), None) == 0, k.spgk_error_string()
        torch.cuda.synchronize()
        for t in ys_t:
            assert bool(t[:n].isnan().all()) and not bool(t[n].any())
            t.zero_()
    assert k.spgk_istream_status(scratch.data_ptr(), None) == -4 and b"bounded wait 9 gave up inside the integer" in k.spgk_error_string()
    scratch.zero_()
    assert k.spgk_istream_forward(Ls, 2, x.data_ptr(), topo[0], ys, n, scratch.data_ptr(), None) == 0, k.spgk_error_string()
    assert k.spgk_istream_status(scratch.data_ptr(), None) == 0
    assert all(bool(t[:n].isfinite().all()) for t in ys_t)


def test_what_is_declined(spg, k):
    import torch
    w, b = torch.zeros(1 << 16, dtype=torch.uint8, device="cuda"), torch.zeros(64, device="cuda")
    ok = spg.abi.KLayer(w.data_ptr(), b.data_ptr(), 1.0, 64, 64, 4, 1)
    assert k.spgk_istream_scratch_bytes(C.byref(ok), 1, 16) > 0
    assert k.spgk_istream_scratch_bytes(C.byref(ok), 1, 513) == 0
    for bad in [spg.abi.KLayer(w.data_ptr(), b.data_ptr(), 1.0, 72, 64, 4, 1),        # packed rows of 36 bytes
                spg.abi.KLayer(w.data_ptr() + 4, b.data_ptr(), 1.0, 64, 64, 4, 1),    # base not 16-byte aligned
                spg.abi.KLayer(w.data_ptr(), b.data_ptr(), 1.0, 64, 64, 2, 1)]:       # not an integer file
        assert k.spgk_istream_scratch_bytes(C.byref(bad), 1, 16) == 0
    pair = (spg.abi.KLayer * 2)(spg.abi.KLayer(w.data_ptr(), b.data_ptr(), 1.0, 64, 64, 4, 5), ok)      # softmax inside the net
    assert k.spgk_istream_scratch_bytes(pair, 2, 16) == 0


# values on two and on three scales, an eighth of small ones and one more, a row of one value, next to ordinary rows
@pytest.mark.parametrize("prec", [3, 4, 5])
@pytest.mark.parametrize("out,inn,n", [(70, 576, 7), (500, 2048, 33), (130, 17408, 80)])
def test_rows_of_wide_range(spg, k, oracle, prec, out, inn, n):
    import torch
    rng = np.random.default_rng(out + inn + n)
    few = slice(0, 5)
    L, dec, bias, hold = _layer(spg, oracle, rng, out, inn, prec, 6, unused=few)
    x = rng.choice([-1.0, 1.0], (n, inn)) * rng.uniform(1.0, 2.0, (n, inn))
    x[0, few] *= 1e7
    x[1, few], x[1, 5:inn // 2] = x[1, few] * 1e20, x[1, 5:inn // 2] * 1e-9
    x[2, :inn // 8] *= 1e-6                         # as many small ones as a row may have that is not a wide one
    x[3, :inn // 8 + 1] *= 1e-6
    x[4] = 0.0
    x[4, 1] = -3.0
    x[5, few] *= 1e-38                              # few small ones, denormal
    x[6, 3] = 3e38
    x = x.astype(np.float32)
    wide, _ = _is_wide(x.astype(np.float64))
    assert wide[[0, 1, 3, 6]].all() and not wide[[2, 4, 5]].any() and not wide[7:].any()
    scratch = torch.zeros(k.spgk_istream_scratch_bytes(C.byref(L), 1, n), dtype=torch.uint8, device="cuda")
    y = torch.zeros(n, out, device="cuda")
    ys = (C.c_void_p * 1)(y.data_ptr())
    for rows in (np.arange(n), np.roll(np.arange(n), 2), np.flatnonzero(~wide)):        # the last: back to ordinary rows alone
        xr = x[rows]
        xd = torch.from_numpy(xr).cuda()
        assert k.spgk_istream_forward(C.byref(L), 1, xd.data_ptr(), inn, ys, len(rows), scratch.data_ptr(), None) == 0, k.spgk_error_string()
        assert k.spgk_istream_status(scratch.data_ptr(), None) == 0, k.spgk_error_string()
        want = xr.astype(np.float64) @ dec.T + bias
        err = np.abs(y.cpu().numpy()[:len(rows)] - want)
        assert np.all(err <= _bound(xr.astype(np.float64), dec, want)), err.max(1)


@pytest.mark.parametrize("mode", ["auto", "exact"])
@pytest.mark.parametrize("n", [8, 25, 64, 200])
def test_one_large_input_that_has_no_weight(spg, has_gpu, tmp_path, mode, n):
    """One input of 1e3 to 1e30 beside 4095 ordinary ones; every weight on it is zero.  The other inputs have to keep the 16
    bits that two bf16 terms hold (each off by less than 2^-18 of itself, independently): 8 standard deviations of their sum, and
    2^-24 of a partial sum of ordinary size for each time a tensor core adds 16 products to it (twice 4096 products in EXACT)."""
    a = spg.abi
    topo = [4096, 2048]
    net = spg.Network.build(topo, [a.ACT_LEAKY_RELU], a.WEIGHT_INITIALIZATION_HE, seed=11)
    w = net.weights.reshape(topo[1], topo[0])
    w[:, 77] = 0.0
    net.save(str(tmp_path / "m.nn"), a.PRECISION_INT4)
    net.free()
    net = spg.Network.load(str(tmp_path / "m.nn"))
    w, b = net.weights.reshape(topo[1], topo[0]).astype(np.float64), net.biases.astype(np.float64)
    assert not w[:, 77].any()
    x = np.random.default_rng(n).standard_normal((n, topo[0])).astype(np.float32)
    x[:, 77] = 10.0 ** (3 + np.arange(n) % 28)
    spg.set_math_mode(a.MATH_AUTO if mode == "auto" else a.MATH_EXACT)
    try:
        got = net.forward_batch(x)
    finally:
        spg.set_math_mode(a.MATH_AUTO)
    z = x.astype(np.float64) @ w.T + b
    tol = (8 * 2.0 ** -18 + 2 * 4096 / 16 * 2.0 ** -24) * np.sqrt((x.astype(np.float64) ** 2 * (np.arange(topo[0]) != 77)) @ (w ** 2).T)
    err = np.abs(got - np.where(z > 0, z, 0.01 * z))
    assert np.all(err <= tol), (err / tol).max(1)
    net.free()


def _loaded(spg, tmp_path, topo, acts, prec, seed=3):
    net = spg.Network.build(topo, acts, spg.abi.WEIGHT_INITIALIZATION_HE, seed=seed)
    net.save(str(tmp_path / "m.nn"), prec)
    net.free()
    return spg.Network.load(str(tmp_path / "m.nn"))


@pytest.mark.parametrize("prec", [3, 4, 5])
def test_one_net_over_batches_of_changing_size(spg, has_gpu, tmp_path, prec):
    """The counters and sums of a net's scratch are at zero after every call, wherever the next batch's plan looks for them: a
    sequence that grows, shrinks, changes the number of groups and meets wide rows in between, on host and device buffers.
    Bound: both layers' 28 bits and fp32 rounding, eight deviations of the sums of independent errors."""
    import torch
    a = spg.abi
    topo = [4096, 4096, 130]
    net = _loaded(spg, tmp_path, topo, [a.ACT_RELU, a.ACT_LEAKY_RELU], prec)
    w = [torch.from_numpy(v.astype(np.float64)).cuda() for v in np.split(net.weights, [topo[0] * topo[1]])]
    b = [torch.from_numpy(v.astype(np.float64)).cuda() for v in np.split(net.biases, [topo[1]])]
    w = [v.view(o, i) for v, i, o in zip(w, topo, topo[1:])]
    net.set_stream(torch.cuda.current_stream().cuda_stream)
    for step, n in enumerate([200, 7, 65, 8, 256, 33, 200, 96, 97]):
        x = torch.randn(n, topo[0], generator=torch.Generator("cuda").manual_seed(n + step), device="cuda")
        if step in (2, 5):
            x[n // 2, 9] = 1e5
        if step % 2:
            got = torch.from_numpy(net.forward_batch(x.cpu().numpy())).cuda()
        else:
            got = torch.empty(n, topo[-1], device="cuda")
            net.forward_batch_ptr(x.data_ptr(), n, got.data_ptr())
            net.synchronize()
        assert spg.last_path() == "istream"
        h, tol = x.double(), torch.zeros_like(x, dtype=torch.float64)
        for w_, b_, slope in zip(w, b, (0.0, 0.01)):
            z, w2 = h @ w_.T + b_, (w_ ** 2).T
            fixed = h.abs().amax(1, keepdim=True) * 2.0 ** -27.9 * w2.sum(0).sqrt()
            # tol: of one value so far, eight deviations; the second term is the rounding of the weights compared with to fp32
            tol = 8 * (fixed + 2.0 ** -24 * (h ** 2 @ w2).sqrt()) + (tol ** 2 @ w2).sqrt() + 4e-7 * z.abs()
            h = torch.where(z > 0, z, slope * z)
        err = (got.double() - h).abs()
        assert bool((err <= tol + 1e-30).all()), (step, n, float((err / tol).max()))
    net.free()


@pytest.mark.parametrize("n", [1, 64, 200, 400])
def test_a_small_auto_batch_recomputes_no_rows(spg, has_gpu, tmp_path, n):
    """spingalett_last_repaired is about the last AUTO call, also when that one had nothing to recompute."""
    a, lib = spg.abi, spg.lib()
    net = _loaded(spg, tmp_path, [4096, 2048, 10], [a.ACT_RELU, a.ACT_SOFTMAX], 4)
    x = np.random.default_rng(n).standard_normal((2048, 4096)).astype(np.float32)
    lib.spingalett_set_auto_margin(5.0)
    try:
        for read in (True, False):
            net.forward_batch(x)
            if read:
                assert lib.spingalett_last_repaired(net._h) > 0
            net.forward_batch(x[:n])
            assert lib.spingalett_last_repaired(net._h) == 0, (read, spg.last_path())
    finally:
        lib.spingalett_set_auto_margin(0.0)
    net.free()


def test_the_rows_widths_and_modes_that_take_the_path(spg, has_gpu, tmp_path):
    """Just inside and just outside of every line that the dispatch draws."""
    a, lib = spg.abi, spg.lib()
    modes = {"auto": a.MATH_AUTO, "exact": a.MATH_EXACT, "fast": a.MATH_FAST}
    small, medium, less = [128, 64, 10], [4096, 2048], [4096, 2047]                  # 4 MB of INT4, and not quite
    soft = [a.ACT_RELU, a.ACT_SOFTMAX]
    for topo, acts, prec, rows in [
            (small, soft, 3, {("auto", 6): 0, ("auto", 7): 1, ("auto", 96): 1, ("auto", 97): 0, ("exact", 24): 1, ("exact", 25): 0, ("fast", 96): 1}),
            (small, soft, 4, {("auto", 7): 1}), (small, soft, 5, {("auto", 7): 1}), (small, soft, 1, {("auto", 7): 0}), (small, soft, 0, {("auto", 7): 0}),
            (medium, soft[1:], 4, {("auto", 97): 1, ("auto", 256): 1, ("auto", 257): 0, ("exact", 97): 0, ("fast", 97): 0}),
            (less, soft[1:], 4, {("auto", 96): 1, ("auto", 97): 0}),
            ([72, 64, 10], soft, 4, {("auto", 16): 0}),                                 # packed rows of 36 bytes
            ([128, 72, 10], soft, 4, {("auto", 16): 0}),                                # the same, in the second layer
            (small, [a.ACT_SOFTMAX, a.ACT_SOFTMAX], 4, {("auto", 16): 0})]:
        net = _loaded(spg, tmp_path, topo, acts, prec)
        for (mode, n), takes in rows.items():
            spg.set_math_mode(modes[mode])
            try:
                y = net.forward_batch(np.random.default_rng(n).standard_normal((n, topo[0])).astype(np.float32))
            finally:
                spg.set_math_mode(a.MATH_AUTO)
            assert (spg.last_path() == "istream") == bool(takes), (topo, prec, mode, n, spg.last_path())
            assert np.all(np.isfinite(y))
            if takes and n == 7:
                lib.spgk_gemv_set_int_path(0)
                try:
                    other = net.forward_batch(np.random.default_rng(n).standard_normal((n, topo[0])).astype(np.float32))
                finally:
                    lib.spgk_gemv_set_int_path(1)
                assert spg.last_path() != "istream" and np.abs(other - y).max() <= 1e-4      # two bf16 terms: 2^-17 of a value
        net.free()
