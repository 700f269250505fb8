"""The few-tiles tensor-core layer (spg_gemm_split.cu), reached through spgk_layer_gemm_tc for products of few tiles: sizes at
the edges of its tiles and splits, both 16-bit types, one and two planes of either operand, row counts known on the device."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TIMEOUT = -4                                           # SPGK_E_TIMEOUT
ACT = {6: lambda v: v, 1: lambda v: np.maximum(v, 0), 3: lambda v: np.where(v > 0, v, 0.01 * v), 2: np.tanh,
       0: lambda v: 1 / (1 + np.exp(-v)), 4: lambda v: np.where(v > 1, 1 + 0.01 * (v - 1), np.where(v < 0, 0.01 * v, v))}


@pytest.fixture(scope="module")
def lib(spg):
    lib, vp = spg.lib(), C.c_void_p
    lib.spgk_layer_gemm_tc.argtypes = [C.POINTER(spg.abi.KLayer), vp, C.c_uint32, C.c_uint64, C.c_int, C.c_int,
                                       vp, C.c_uint32, C.c_uint64, C.c_int, C.c_int, vp, C.c_uint32, C.c_uint64, C.c_int,
                                       vp, C.c_uint32, C.c_uint32, C.c_int, vp, vp]
    lib.spgk_gemm_tc_status.argtypes = [vp, vp]
    lib.spgk_set_dynamic_rows.argtypes = [vp, C.c_uint32]
    lib.spgk_set_output_rows.argtypes = [vp]
    lib.spgk_set_margin_sink.argtypes = [C.c_float, vp, vp]
    lib.spgk_gemm_tc_arrangement.argtypes = [C.POINTER(C.c_uint32 * 4)]
    lib.spgk_gemm_tc_arrangement.restype = None
    lib.spgk_error_string.restype = C.c_char_p
    return lib


def arrangement(lib):
    """Of the last launch: few-tiles kernel or not, columns of a tile, CTAs that share one, stages of the operand ring."""
    out = (C.c_uint32 * 4)()
    lib.spgk_gemm_tc_arrangement(C.byref(out))
    return tuple(out)


def planes(x, dt, parts):
    """x as `parts` planes of 16-bit values, rows padded to a multiple of 8 with values that must not be read as data"""
    import torch
    ld = (x.shape[1] + 7) & ~7
    out = torch.full((parts, x.shape[0], ld), 3.0, dtype=dt)
    rest = torch.from_numpy(x).double()
    for p in range(parts):
        out[p, :, :x.shape[1]] = rest.to(dt)
        rest = rest - out[p, :, :x.shape[1]].double()
    return out.cuda()


def product(spg, lib, M, N, K, a_parts, w_parts, t16, act, softmax=0, cap=None, seed=0):
    import torch
    rng = np.random.default_rng(seed)
    cap = cap or M
    dt = torch.float16 if t16 == 0 else torch.bfloat16
    a = planes(rng.standard_normal((cap, K)).astype(np.float32), dt, a_parts)
    w = planes((rng.standard_normal((N, K)) / np.sqrt(K)).astype(np.float32), dt, w_parts)
    bias = torch.from_numpy(rng.standard_normal(N).astype(np.float32)).cuda()
    layer = spg.abi.KLayer(w.data_ptr(), bias.data_ptr(), 0.75, K, N, 0, act)
    status = torch.zeros(16, dtype=torch.int32, device="cuda")
    ld, ldo = a.shape[2], (N + 7) & ~7
    A, W = [v.double().cpu().numpy()[:, :, :K] for v in (a, w)]
    x = A[0] @ W[0].T + (A[1] @ W[0].T if a_parts > 1 else 0) + (A[0] @ W[1].T if w_parts > 1 else 0)
    z = x * 0.75 + bias.double().cpu().numpy()
    size = 0.75 * (np.abs(A).sum(0) @ np.abs(W).sum(0).T) + np.abs(z)      # what the sum's rounding errors are relative to

    def run(out_parts, fails=False):
        o16 = torch.full((2, cap, ldo), 7.0, dtype=dt, device="cuda")
        o32 = torch.full((cap + 1, N), -3.0, device="cuda")
        rc = lib.spgk_layer_gemm_tc(C.byref(layer), w.data_ptr(), ld, N * ld, w_parts, t16, a.data_ptr(), ld, cap * ld, a_parts, t16,
                                    o16.data_ptr() if out_parts else None, ldo, cap * ldo, max(out_parts, 1), o32.data_ptr(), N, cap, softmax,
                                    status.data_ptr(), None)
        assert rc == 0, lib.spgk_error_string()
        rc = lib.spgk_gemm_tc_status(status.data_ptr(), None)
        assert rc == (TIMEOUT if fails else 0), (rc, lib.spgk_error_string())
        return o16.double().cpu().numpy()[:, :, :N], o32.cpu().numpy()
    run.bias = bias                                    # `layer` holds its address only
    return z, size, run


# fp32 sums of K products in any order: at most K + S + 4 roundings of 2^-24 each, relative to the sum of magnitudes; the
# tensor cores may truncate, hence 2^-23
def bound(K):
    return (K + 12) * 2.0 ** -23


SIZES = [(1, 1, 1), (1, 16, 8), (9, 17, 63), (127, 33, 64), (128, 128, 65), (129, 10, 1000), (200, 1000, 512), (256, 512, 784),
         (300, 129, 1024), (1025, 100, 129), (3001, 777, 301), (3001, 37, 129), (64, 2048, 2048), (700, 512, 512)]


@pytest.mark.parametrize("M,N,K", SIZES)
@pytest.mark.parametrize("t16,a_parts,w_parts", [(0, 1, 1), (0, 2, 1), (1, 2, 1), (1, 2, 2), (1, 1, 2)])
def test_products_of_few_tiles(spg, lib, M, N, K, t16, a_parts, w_parts):
    act = (6, 1, 3, 2, 0, 4)[(M + N + K) % 6]
    z, size, run = product(spg, lib, M, N, K, a_parts, w_parts, t16, act)
    want = ACT[act](z)
    for out_parts in (1, 2):
        o16, o32 = run(out_parts)
        assert arrangement(lib)[0] == 1
        # (1e-6: the activation's own rounding; none of them stretches a difference)
        assert np.all(np.abs(o32[:M] - want) <= bound(K) * size + 1e-6 * np.maximum(1, np.abs(want)))
        assert np.all(o32[M] == -3.0)
        eps = (2.0 ** -11 if t16 == 0 else 2.0 ** -8) ** out_parts
        tiny = 2.0 ** -24 if t16 == 0 else 0.0         # the spacing of fp16's smallest numbers
        assert np.all(np.abs(o16[:out_parts].sum(0) - o32[:M]) <= 1.01 * eps * np.abs(o32[:M]) + tiny)
        if out_parts == 1:
            assert np.all(o16[1] == 7.0)


def test_the_sizes_meet_every_arrangement(spg, lib):
    met = set()
    for M, N, K in SIZES:
        for parts in ((1, 1), (2, 1), (2, 2)):
            product(spg, lib, M, N, K, *parts, 1, 6)[2](1)
            met.add(arrangement(lib))
    columns = {a[1] for a in met}
    assert {a[0] for a in met} == {1} and {a[2] for a in met} == {1, 2, 4, 8}
    assert any(c & (c - 1) for c in columns) and any(320 % (c // 4) for c in columns)      # (of 320 threads, some have no row)
    assert min(columns) == 16 and max(columns) >= 128 and len({a[3] for a in met}) >= 3


@pytest.mark.parametrize("M,N,K", [(1, 2, 8), (130, 10, 1000), (256, 16, 64), (257, 17, 130), (500, 64, 64), (40, 128, 700), (3, 100, 256)])
def test_softmax_rows_and_their_margin(spg, lib, M, N, K):
    import torch
    z, size, run = product(spg, lib, M, N, K, 2, 1, 1, 5, softmax=1, seed=3)
    gap = np.diff(np.partition(z, N - 2, axis=1)[:, N - 2:], axis=1)[:, 0]
    theta = float(np.sort(gap)[M // 2])
    err = (bound(K) * size).max(1)
    idx, count = torch.zeros(M, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    lib.spgk_set_margin_sink(theta, idx.data_ptr(), count.data_ptr())
    try:
        _, o32 = run(0)
    finally:
        lib.spgk_set_margin_sink(0.0, None, None)
    e = np.exp(z - z.max(1, keepdims=True))
    want = e / e.sum(1, keepdims=True)
    assert np.all(np.abs(o32[:M] - want) <= want * (2 * err[:, None] + 1e-5) + 1e-7)
    listed = np.zeros(M, bool)
    listed[idx.cpu().numpy()[:int(count)]] = True
    assert int(count) == listed.sum()
    clear = np.abs(gap - theta) > 2 * err
    assert np.array_equal(listed[clear], (gap < theta)[clear])


# (tiles of 48 and 112 columns leave threads of the last warp without a row, and lanes of a warp with different numbers of rows)
@pytest.mark.parametrize("N,K", [(512, 784), (1000, 512), (10, 1000), (40, 64), (333, 777), (48, 1000), (112, 700)])
@pytest.mark.parametrize("rows", [0, 1, 300, 2900])
def test_rows_counted_on_the_device_do_not_hang_on_the_guess(spg, lib, N, K, rows):
    """The guess of the count steers tiles only: same bits for any guess, right rows scattered, nothing else written."""
    import torch
    cap = 3000
    z, size, run = product(spg, lib, rows, N, K, 2, 1, 1, 1, cap=cap, seed=rows + N)
    where = np.random.default_rng(1).permutation(cap).astype(np.int32)
    n, to = torch.tensor([rows], dtype=torch.int32, device="cuda"), torch.from_numpy(where).cuda()
    results = []
    try:
        lib.spgk_set_output_rows(to.data_ptr())
        for guess in (0, 1, 300, 3000):
            lib.spgk_set_dynamic_rows(n.data_ptr(), guess)
            results.append(run(0)[1])
    finally:
        lib.spgk_set_dynamic_rows(None, 0)
        lib.spgk_set_output_rows(None)
    for r in results[1:]:
        assert np.array_equal(results[0], r)
    assert np.all(np.abs(results[0][where[:rows]] - np.maximum(z, 0)[:rows]) <= bound(K) * size[:rows] + 1e-6)
    rest = np.ones(cap + 1, bool)
    rest[where[:rows]] = False
    assert np.all(results[0][rest] == -3.0)


@pytest.mark.parametrize("N,K", [(10, 60), (37, 64), (128, 24), (10, 1000)])
def test_a_softmax_of_counted_rows_does_not_hang_on_the_guess(spg, lib, N, K):
    """Guesses on both sides of what the device holds at once, with K in one piece and in several: same bits."""
    import torch
    cap, rows = 24000, 21000
    z, _, run = product(spg, lib, rows, N, K, 2, 1, 1, 5, softmax=1, cap=cap, seed=N)
    n = torch.tensor([rows], dtype=torch.int32, device="cuda")
    results = []
    try:
        for guess in (0, 100, 5000, 18000, 21000, cap):
            lib.spgk_set_dynamic_rows(n.data_ptr(), guess)
            results.append(run(0)[1])
            assert arrangement(lib)[0] == 1
    finally:
        lib.spgk_set_dynamic_rows(None, 0)
    for r in results[1:]:
        assert np.array_equal(results[0], r)
    e = np.exp(z - z.max(1, keepdims=True))
    assert np.abs(results[0][:rows] - (e / e.sum(1, keepdims=True))[:rows]).max() <= 1e-4
    assert np.all(results[0][rows:] == -3.0)


@pytest.mark.parametrize("N,K,rows", [(512, 784, (1500, 3072, 3073, 20000)), (256, 2048, (1500, 4096, 4700, 24000)), (128, 130, (2100, 24000)),
                                      (100, 1000, (1900, 2100, 4300)), (777, 301, (4800, 9000))])
def test_counts_beyond_what_the_device_holds_at_once(spg, lib, N, K, rows):
    """K is cut up to a count that hangs on the layer alone: same bits for any guess on either side of it, in all outputs."""
    import torch
    cap = 24000
    z, size, run = product(spg, lib, cap, N, K, 2, 1, 1, 1, seed=N)
    want = np.maximum(z, 0)
    kernels = set()
    try:
        for count in rows:
            n = torch.tensor([count], dtype=torch.int32, device="cuda")
            results = []
            for guess in (0, 100, count, cap):
                lib.spgk_set_dynamic_rows(n.data_ptr(), guess)
                results.append(run(2))
                kernels.add(arrangement(lib)[0])
            for o16, o32 in results[1:]:
                assert np.array_equal(results[0][0], o16) and np.array_equal(results[0][1], o32), count
            o16, o32 = results[0]
            assert np.all(np.abs(o32[:count] - want[:count]) <= bound(K) * size[:count] + 1e-6 * np.maximum(1, want[:count]))
            assert np.all(o32[count:] == -3.0) and np.all(o16[:, count:] == 7.0)
    finally:
        lib.spgk_set_dynamic_rows(None, 0)
    assert kernels == {0, 1}                           # few rows expected, and many


@pytest.mark.parametrize("M,N,K,softmax", [(200, 1000, 512, 0), (256, 512, 784, 0), (300, 129, 1024, 0), (64, 2048, 2048, 0), (130, 10, 1000, 1), (1, 1, 1, 0)])
def test_a_wait_that_gave_up_leaves_the_outputs_alone(spg, lib, M, N, K, softmax):
    """Every tile's wait is given up: nothing is written or listed, the status says so, and the next call is sound."""
    import torch
    z, size, run = product(spg, lib, M, N, K, 2, 1, 1, 5 if softmax else 6, softmax=softmax)
    idx, count = torch.zeros(M, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    lib.spgk_set_margin_sink(1e30, idx.data_ptr(), count.data_ptr())
    try:
        for _ in range(2):
            lib.spgk_selftest_impatient(1)
            o16, o32 = run(0 if softmax else 2, fails=True)
            assert np.all(o32 == -3.0) and np.all(o16 == 7.0) and int(count) == 0
            lib.spgk_selftest_impatient(0)
            o32 = run(0 if softmax else 2)[1][:M]
            if softmax:
                assert int(count) == M and np.allclose(o32.sum(1), 1, atol=1e-5)
                count.zero_()
            else:
                assert np.all(np.abs(o32 - z) <= bound(K) * size + 1e-6)
    finally:
        lib.spgk_selftest_impatient(0)
        lib.spgk_set_margin_sink(0.0, None, None)


@pytest.mark.parametrize("M,N,K,a_parts,few", [(1500, 2000, 256, 1, 0), (1500, 2000, 256, 2, 1), (700, 3000, 1984, 1, 1), (700, 3000, 2040, 1, 0),
                                               (1500, 2000, 4096, 2, 1), (1500, 2000, 4104, 2, 0), (130, 512, 4104, 1, 1)])
def test_long_or_wide_uncut_tiles_are_left_to_the_persistent_kernel(spg, lib, M, N, K, a_parts, few):
    z, size, run = product(spg, lib, M, N, K, a_parts, 1, 1, 6)
    o32 = run(0)[1]
    assert arrangement(lib)[0] == few
    assert np.all(np.abs(o32[:M] - z) <= bound(K) * size + 1e-6)
