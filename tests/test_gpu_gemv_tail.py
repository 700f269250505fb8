"""A net in one launch of the weight-streaming GEMV whose layers end well short of a chunk: the tail of every layer's staged input is
cleared by all CTAs together, by fewer of them where a layer has fewer groups of 16 outputs than the device has processors."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1, 2, 3, 4, 5])
@pytest.mark.parametrize("topo", [[256, 256, 256, 9], [512, 1088, 320, 130], [320, 4096, 2432, 256, 40]], ids=["one", "few", "all"])
@pytest.mark.parametrize("n", [1, 3, 8])
def test_tails(spg, oracle, prec, topo, n):
    import torch
    k, vp = spg.lib(), C.c_void_p
    k.spgk_gemv_forward_chain.argtypes = [C.POINTER(spg.abi.KLayer), C.c_uint32, vp, C.c_uint32, C.POINTER(vp), C.c_uint32, vp, vp, vp, vp]
    k.spgk_gemv_staged_bytes.argtypes, k.spgk_gemv_staged_bytes.restype = [C.c_uint32, C.c_uint32], C.c_size_t
    k.spgk_gemv_scratch_bytes.argtypes, k.spgk_gemv_scratch_bytes.restype = [C.POINTER(spg.abi.KLayer), C.c_uint32], C.c_size_t
    k.spgk_gemv_status.argtypes = [vp, vp]
    k.spgk_error_string.restype = C.c_char_p
    rng = np.random.default_rng(n + prec)
    q = {3: 127.0, 4: 7.0, 5: 1.0}.get(prec)
    Ls, decs, biases, hold = [], [], [], []
    for inn, out in zip(topo, topo[1:]):
        raw = oracle.Oracle.encode((rng.standard_normal(out * inn) / np.sqrt(inn)).astype(np.float32), prec)
        dec = oracle.Oracle.decode(raw, out * inn, prec).astype(np.float64).reshape(out, inn)
        scale = float(np.float32(np.frombuffer(raw[:4].tobytes(), np.float32)[0] / q)) if q else 1.0
        decs.append(np.rint(dec / scale) * scale if q else dec)
        biases.append(rng.standard_normal(out).astype(np.float32) * 0.1)
        hold.append((torch.from_numpy(np.concatenate([raw[4:] if q else raw, np.zeros(256, np.uint8)])).cuda(), torch.from_numpy(biases[-1]).cuda()))
        Ls.append(spg.abi.KLayer(hold[-1][0].data_ptr(), hold[-1][1].data_ptr(), scale, inn, out, prec, 1, float(np.abs(biases[-1]).max())))
    count = len(Ls)
    x = rng.standard_normal((n, topo[0])).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    ys_t = [torch.zeros(n, o, device="cuda") for o in topo[1:]]
    # NaN in the 16-bit types wherever nothing is written
    staged = [torch.full((max(k.spgk_gemv_staged_bytes(i, n) for i in topo[:-1]),), 0xFF, dtype=torch.uint8, device="cuda") for _ in range(2)]
    scratch = torch.zeros(max(k.spgk_gemv_scratch_bytes(C.byref(L), n) for L in Ls), dtype=torch.uint8, device="cuda")
    rc = k.spgk_gemv_forward_chain((spg.abi.KLayer * count)(*Ls), count, xd.data_ptr(), topo[0], (vp * count)(*[t.data_ptr() for t in ys_t]), n,
                                   staged[0].data_ptr(), staged[1].data_ptr(), scratch.data_ptr(), None)
    assert rc == 0, k.spgk_error_string()
    assert k.spgk_gemv_status(scratch.data_ptr(), None) == 0
    a = x.astype(np.float64)
    for t, inn, dec, bias in zip(ys_t, topo, decs, biases):
        want, got = np.maximum(a @ dec.T + bias, 0), t.cpu().numpy().astype(np.float64)
        # a layer on the input that the device had: 28 bits of the row's range, or bf16 terms of it, three at one row (24 bits), else two (16)
        tol = (3e-6 if n == 1 or q else 3e-5) * max(1.0, np.abs(want).max()) * np.sqrt(max(inn, 256) / 256)
        assert np.abs(got - want).max() <= tol, (inn, np.abs(got - want).max(), tol)
        a = got
