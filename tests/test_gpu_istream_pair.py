"""The 8-bit integer streaming kernel on pairs of CTAs: layers of more than 32 rows a group of which a CTA alone would have at least 16 blocks in
a row, against float64 with the bounds and inputs (rows of scales of their own, a zero row, a row of wide range) of the layers on single
CTAs; and layers of both kinds on one scratch buffer."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_istream import _bound, _layer, k, test_layer_against_float64 as layer_against_float64  # noqa: F401  (k: fixture)

gpu = pytest.mark.gpu


def arrangement(spg, prec, out, inn, n, sms=0):
    """CTAs that share a tile, batch rows a group, tiles, CTAs; None where the kernel does not take the layer."""
    lib = spg.lib()
    lib.spgk_istream_arrangement.argtypes = [C.POINTER(spg.abi.KLayer), C.c_uint32, C.c_uint32, C.POINTER(C.c_uint32)]
    got = (C.c_uint32 * 4)()
    layer = spg.abi.KLayer(None, None, 1.0, inn, out, prec, 6)
    return tuple(got) if lib.spgk_istream_arrangement(C.byref(layer), n, sms, got) else None


@pytest.mark.parametrize("prec,out,inn,n,pair", [
    (4, 1000, 8192, 64, 1), (4, 1000, 7936, 64, 0),           # a tile in four pieces: 16 blocks a CTA, and 15.5
    (4, 18944, 2048, 64, 1), (4, 18816, 2048, 64, 0),         # 148 tiles: 16 a CTA; 147
    (5, 1000, 8192, 33, 1), (5, 1000, 8192, 32, 0), (5, 1000, 8192, 128, 1), (5, 129, 8192, 64, 1), (5, 128, 8192, 64, 0),
    (3, 1000, 8192, 64, 0), (3, 1000, 8192, 66, 1), (4, 1000, 8192, 65, 1), (3, 1000, 8064, 66, 0)])
def test_which_layers_go_to_pairs(spg, prec, out, inn, n, pair):
    shared, rows, tiles, ctas = arrangement(spg, prec, out, inn, n, sms=148)
    assert shared == 1 + pair and rows % (8 if pair else 4) == 0 and rows * -(-n // 64) >= n
    assert tiles == -(-out // (128 << pair)) * -(-n // 64) and ctas <= 148 and ctas % shared == 0


@pytest.mark.parametrize("prec", [3, 4, 5])
@pytest.mark.parametrize("out,inn,n,shared", [
    (128 * 2 * 682, 4096, 192, 2),                            # 2046 pairs' tiles: two counters each
    (128 * 2 * 682 + 1, 4096, 192, 1),                        # 2049, and 4095 of single CTAs
    (128 * 1365, 4096, 192, 1), (128 * 1365 + 1, 4096, 192, None), (128 * 4096, 64, 32, 1), (128 * 4096 + 1, 64, 32, None)])
def test_layers_of_as_many_tiles_as_there_are_counters(spg, prec, out, inn, n, shared):
    got = arrangement(spg, prec, out, inn, n, sms=148)
    assert (got and got[0]) == shared and (not got or got[2] * got[0] <= 4096)


# one output into a pair's first CTA, whole pairs, two into its second; a padded group; packed rows that end inside a box
@gpu
@pytest.mark.parametrize("prec", [3, 4, 5])
@pytest.mark.parametrize("out,inn,n", [(2561, 4096, 512), (1280, 8192, 450), (2434, 4160, 500), (129, 8192, 33),
                                       (1000, 8256, 65), (300, 16384, 40)])
def test_layer_of_many_blocks(spg, k, oracle, prec, out, inn, n):  # noqa: F811
    pair = arrangement(spg, prec, out, inn, n)[0] == 2
    assert pair == (prec != 3 or n > 64)
    layer_against_float64(spg, k, oracle, prec, out, inn, n)


@gpu
@pytest.mark.parametrize("prec", [3, 4, 5])
def test_layers_of_both_kinds_on_one_scratch_buffer(spg, k, oracle, prec):  # noqa: F811
    """65 rows: groups of 40 where pairs of CTAs share a tile, of 36 where they do not; sums and counters lie in other slots."""
    import torch
    rng = np.random.default_rng(prec)
    topo, n = [8192, 1024, 576, 8192, 640], 65
    assert [arrangement(spg, prec, o, i, n)[:2] for i, o in zip(topo, topo[1:])] == [(2, 40), (1, 36), (1, 36), (2, 40)]
    built = [_layer(spg, oracle, rng, o, i, prec, 6) for i, o in zip(topo, topo[1:])]
    layers = (spg.abi.KLayer * 4)(*[b[0] for b in built])
    ys_t = [torch.zeros(n, o, device="cuda") for o in topo[1:]]
    ys = (C.c_void_p * 4)(*[t.data_ptr() for t in ys_t])
    scratch = torch.zeros(k.spgk_istream_scratch_bytes(layers, 4, n), dtype=torch.uint8, device="cuda")
    for seed in (1, 2):                                       # the second call finds what the first one left
        x = np.random.default_rng(seed).standard_normal((n, topo[0])).astype(np.float32)
        xd = torch.from_numpy(x).cuda()
        assert k.spgk_istream_forward(layers, 4, xd.data_ptr(), topo[0], ys, n, scratch.data_ptr(), None) == 0, k.spgk_error_string()
        assert k.spgk_istream_status(scratch.data_ptr(), None) == 0, k.spgk_error_string()
        a = x.astype(np.float64)
        for t, (_, dec, bias, _) in zip(ys_t, built):         # every layer on what the one before gave
            got, want = t.cpu().numpy(), a @ dec.T + bias
            assert np.all(np.abs(got - want) <= _bound(a, dec, want))
            a = got.astype(np.float64)
