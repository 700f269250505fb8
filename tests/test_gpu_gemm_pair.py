"""The tensor-core layer on pairs of CTAs (spg_gemm_pair_kernel), reached through spgk_layer_gemm_tc for products of more tiles than the GPU has SMs:
rows, columns and k at the edges of a pair's tiles, one and two planes of either operand, row counts known on the device."""
import numpy as np
import pytest

from test_gpu_gemm_split import ACT, arrangement, bound, lib, product  # noqa: F401  (lib: fixture)

pytestmark = pytest.mark.gpu


# rows: whole pairs, one row into a pair's second CTA, one row into its first; columns: one into a second tile, whole tiles, not even an 8th of one more
@pytest.mark.parametrize("M,N,K", [(9728, 512, 512), (9601, 513, 449), (12672, 257, 520), (19073, 160, 450), (2432, 2056, 1001)])
@pytest.mark.parametrize("t16,a_parts,w_parts", [(0, 1, 1), (0, 2, 1), (1, 2, 2), (1, 1, 2)])
def test_products_of_many_tiles(spg, lib, M, N, K, t16, a_parts, w_parts):  # noqa: F811
    act = (6, 1, 3, 2, 0, 4)[(M + N + K) % 6]
    z, size, run = product(spg, lib, M, N, K, a_parts, w_parts, t16, act)
    want = ACT[act](z)
    for out_parts in (1, 2):
        o16, o32 = run(out_parts)
        assert arrangement(lib)[0] == 0 and arrangement(lib)[2] == 2
        assert np.all(np.abs(o32[:M] - want) <= bound(3 * K) * size + 1e-6 * np.maximum(1, np.abs(want)))
        assert np.all(o32[M] == -3.0)
        eps = (2.0 ** -11 if t16 == 0 else 2.0 ** -8) ** out_parts
        tiny = 2.0 ** -24 if t16 == 0 else 0.0
        assert np.all(np.abs(o16[:out_parts].sum(0) - o32[:M]) <= 1.01 * eps * np.abs(o32[:M]) + tiny)
        if out_parts == 1:
            assert np.all(o16[1] == 7.0)


@pytest.mark.parametrize("N,K,shared", [(2048, 300, {1, 2}), (8200, 200, {2})])
def test_counted_rows(spg, lib, N, K, shared):  # noqa: F811
    """Any count under any guess, on pairs (whose width hangs on the guess) and, where a guess gives few tiles, on single CTAs: same bits, nothing beyond
    the count."""
    import torch
    cap = 2600
    z, size, run = product(spg, lib, cap, N, K, 2, 1, 1, 1, seed=N)
    want = np.maximum(z, 0)
    seen = set()
    try:
        for count in (0, 1, 128, 129, 256, 257, 661, 2599):
            n = torch.tensor([count], dtype=torch.int32, device="cuda")
            results = []
            for guess in (661, 1400, 2600):
                lib.spgk_set_dynamic_rows(n.data_ptr(), guess)
                results.append(run(2))
                seen.add(arrangement(lib)[1:3])
            for o16, o32 in results[1:]:
                assert np.array_equal(results[0][0], o16) and np.array_equal(results[0][1], o32), count
            o16, o32 = results[0]
            assert np.all(np.abs(o32[:count] - want[:count]) <= bound(2 * K) * size[:count] + 1e-6 * np.maximum(1, want[:count]))
            assert np.all(o32[count:] == -3.0) and np.all(o16[:, count:] == 7.0)
    finally:
        lib.spgk_set_dynamic_rows(None, 0)
    assert {s for _, s in seen} == shared and len(seen) >= 2, seen
