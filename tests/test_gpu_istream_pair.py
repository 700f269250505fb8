"""The 8-bit integer streaming kernel on pairs of CTAs: layers of at least 32 blocks an SM or 8192 inputs and more
than 32 rows a group, against float64 with the
bounds and inputs (rows of scales of their own, a zero row, a row of wide range) of the layers on single CTAs."""
import pytest

from test_gpu_istream import k, test_layer_against_float64 as layer_against_float64  # noqa: F401  (k: fixture)

pytestmark = pytest.mark.gpu


# one output into a pair's first CTA, whole pairs, two into its second; a padded group; packed rows that end inside a box
@pytest.mark.parametrize("prec", [3, 4, 5])
@pytest.mark.parametrize("out,inn,n", [(2561, 4096, 512), (1280, 8192, 450), (2434, 4160, 500), (129, 8192, 33),
                                       (1000, 8256, 65), (300, 16384, 40)])
def test_layer_of_many_blocks(spg, k, oracle, prec, out, inn, n):  # noqa: F811
    layer_against_float64(spg, k, oracle, prec, out, inn, n)
