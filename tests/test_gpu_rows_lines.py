"""Which nets of more than 8 Mi weights the small-net kernel takes (one to eight rows): on either side of the lines, and right on both."""
import pytest

from test_gpu_rows import test_a_sample_from_host_memory_gives_what_a_batch_of_one_gives as check_sample
from test_gpu_rows import test_which_nets_go_there as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("topo,precision,n,rows", [
    # floats the GEMV takes: 32 Mi in a layer at one row; 10 Mi a layer in three layers
    ([4096, 8192, 8], "bf16", 1, True), ([4096, 8200, 8], "bf16", 1, False), ([4096, 2560, 4096, 2560], "fp16", 2, True), ([4096, 2560, 4096, 2576], "fp16", 2, False),
    # rows that end on half a lane's values
    ([1772, 1772, 1772, 1772], "fp32", 8, True), ([1780, 1780, 1780, 1780], "fp32", 8, False),
    # integers that stream: 4 Mi a layer and 16 Mi in all, at two and three rows
    ([2048, 2048, 2048, 2048], "int8", 3, True), ([2048, 2048, 2048, 2064], "int8", 3, False), ([2048, 2048, 2048, 2048], "int4", 4, False), ([2048, 2048, 2048, 2048], "int2", 1, False),
    # rows for the general kernel: 18 Mi in a layer
    ([4008, 4704, 16], "int4", 1, True), ([4008, 4712, 16], "int4", 8, False), ([3000, 6300, 10], "int2", 6, False),
    # odd rows: 3 Mi a layer, 12 Mi at two, three and eight rows
    ([1777, 1770, 1770, 1770], "int8", 5, True), ([1777, 1777, 1777, 1777], "int8", 6, False), ([3001, 4003, 13], "int4", 3, True), ([3001, 4003, 13], "int4", 4, False),
    ([5003, 5029, 13], "int4", 8, False), ([1777, 1770, 1770, 1770], "fp32", 8, True), ([1777, 1770, 1770, 1770], "fp32", 4, False), ([1777, 1770, 1770, 1770], "fp32", 6, False)])
def test_which_large_nets_go_there(spg, tmp_path, topo, precision, n, rows):
    check(spg, tmp_path, topo, precision, n, rows)


@pytest.mark.parametrize("topo", [[2048, 2048, 2048, 1000], [4096, 2560, 100]])
def test_a_sample_of_a_large_net(spg, topo):
    check_sample(spg, topo, 5)
