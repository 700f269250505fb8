"""A whole net in one launch (spg_chain.cu) on blocks of every size around the lines where the number of epilogue warps changes: 16 rows, and
32 and 48 rows with plain epilogues and a last layer that is cut along K."""
import numpy as np
import pytest

from test_gpu_chain import Net, inputs, lib  # noqa: F401  (lib: fixture)

pytestmark = pytest.mark.gpu


class OnBlocks:
    """The library with plans of blocks of R rows on clusters of two."""

    def __init__(self, lib, R, hidden, clusters=20):
        self._lib, self._R, self._hidden, self._clusters = lib, R, hidden, clusters

    def __getattr__(self, name):
        return getattr(self._lib, name)

    def spgk_chain_plan(self, layers, count, rows, w_parts, a_parts, softmax, plan):
        rc = self._lib.spgk_chain_plan(layers, count, rows, w_parts, a_parts, softmax, plan)
        p = plan._obj
        p.C, p.R, p.clusters = 2, self._R, min(-(-rows // self._R), self._clusters)
        p.exchange_bytes = p.R * 128 * a_parts * -(-max(self._hidden) // 64)
        p.scratch_bytes = p.clusters * 2 * p.exchange_bytes
        return rc


@pytest.mark.parametrize("t16,a_parts,w_parts", [(0, 1, 1), (1, 2, 1), (1, 2, 2)])
@pytest.mark.parametrize("topology,acts", [([70, 130, 90, 33], [1, 2, 0]), ([70, 130, 90, 33], [1, 3, 2]), ([70, 90, 200], [1, 1])],
                         ids=["plain", "curved", "wide"])
def test_blocks(spg, lib, topology, acts, t16, a_parts, w_parts):  # noqa: F811
    x, xd = inputs(1003, topology[0])                          # 1003 rows: more blocks than clusters, and a last one of a part
    n = Net(spg, lib, topology, acts, t16, a_parts, w_parts, seed=5)
    want, err = n.want(x)
    first = None
    for R in (16, 32, 48, 64):
        n.lib = OnBlocks(lib, R, topology[1:-1])
        y, plan = n.run(xd)
        assert (plan.C, plan.R) == (2, R)
        assert np.all(np.abs(y - want) <= err), (R, np.max(np.abs(y - want) / err))
        first = y if first is None else first
        assert np.array_equal(y, first), R                     # no sum depends on the rows of a block


@pytest.mark.parametrize("t16,a_parts,w_parts", [(0, 1, 1), (1, 2, 1), (1, 2, 2)])
@pytest.mark.parametrize("width,sizes", [(900, (16, 32, 64)), (300, (32, 64, 96, 112))])
def test_wide_last_layers_over_many_blocks(spg, lib, width, sizes, t16, a_parts, w_parts):  # noqa: F811
    """A last layer that is not cut, of several tiles a CTA and a long epilogue, block upon block in every cluster, where one stage holds a block's whole input: its
    sums are read before the next block's products take their place."""
    x, xd = inputs(2500, 100)
    n = Net(spg, lib, [100, 130, width], [1, 2], t16, a_parts, w_parts, seed=width)
    want, err = n.want(x)
    for R in sizes:
        n.lib = OnBlocks(lib, R, [130], clusters=3)
        first, plan = n.run(xd)
        assert (plan.R, plan.clusters) == (R, 3)
        assert np.all(np.abs(first - want) <= err), (R, np.max(np.abs(first - want) / err))
        for _ in range(5):
            assert np.array_equal(n.run(xd)[0], first), R
