"""GPU: the CSR build's packed keys at the vertex counts where their width changes,
with self-loops, repeats and the edge (n-1, n-1) whose key is all ones, against
gm_graph's CSR; ids outside the range are refused."""
import numpy as np
import pytest

from oracle import oracle as O
from dynamicgraphs_scc_b200 import Graph, SccError, capi
from tests.helpers import random_graph

pytestmark = pytest.mark.gpu

KEEP, DEDUP, NO_SELF = 0, capi.SCC_BUILD_DEDUP, capi.SCC_BUILD_NO_SELF_LOOPS


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 255, 256, 257, 65535, 65536, 65537, (1 << 20) + 1])
@pytest.mark.parametrize("flags", [KEEP, DEDUP, NO_SELF, DEDUP | NO_SELF])
def test_widths(gpu, n, flags):
    s, d = random_graph(n, 9000, n)
    last = np.full(5, n - 1, np.int32)
    s, d = np.concatenate([s, last, s[:100]]), np.concatenate([d, last, d[:100]])
    g = Graph.from_edges(n, s, d, flags=flags)
    if flags & NO_SELF:
        keep = s != d
        s, d = s[keep], d[keep]
    if flags & DEDUP:
        k = np.unique(s.astype(np.int64) << 32 | d)
        s, d = (k >> 32).astype(np.int32), (k & 0xFFFFFFFF).astype(np.int32)
    for got, exp in zip(g.csr(), O.build_csr(n, s, d)):
        assert np.array_equal(got, exp)
    g.free()


@pytest.mark.parametrize("bad", [-1, 100, 1 << 30])
def test_ids_outside_the_range(gpu, bad):
    s, d = random_graph(100, 50, 1)
    for a, b in ((bad, 3), (3, bad), (bad, bad)):
        with pytest.raises(SccError) as ei:
            Graph.from_edges(100, np.append(s, a), np.append(d, b), flags=DEDUP | NO_SELF)
        assert ei.value.status == 1
