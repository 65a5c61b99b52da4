"""GPU: sorts of at most one tile (4,096 elements, one block) and just above it, seen
through what they order: the CSR of small edge lists, their transposes, the batch keys of
an update, and the classes of the recursion's tail; canonical labels of
components whose representative is their largest, smallest or no member."""
import numpy as np
import pytest

from oracle import oracle as O
from dynamicgraphs_scc_b200 import Graph, State
from tests.helpers import random_graph
from tests.test_gpu_update import apply_batch, check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 31, 32, 511, 512, 513, 4095, 4096, 4097, 8193])
@pytest.mark.parametrize("n", [2, 300, 70000])
def test_csr_and_transpose(gpu, m, n):
    s, d = random_graph(n, m, m + n)
    g = Graph.from_edges(n, s, d)
    for got, exp in zip(g.csr(), O.build_csr(n, s, d)):
        assert np.array_equal(got, exp)
    g.free()


@pytest.mark.parametrize("k", [(1, 0), (0, 1), (1023, 1024), (1024, 1024), (1025, 1024), (3000, 10)])
def test_update_keys(gpu, k):
    # 2 (inserts + deletes) keys in one sort: one tile holds 4,096
    n = 5000
    s, d = random_graph(n, 9000, 1)
    rng = np.random.default_rng(sum(k))
    ins = (rng.integers(0, n, k[0]).astype(np.int32), rng.integers(0, n, k[0]).astype(np.int32))
    pick = rng.integers(0, len(s), k[1])
    g = Graph.from_edges(n, s, d)
    st = State(g)
    st.run(2)
    st.update_batch(*ins, s[pick], d[pick])
    check(g, st, n, *apply_batch(s, d, *ins, s[pick], d[pick]))
    st.free(); g.free()


@pytest.mark.parametrize("n", [1, 2, 300, 100003])
def test_canonical_labels_of_given_representatives(gpu, n):
    rng = np.random.default_rng(n)
    g = Graph.from_edges(n, [0], [0])
    st = State(g)
    cls = rng.integers(0, max(1, n // 3), n)
    cls[rng.random(n) < 0.5] = 0                       # one giant component
    first = np.full(n + 1, n, np.int64)
    np.minimum.at(first, cls, np.arange(n))
    last = np.zeros(n + 1, np.int64)
    np.maximum.at(last, cls, np.arange(n))
    for rep in (first[cls], last[cls], cls):           # the last: an id that need not be a member
        st.set_scc(rep.astype(np.int32))
        assert np.array_equal(st.canonical_labels(), first[cls])
    part = np.where(rng.random(n) < 0.2, -1, last[cls]).astype(np.int32)
    st.set_scc(part)
    want = np.full(n, -1)
    low = np.full(n + 1, n, np.int64)
    np.minimum.at(low, cls[part >= 0], np.arange(n)[part >= 0])
    want[part >= 0] = low[cls[part >= 0]]
    assert np.array_equal(st.canonical_labels(), want)
    st.free(); g.free()
