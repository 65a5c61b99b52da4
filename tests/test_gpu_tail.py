"""GPU: the recursion's tail, its classes in shared memory and those that do not fit
(too many members, a long list, too many edges), against Tarjan."""
import numpy as np
import pytest

from oracle import oracle as O
from dynamicgraphs_scc_b200 import Graph, State
from tests.helpers import random_graph, seeded_graph

pytestmark = pytest.mark.gpu


def decompose(n, s, d, **tuning):
    s, d = np.asarray(s, np.int32), np.asarray(d, np.int32)
    g = Graph.from_edges(n, s, d)
    st = State(g)
    if tuning:
        st.set_tuning(**tuning)
    csr = O.build_csr(n, s, d)
    exp = O.tarjan_canonical(csr[0], csr[1])
    for _ in range(2):
        st.reset()
        st.run(2)
        assert np.array_equal(st.canonical_labels(), exp)
    st.free(); g.free()


@pytest.mark.parametrize("size", [2, 3, 31, 200, 1000, 1024, 1025, 1500])
@pytest.mark.parametrize("degree", [1.3, 2.0, 3.9, 4.1, 12.0])
@pytest.mark.parametrize("tail_class", [1024, 4096])
def test_layered_blocks(gpu, size, degree, tail_class):
    # blocks of one size joined forward: rounds leave many classes of that order for the tail
    k = max(4, 6000 // size)
    parts = [random_graph(size, int(degree * size), 17 * size + i) for i in range(k)]
    s = np.concatenate([p[0] + i * size for i, p in enumerate(parts)])
    d = np.concatenate([p[1] + i * size for i, p in enumerate(parts)])
    rng = np.random.default_rng(size)
    a, b = rng.integers(0, size * k, (2, 4 * k))
    keep = a // size < b // size
    decompose(size * k, np.concatenate([s, a[keep]]), np.concatenate([d, b[keep]]), tail_class=tail_class)


@pytest.mark.parametrize("k", [255, 256, 257, 400])
def test_long_lists(gpu, k):
    # a small cycle whose vertices also point at k vertices outside their class
    n = 3000
    s, d = random_graph(n, 2 * n, k)
    rng = np.random.default_rng(k)
    hub = rng.choice(n, 30, replace=False)
    s = np.concatenate([s, np.repeat(hub, k)])
    d = np.concatenate([d, rng.integers(0, n, 30 * k)])
    decompose(n, s, d)
    decompose(n, d, s)


@pytest.mark.parametrize("seed", [1, 2, 3, 4])
def test_low_ids_and_grids(gpu, seed):
    # colours of classes not started yet lie in the range of a class's own
    n, s, d, _ = seeded_graph(rmat_scale=9, edge_factor=3, grid_side=40 + seed, seed=seed)
    decompose(n, s, d)
