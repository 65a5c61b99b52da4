"""GPU: rounds in one cooperative launch, at the list lengths where its chunks
begin and end, with one and with many classes, on both sides of the mean degree up
to which it is taken, and ending in a drain, against Tarjan."""
import numpy as np
import pytest

from oracle import oracle as O
from dynamicgraphs_scc_b200 import Graph, PivotModel, State, collect_pivot_records  # noqa: F401
from tests.helpers import random_graph, seeded_graph

pytestmark = pytest.mark.gpu


def decompose(n, s, d, method=2, **tuning):
    s, d = np.asarray(s, np.int32), np.asarray(d, np.int32)
    g = Graph.from_edges(n, s, d)
    st = State(g)
    if tuning:
        st.set_tuning(**tuning)
    csr = O.build_csr(n, s, d)
    exp = O.tarjan_canonical(csr[0], csr[1])
    for _ in range(2):
        st.reset()
        r = st.run(method)
        assert np.array_equal(st.canonical_labels(), exp)
        assert r["num_sccs"] == len(np.unique(exp))
    st.free(); g.free()


@pytest.mark.parametrize("k", [255, 256, 257, 1023, 1024, 1025, 2048, 5000])
@pytest.mark.parametrize("bu_alpha", [1, 14, 1 << 20])
def test_list_lengths(gpu, k, bu_alpha):
    # a random digraph with ten vertices of k out- and k in-edges; bu_alpha 1: top-down
    # levels only, 2^20: sweeps from the second level on
    n = 20000
    s, d = random_graph(n, 2 * n, k)
    rng = np.random.default_rng(k + 1)
    hub = rng.choice(n, 10, replace=False)
    s = np.concatenate([s, np.repeat(hub, k), rng.integers(0, n, 10 * k)])
    d = np.concatenate([d, rng.integers(0, n, 10 * k), np.repeat(hub, k)])
    decompose(n, s, d, bu_alpha=bu_alpha)


@pytest.mark.parametrize("degree", [100, 127, 129, 200])
def test_dense_graphs(gpu, degree):
    # the chunk list has room up to a mean degree of 128; denser graphs go level by level
    n = 300
    decompose(n, *random_graph(n, degree * n, degree))


@pytest.mark.parametrize("method", [0, 1, 2])
def test_many_classes(gpu, method):
    # 64 blocks joined by one-way edges, each a random digraph: many classes a round
    m, k = 300, 64
    parts = [random_graph(m, 3 * m, 50 + i) for i in range(k)]
    s = np.concatenate([p[0] + i * m for i, p in enumerate(parts)])
    d = np.concatenate([p[1] + i * m for i, p in enumerate(parts)])
    rng = np.random.default_rng(2)
    a, b = rng.integers(0, m * k, (2, 2000))
    keep = a // m < b // m
    decompose(m * k, np.concatenate([s, a[keep]]), np.concatenate([d, b[keep]]), method)


@pytest.mark.parametrize("n", [2, 63, 64, 65, 1000])
def test_small_and_narrow(gpu, n):
    v = np.arange(n)
    decompose(n, v, (v + 1) % n)                                     # narrow levels end in the plain drain
    decompose(n, *random_graph(n, 3 * n, n))
    nn, s, d, _ = seeded_graph(rmat_scale=8, edge_factor=6, grid_side=16, seed=n)
    decompose(nn, s, d)


@pytest.mark.parametrize("k", [8 * 1024, 8 * 1024 + 1, 9 * 1024 - 1, 600000])
@pytest.mark.parametrize("back", [0, 1, 2])
def test_hub_lists(gpu, k, back):
    # a cycle of 19 with a hub of k out- and k in-neighbours, lists that a lane or its
    # warp enters into the chunk list.  back 0: the neighbours peel off and the 19 stay live;
    # 1: every out-neighbour returns through the cycle; 2: half of them do
    c = np.arange(19)
    out, inn = 19 + np.arange(k), 19 + k + np.arange(k)
    s = np.concatenate([c, np.zeros(k, np.int64), inn])
    d = np.concatenate([(c + 1) % 19, out, np.zeros(k, np.int64)])
    if back:
        s, d = np.concatenate([s, out[::back]]), np.concatenate([d, out[::back] % 19])
    decompose(19 + 2 * k, s, d)
