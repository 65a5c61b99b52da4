"""GPU: the record drain (sparse rounds with a long way to go) at the shapes where
its records and its queue can go wrong, against Tarjan: chains, cycles, grids,
vertices of exactly four, five, eight and nine class neighbours, long lists,
repeated edges and self-loops, neighbours outside the live list, a frontier that is
handed back, the injected wait."""
import numpy as np
import pytest

from oracle import oracle as O
from dynamicgraphs_scc_b200 import Graph, SccError, State, capi
from tests.helpers import seeded_graph

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


def ring(n):
    v = np.arange(n)
    return v, (v + 1) % n


@pytest.mark.parametrize("side", [129, 200, 301])
@pytest.mark.parametrize("tuning", [{}, {"async_max": 1}, {"async_max": 1 << 20}])
def test_grids(gpu, side, tuning):
    # async_max 1: the drain is entered late and hands back at 65,536 items; 2^20: it takes any frontier
    n, s, d, _ = seeded_graph(grid_side=side, seed=side)
    decompose(n, s, d, **tuning)


@pytest.mark.parametrize("n", [8193, 20000, 70001])
def test_rings_and_chains(gpu, n):
    s, d = ring(n)
    decompose(n, s, d)
    decompose(n, np.concatenate([s, d]), np.concatenate([d, s]))          # both ways
    decompose(n, s[:-1], d[:-1])                                          # no cycle


@pytest.mark.parametrize("k", [3, 4, 5, 7, 8, 9, 63, 64, 65, 200])
def test_vertices_of_k_neighbours_on_a_ring(gpu, k):
    # every 500th vertex of a long ring also points at k - 1 others (and one at itself), repeated edges among them
    n = 30000
    s, d = ring(n)
    rng = np.random.default_rng(k)
    hub = np.arange(0, n, 500)
    t = (hub[:, None] + rng.permutation(5000)[None, : k - 1] + 2) % n
    s2 = np.concatenate([s, np.repeat(hub, k - 1), hub[:3], np.repeat(hub, k - 1)[: 2 * k]])
    d2 = np.concatenate([d, t.reshape(-1), hub[:3], t.reshape(-1)[: 2 * k]])
    decompose(n, s2, d2)
    decompose(n, d2, s2)


def test_many_classes_of_long_cycles(gpu):
    # 40 rings joined by one-way edges: each round's wave runs through many classes at once
    m, k = 2000, 40
    s = np.concatenate([ring(m)[0] + i * m for i in range(k)])
    d = np.concatenate([ring(m)[1] + i * m for i in range(k)])
    rng = np.random.default_rng(1)
    a, b = rng.integers(0, m * k, (2, 3000))
    lo, hi = np.minimum(a, b) // m, np.maximum(a, b) // m
    keep = lo < hi
    decompose(m * k, np.concatenate([s, np.minimum(a, b)[keep]]), np.concatenate([d, np.maximum(a, b)[keep]]))


def test_neighbour_outside_the_live_list(gpu):
    # the phase calls take colours as the caller sets them: a class vertex that the
    # compact list does not hold is still walked through
    n = 40000
    s, d = ring(n)
    g = Graph.from_edges(n, s.astype(np.int32), d.astype(np.int32))
    st = State(g)
    done = np.full(n, -1, np.int32)
    done[[5, 17, 20000]] = -2
    st.set_color(done)
    st.create_trim1_compact()
    st.set_color(np.full(n, -1, np.int32))
    found = st.do_fw_bw_global_pivot(-1, 100)
    assert found == n - 3           # every listed vertex is reached both ways through the others
    st.free(); g.free()


def test_wait_limit_reports_timeout_and_recovers(gpu):
    n, s, d, csr = seeded_graph(grid_side=200, seed=3)
    g = Graph.from_edges(n, s, d)
    st = State(g)
    capi.call("scc_debug_inject", 2, 1)
    try:
        with pytest.raises(SccError) as ei:
            st.run(2)
        assert ei.value.status == 4
    finally:
        capi.call("scc_debug_inject", 2, 0)
    st.reset()
    st.run(2)
    assert np.array_equal(st.canonical_labels(), O.tarjan_canonical(csr[0], csr[1]))
    st.free(); g.free()
