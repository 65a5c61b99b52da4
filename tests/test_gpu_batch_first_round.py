"""GPU: the batched launch's first round (marks in shared memory, top-down levels
and sweeps) at the shapes where it can go wrong, against Tarjan."""
import numpy as np
import pytest

from oracle import oracle as O
from dynamicgraphs_scc_b200 import BatchPlan, Graph, State
from tests.helpers import random_graph

pytestmark = pytest.mark.gpu


def union(parts):
    """Disjoint union of (n, src, dst) parts: (offsets, src, dst)."""
    offs = np.concatenate([[0], np.cumsum([p[0] for p in parts])]).astype(np.int32)
    s = np.concatenate([np.asarray(p[1], np.int32) + o for p, o in zip(parts, offs)])
    d = np.concatenate([np.asarray(p[2], np.int32) + o for p, o in zip(parts, offs)])
    return offs, s.astype(np.int32), d.astype(np.int32)


def check(parts, tuning=None):
    offs, s, d = union(parts)
    n = int(offs[-1])
    g = Graph.from_edges(n, s, d)
    st = State(g)
    plan = BatchPlan(g, st, offs, tuning=tuning)
    csr = O.build_csr(n, s, d)
    exp = O.tarjan_canonical(csr[0], csr[1])
    for _ in range(2):
        plan.run()
        assert np.array_equal(st.canonical_labels(), exp)
    plan.free(); st.free(); g.free()


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 511, 513, 4099])
@pytest.mark.parametrize("degree", [0.4, 1.5, 6.0, 20.0])
def test_sizes_and_densities(gpu, n, degree):
    # several graphs of one size: their lists start at every offset modulo 4, the last
    # ones end at the end of the adjacency arrays
    check([(n, *random_graph(n, int(degree * n) + k, 11 * n + k)) for k in range(5)])


def test_shapes(gpu):
    i = np.arange(3000, dtype=np.int32)
    hub = np.zeros(3000, np.int32)
    star = (3001, np.concatenate([hub, i[:1500] + 1]), np.concatenate([i + 1, hub[:1500]]))
    deep = (3000, i, (i + 1) % 3000)                        # one long cycle
    path = (3000, i[:-1], i[1:])                            # no cycle at all
    in_star = (3001, i + 1, hub)                            # a hub nobody reaches
    # 100 vertices of 700 out- and in-neighbours: more block-wide lists in a level than it sets aside
    rng = np.random.default_rng(3)
    big = np.repeat(np.arange(100, dtype=np.int32), 700)
    many = (5000, np.concatenate([big, rng.integers(0, 5000, big.size)]),
            np.concatenate([rng.integers(0, 5000, big.size), big]))
    empty = (0, i[:0], i[:0])
    check([star, deep, empty, path, in_star, many, (1, i[:1], i[:1]), empty])
    check([star, many, deep], tuning=dict(threads=64, blocks_per_sm=8, warp_deg=1))
    check([star, many, deep], tuning=dict(threads=1024, blocks_per_sm=1, warp_deg=64))


@pytest.mark.parametrize("n", [204800, 204801])
def test_around_the_shared_memory_limit(gpu, n):
    check([(n, *random_graph(n, 4 * n, 5)), (100, *random_graph(100, 300, 6))])


def test_edges_leaving_a_graph_are_ignored(gpu):
    # two ranges of one strongly connected graph: each is decomposed as its induced subgraph
    n = 600
    s, d = random_graph(n, 3000, 8)
    g = Graph.from_edges(n, s, d)
    st = State(g)
    plan = BatchPlan(g, st, np.array([0, 250, n], np.int32))
    plan.run()
    same = (s < 250) == (d < 250)
    csr = O.build_csr(n, s[same], d[same])
    assert np.array_equal(st.canonical_labels(), O.tarjan_canonical(csr[0], csr[1]))
    plan.free(); st.free(); g.free()
