"""GPU: batches of graphs whose vertices the first round sets aside for want of in- or
out-edges: acyclic graphs, self-loops, a pivot without a product of degrees, edges
that leave the graph; against Tarjan."""
import numpy as np
import pytest

from oracle import oracle as O
from dynamicgraphs_scc_b200 import BatchPlan, Graph, State
from tests.helpers import random_graph

pytestmark = pytest.mark.gpu


def check(parts):
    offs = np.concatenate([[0], np.cumsum([p[0] for p in parts])]).astype(np.int32)
    s = np.concatenate([np.asarray(p[1], np.int64) + o for p, o in zip(parts, offs)]).astype(np.int32)
    d = np.concatenate([np.asarray(p[2], np.int64) + o for p, o in zip(parts, offs)]).astype(np.int32)
    n = int(offs[-1])
    g = Graph.from_edges(n, s, d)
    st = State(g)
    plan = BatchPlan(g, st, offs)
    csr = O.build_csr(n, s, d)
    exp = O.tarjan_canonical(csr[0], csr[1])
    for _ in range(2):
        plan.run()
        assert np.array_equal(st.canonical_labels(), exp)
        assert st.count_sccs() == len(np.unique(exp))
    plan.free(); st.free(); g.free()


@pytest.mark.parametrize("n", [2, 31, 33, 1000, 20000])
def test_acyclic(gpu, n):
    i = np.arange(1, n)
    s, d = random_graph(n, 3 * n, n, self_loops=False)
    tree = (n, (i - 1) // 2, i)
    dag = (n, np.minimum(s, d), np.maximum(s, d))
    one_way = (n, s // 2, n // 2 + d // 2)                     # every product of degrees is 0
    loops = (n, np.arange(n), np.arange(n))                    # a vertex on its own loop has both degrees
    check([tree, dag, one_way, loops, (n, i, i - 1), (n, i[:0], i[:0])])


@pytest.mark.parametrize("n", [50, 3000])
def test_cycles_among_leaves(gpu, n):
    # a core, sources into it, sinks out of it, sources straight into sinks
    s, d = random_graph(n, 3 * n, 3)
    rng = np.random.default_rng(4)
    src, snk = n + np.arange(2 * n), 3 * n + np.arange(2 * n)
    check([(5 * n, np.concatenate([s, src, rng.integers(0, n, 2 * n), src]),
            np.concatenate([d, rng.integers(0, n, 2 * n), snk, rng.permutation(snk)]))] * 3)


def test_edges_that_leave_the_graph_are_no_reason_to_keep_a_vertex(gpu):
    # vertices 0..99 and 100..199: every vertex has an in- and an out-edge, but some only across the border
    a = np.arange(100)
    s = np.concatenate([a, a + 100, a[:60], a[:60] + 100]).astype(np.int32)
    d = np.concatenate([a + 100, a, (a[:60] + 1) % 60, (a[:60] + 1) % 60 + 100]).astype(np.int32)
    g = Graph.from_edges(200, s, d)
    st = State(g)
    plan = BatchPlan(g, st, np.array([0, 100, 200], np.int32))
    plan.run()
    exp = np.concatenate([np.zeros(60), a[60:], np.full(60, 100), a[60:] + 100]).astype(np.int32)
    assert np.array_equal(st.canonical_labels(), exp)
    plan.free(); st.free(); g.free()
