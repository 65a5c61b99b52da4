"""GPU: batches whose graphs do not all keep the first round's marks in shared memory:
none of them, or the largest of those that do beside larger ones, against Tarjan."""
import numpy as np
import pytest

from oracle import oracle as O
from dynamicgraphs_scc_b200 import BatchPlan, Graph, State
from tests.helpers import random_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[204801, 204804], [204801, 3001, 50], [300000, 204800, 204797], [210000, 0, 1]])
def test_graphs_above_the_shared_memory_limit(gpu, sizes):
    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    parts = [random_graph(max(k, 1), 3 * k, 5 + i) for i, k in enumerate(sizes)]
    s = np.concatenate([p[0] + o for p, o in zip(parts, offs)]).astype(np.int32)
    d = np.concatenate([p[1] + o for p, o in zip(parts, offs)]).astype(np.int32)
    n = int(offs[-1])
    g = Graph.from_edges(n, s, d)
    st = State(g)
    plan = BatchPlan(g, st, offs)
    csr = O.build_csr(n, s, d)
    exp = O.tarjan_canonical(csr[0], csr[1])
    for _ in range(2):
        plan.run()
        assert np.array_equal(st.canonical_labels(), exp)
    plan.free(); st.free(); g.free()
