"""GPU: a round of more levels than one launch counts leaves the rest to the host."""
import numpy as np
import pytest

from dynamicgraphs_scc_b200 import Graph, State

pytestmark = pytest.mark.gpu


def test_a_chain_with_the_drains_tuned_away(gpu):
    # a cycle walked in both directions: two items a level, never a narrow frontier at async_max 1
    n = 400000
    v = np.arange(n, dtype=np.int32)
    g = Graph.from_edges(n, v, (v + 1) % n)
    st = State(g)
    st.set_tuning(async_max=1)
    r = st.run(1)
    assert r["num_sccs"] == 1 and r["first_scc_size"] == n
    assert 2**18 <= r["traversal_steps"] < 2**18 + 1000
    assert not st.canonical_labels().any()
    st.free(); g.free()
