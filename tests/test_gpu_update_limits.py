"""GPU: batches that would take the edge count past int32 are refused before their
arrays are read, and leave the graph as it was."""
import ctypes as C

import numpy as np
import pytest

from dynamicgraphs_scc_b200 import Graph, SccError, State, capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_ins", [2**31 - 1 - 8, 2**31, 2**40])
def test_edge_count_past_int32_is_refused(gpu, n_ins):
    v = np.arange(8, dtype=np.int32)
    g = Graph.from_edges(8, v, (v + 1) % 8)              # 8 edges
    st = State(g)
    st.run(2)
    before = [a.copy() for a in g.csr()]
    one = capi.i32p(np.zeros(1, np.int32))               # never read
    run, upd = capi.RunStats(), capi.UpdateStats()
    for name, args in (("scc_insert_idea1", (one, one, C.byref(run))),
                       ("scc_update_batch", (one, one, 0, None, None, 0, C.byref(upd)))):
        with pytest.raises(SccError) as ei:
            capi.call(name, g.handle, st.handle, n_ins, *args)
        assert ei.value.status == 1, name                # SCC_ERR_INVALID
    for a, b in zip(g.csr(), before):
        assert np.array_equal(a, b)
    assert not st.canonical_labels().any()
    st.free(); g.free()
