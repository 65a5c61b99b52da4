"""GPU: the record drain meets class vertices that the live list does not hold, in the
first frontier (next to the pivot, or the pivot itself) and in runs of up to
three, after calls that leave different contents in its scratch.  A cycle through half
of the ids with chains into it and out of it: a start at a wrong vertex reaches
another set.  Compared with a breadth-first search on the host."""
import numpy as np
import pytest
from scipy.sparse import csr_matrix
from scipy.sparse.csgraph import breadth_first_order

from dynamicgraphs_scc_b200 import Graph, State

pytestmark = pytest.mark.gpu

N = 60000


def cycle_with_chains(seed):
    """A cycle of N/2 vertices in random id order; the rest are chains of 500, half of them leading
    into the cycle and half out of it.  Returns (src, dst, the cycle's order)."""
    order = np.random.default_rng(seed).permutation(N)
    cyc, rest = order[: N // 2], order[N // 2:]
    s, d = [cyc], [np.roll(cyc, -1)]
    for i, c in enumerate(rest.reshape(-1, 500)):
        s.append(c[:-1]); d.append(c[1:])
        at = cyc[(997 * i) % cyc.size]
        s.append([c[-1]] if i % 2 else [at])
        d.append([at] if i % 2 else [c[0]])
    return np.concatenate(s).astype(np.int32), np.concatenate(d).astype(np.int32), cyc


def reach(s, d, pivot):
    m = csr_matrix((np.ones(s.size, np.int8), (s, d)), shape=(N, N))
    out = []
    for a in (m, m.T.tocsr()):
        r = np.zeros(N, bool)
        r[breadth_first_order(a, pivot, return_predecessors=False)] = True
        out.append(r)
    return out


@pytest.mark.parametrize("before", ["nothing", "peel", "canonical"])
@pytest.mark.parametrize("run", [[1], [-1], [1, 2], [1, 2, 3], [0], [4000, 4001], [4000, 4001, 4002, 9000], [1, -1, 15000]])
def test_unlisted_vertices_in_the_frontier(gpu, before, run):
    # run: places on the cycle, counted from the pivot, that the list does not hold
    s, d, cyc = cycle_with_chains(len(run))
    g = Graph.from_edges(N, s, d)
    st = State(g)
    if before == "peel":
        st.do_global_trim1()
        st.reset()
    elif before == "canonical":
        st.run(2)
        st.canonical_labels()
        st.reset()
    p = 100
    gone = cyc[[(p + x) % cyc.size for x in run]]
    colour = np.full(N, -1, np.int32)
    colour[gone] = -2
    st.set_color(colour)
    st.create_trim1_compact()
    st.set_color(np.full(N, -1, np.int32))
    found = st.do_fw_bw_global_pivot(-1, int(cyc[p]))
    fw, bw = reach(s, d, int(cyc[p]))
    listed = np.ones(N, bool)
    listed[gone] = False
    assert found == int((fw & bw & listed).sum())
    scc, colour = st.scc(), st.color()
    assert np.array_equal((scc == cyc[p])[listed], (fw & bw)[listed])
    only_fw, only_bw = fw & ~bw & listed, bw & ~fw & listed
    assert len(np.unique(colour[only_fw])) == 1 and len(np.unique(colour[only_bw])) == 1
    assert (colour[listed & ~fw & ~bw] == -1).all()
    assert colour[only_fw][0] != colour[only_bw][0] and colour[only_fw][0] >= 0 and colour[only_bw][0] >= 0
    st.free(); g.free()
