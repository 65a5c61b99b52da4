"""GPU: the record drain after its idle warps gave up beside one warp's long chain.
The chain ends in a tree, so the warp that walked it has work to share that no
other warp is left to take; the traversal still completes.  The idle bound is
shortened by injection, so the chain takes milliseconds instead of seconds."""
import numpy as np
import pytest

from dynamicgraphs_scc_b200 import Graph, SccError, State, capi

pytestmark = pytest.mark.gpu

SCC_INJECT_WAIT, SCC_INJECT_IDLE = 2, 3


def chain_and_tree(chain, depth):
    """0 -> 1 -> ... -> chain - 1, the root of a binary tree of 2^depth - 1 vertices below it."""
    k = 2 ** depth - 1                             # tree vertex j (heap order) is chain - 1 + j
    child = np.arange(1, k)
    s = np.concatenate([np.arange(chain - 1), chain - 1 + (child - 1) // 2])
    d = np.concatenate([np.arange(1, chain), chain - 1 + child])
    return chain - 1 + k, s.astype(np.int32), d.astype(np.int32)


def inject(what, k):
    capi.call("scc_debug_inject", what, k)


@pytest.mark.parametrize("depth", [3, 8, 15])
@pytest.mark.parametrize("back", [False, True])
def test_what_is_shared_after_the_idle_warps_left(gpu, depth, back):
    # back: the leaves lead to the first vertex, so the other direction branches first and joins the chain later
    n, s, d = chain_and_tree(200000, depth)
    if back:
        leaves = np.arange(n - 2 ** (depth - 1), n, dtype=np.int32)
        s, d = np.concatenate([s, leaves]), np.concatenate([d, np.zeros_like(leaves)])
    g = Graph.from_edges(n, s, d)
    st = State(g)
    st.create_trim1_compact()
    inject(SCC_INJECT_IDLE, 64)
    try:
        found = st.do_fw_bw_global_pivot(-1, 0)
    finally:
        inject(SCC_INJECT_IDLE, 0)
    if back:
        assert found == n and not st.scc().any()
    else:
        colour = st.color()
        assert found == 1 and colour[0] == -2 and colour[1] >= 0 and (colour[1:] == colour[1]).all()
    st.free(); g.free()


def test_a_missing_item_is_still_a_timeout(gpu):
    n, s, d = chain_and_tree(100000, 10)
    g = Graph.from_edges(n, s, d)
    st = State(g)
    st.create_trim1_compact()
    inject(SCC_INJECT_IDLE, 64)
    inject(SCC_INJECT_WAIT, 1)
    try:
        with pytest.raises(SccError) as ei:
            st.do_fw_bw_global_pivot(-1, 0)
        assert ei.value.status == 4
    finally:
        inject(SCC_INJECT_IDLE, 0)
        inject(SCC_INJECT_WAIT, 0)
    st.reset()
    st.create_trim1_compact()
    assert st.do_fw_bw_global_pivot(-1, 0) == 1
    colour = st.color()
    assert colour[0] == -2 and (colour[1:] == colour[1]).all()
    st.free(); g.free()
