"""GPU: the compact list at the lengths where its tiles (2,048 elements), its
one-launch form (1,184 tiles) and its look-back (32 tiles a step) begin and end."""
import numpy as np
import pytest

from dynamicgraphs_scc_b200 import Graph, State

pytestmark = pytest.mark.gpu

TILE = 2048
ONE_WAVE = 148 * 8 * TILE


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, TILE - 1, TILE, TILE + 1, 32 * TILE, 33 * TILE + 5, 70 * TILE,
                               ONE_WAVE - 1, ONE_WAVE, ONE_WAVE + 1])
@pytest.mark.parametrize("share", [0.0, 0.02, 0.5, 1.0])
def test_live_list(gpu, n, share):
    rng = np.random.default_rng(n)
    color = np.where(rng.random(n) < share, 7, -2).astype(np.int32)
    g = Graph.from_edges(n, [0], [0])
    st = State(g)
    st.set_color(color)
    assert st.create_trim1_compact() == int((color == 7).sum())
    assert np.array_equal(st.trim_targets(), np.flatnonzero(color == 7))
    # from the list itself, after a part of it has finished
    color[rng.random(n) < 0.3] = -2
    st.set_color(color)
    assert st.create_trim1_compact() == int((color == 7).sum())
    assert np.array_equal(st.trim_targets(), np.flatnonzero(color == 7))
    st.reset()
    assert np.all(st.color() == -1) and np.all(st.scc() == -1) and np.all(st.wcc() == -1)
    st.free(); g.free()
