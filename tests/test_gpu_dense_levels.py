"""GPU: the level-by-level traversal that graphs above 128 edges per vertex take, at
the list lengths where its block-wide expansion (bulk copies of 1,024 entries,
unaligned starts, unstaged tails), its edge-parallel hubs and its sweeps can go
wrong.  Three layers in a ring; a vertex has one edge to its partner in the
next layer, at a random place of a list of 100 or more entries inside its own layer, so a
layer is reached whole only if every list is read whole.  Against Tarjan."""
import numpy as np
import pytest

from oracle import oracle as O
from dynamicgraphs_scc_b200 import Graph, State

pytestmark = pytest.mark.gpu


def layers(width, degree, seed):
    """Three layers in random id order; every 40th vertex a hub of up to 4,000 entries,
    three of them of 6,000, in each direction; 64 vertices that only one layer reaches."""
    rng = np.random.default_rng(seed)
    n = 3 * width + 64
    s, d = [], []
    for k in range(3):
        lo = k * width
        v = lo + np.arange(width)
        s.append(np.repeat(v, degree)); d.append(lo + rng.integers(0, width, width * degree))
        s.append(v); d.append((k + 1) % 3 * width + rng.permutation(width))
        hub = v[::40]
        more = rng.integers(100, 4000, hub.size)
        more[:3] = 6000
        s.append(np.repeat(hub, more)); d.append(lo + rng.integers(0, width, more.sum()))
        s.append(lo + rng.integers(0, width, more.sum())); d.append(np.repeat(hub, more))
    s.append(rng.integers(0, width, 64)); d.append(3 * width + np.arange(64))
    name = rng.permutation(n)
    s, d = name[np.concatenate(s)].astype(np.int32), name[np.concatenate(d)].astype(np.int32)
    return n, s, d


@pytest.fixture(scope="module")
def graphs():
    out = {}
    for width, degree in ((700, 140), (38000, 100)):     # edge-parallel; levels of more than 148 blocks
        n, s, d = layers(width, degree, width)
        csr = O.build_csr(n, s, d)
        assert s.size > 128 * n
        out[width] = (n, s, d, O.tarjan_canonical(csr[0], csr[1]))
    return out


@pytest.mark.parametrize("width", [700, 38000])
@pytest.mark.parametrize("tuning", [dict(bu_alpha=1, cta_deg=64), dict(bu_alpha=1, cta_deg=99), dict(bu_alpha=1, cta_deg=1024),
                                    dict(bu_alpha=1, cta_deg=-1), dict(bu_alpha=1, cta_deg=64, huge_deg=65),
                                    {}, dict(bu_alpha=1 << 20, bu_div=48)])
def test_every_list_is_read_whole(gpu, graphs, width, tuning):
    n, s, d, exp = graphs[width]
    g = Graph.from_edges(n, s, d)
    st = State(g)
    st.set_tuning(**tuning)
    for method in (0, 2):
        st.reset()
        r = st.run(method)
        assert np.array_equal(st.canonical_labels(), exp), method
        assert r["num_sccs"] == len(np.unique(exp))
    st.free(); g.free()
