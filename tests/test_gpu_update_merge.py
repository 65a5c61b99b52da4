"""GPU: the batch merge at the sizes where its tiles (512 old entries), warps of
offsets (128 vertices) and 33-way searches can go wrong, against gm_graph's CSR
of the updated edge list and a full Tarjan."""
import numpy as np
import pytest

from dynamicgraphs_scc_b200 import Graph, State
from tests.helpers import random_graph
from tests.test_gpu_update import apply_batch, check

pytestmark = pytest.mark.gpu


def run_batch(n, s, d, ins, dele):
    g = Graph.from_edges(n, s, d)
    st = State(g)
    st.run(2)
    stats = st.update_batch(*ins, *dele)
    s2, d2 = apply_batch(s, d, *ins, *dele)
    check(g, st, n, s2, d2)
    assert stats["m_after"] == len(s2)
    st.free(); g.free()


@pytest.mark.parametrize("m", [0, 1, 511, 512, 513, 1024, 12289])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 700])
def test_tile_and_offset_edges(gpu, m, n):
    s, d = random_graph(n, m, 7 * m + n)
    rng = np.random.default_rng(m + n)
    pick = rng.integers(0, m, min(m, 40)) if m else np.zeros(0, np.int64)
    ins = (rng.integers(0, n, 33).astype(np.int32), rng.integers(0, n, 33).astype(np.int32))
    run_batch(n, s, d, ins, (s[pick], d[pick]))


@pytest.mark.parametrize("copies", [1, 2, 5000])
def test_runs_of_copies_across_tiles(gpu, copies):
    # one hub whose list holds runs of equal entries longer than a tile, all of
    # one run deleted (asked twice), absent pairs asked beside it, equal pairs inserted
    n = 60
    s0, d0 = random_graph(n, 9000, 3)
    s = np.concatenate([s0, np.full(3 * copies, 7)]).astype(np.int32)
    d = np.concatenate([d0, np.repeat([11, 12, 13], copies)]).astype(np.int32)
    dele = (np.array([7, 7, 7, 59], np.int32), np.array([12, 12, 5, 59], np.int32))
    ins = (np.array([7, 7, 7, 0], np.int32), np.array([12, 11, 12, 0], np.int32))
    run_batch(n, s, d, ins, dele)


@pytest.mark.parametrize("what", ["only insert", "only delete", "delete all"])
def test_one_sided_batches(gpu, what):
    n, m = 3000, 20000
    s, d = random_graph(n, m, 9)
    none = (np.zeros(0, np.int32), np.zeros(0, np.int32))
    rng = np.random.default_rng(4)
    ins = (rng.integers(0, n, 1091).astype(np.int32), rng.integers(0, n, 1091).astype(np.int32))
    run_batch(n, s, d, ins if what == "only insert" else none,
              none if what == "only insert" else (s, d) if what == "delete all" else (s[::19], d[::19]))


def test_hub_among_changed_lists(gpu):
    # a vertex with 50,000 out- and in-neighbours: its lists cover many tiles
    n = 50001
    hub = np.zeros(n - 1, np.int32)
    leaf = np.arange(1, n, dtype=np.int32)
    s, d = np.concatenate([hub, leaf]), np.concatenate([leaf, hub])
    rng = np.random.default_rng(5)
    gone = rng.choice(n - 1, 700, replace=False)
    ins = (rng.integers(0, n, 500).astype(np.int32), rng.integers(0, n, 500).astype(np.int32))
    run_batch(n, s, d, ins, (s[gone], d[gone]))
