"""GPU: the record drain's scratch under the serving budget.  A session whose budget
has room for its requests but not for that scratch is served by the plain drain; with
room, by the record drain; never refused for it, and the labels are Tarjan's."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SERVE = """
import sys
import numpy as np
from oracle import oracle as O
from dynamicgraphs_scc_b200 import Graph, Server
from tests.helpers import seeded_graph
from tests.test_gpu_update import apply_batch
slack, ample = int(sys.argv[1]), int(sys.argv[2])
n, s, d, _ = seeded_graph(grid_side=300, seed=7)
m = len(s)
resident = 8 * (n + 1) + 8 * m + 148 * n + 4096
rng = np.random.default_rng(3)
pick = rng.integers(0, m, 500)
batch = (rng.integers(0, n, 500).astype(np.int32), rng.integers(0, n, 500).astype(np.int32), s[pick], d[pick])
update = 10 * (m + 500) + 64 * 1000 + 16 * n + (1 << 20)
sv = Server(num_slots=2, hbm_budget_bytes=ample or resident + update + slack)
sid = sv.add_graph(Graph.from_edges(n, s, d))
assert sv.wait(sv.submit(sid, *batch))["status"] == 0
sv.drain()
s2, d2 = apply_batch(s, d, *batch)
csr = O.build_csr(n, s2, d2)
assert np.array_equal(sv.labels(sid), O.tarjan_canonical(csr[0], csr[1]))
st = sv.stats()
assert st["rejected"] == 0 and st["completed"] == 1
assert st["bytes_in_use"] == 8 * (n + 1) + 8 * len(s2) + 148 * n + 4096
sv.free()
"""


def serve(slack=0, ample=0):
    """Record drains of a session's decomposition and one update, as the trace counts them."""
    r = subprocess.run([sys.executable, "-c", SERVE, str(slack), str(ample)], cwd=ROOT, capture_output=True, text=True,
                       env={**os.environ, "SCC_TRACE": "1"}, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return sum("reach records live=" in line for line in r.stderr.splitlines())


def test_the_budget_covers_the_drain(gpu):
    assert serve(slack=1 << 20) == 0            # the scratch of 90,000 vertices is 8.7 MB
    assert serve(ample=8 << 30) >= 2
