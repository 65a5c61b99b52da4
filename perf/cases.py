"""Cases that stand for the work a user has this engine do.

Each case is one call sequence of a program that uses the package: decompose a
resident graph, decompose many small graphs in one launch, apply an edge batch
to a served graph, take a host CSR through upload, decomposition and labels
back, or build the CSR and its transpose from an edge list.  Sizes and shapes
are those of the repository's configurations, tests and benchmark: R-MAT
(a/b/c/d = .57/.19/.19/.05) of scale 12 to 24, randomly oriented grids up to
4096 x 4096 (long diameters), planted cycles, hubs of mid degree, batches of up
to 4,096 graphs, and a streamed R-MAT s22 graph.

Outputs are int32 labels, counts and CSR arrays: whole numbers, the same for any
correct implementation (labels are the smallest member id of each component,
adjacency lists are sorted).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from dynamicgraphs_scc_b200 import PIVOT_DEGREE, PIVOT_LEARNED, BatchPlan, Graph, PivotModel, State, capi

BUILD = capi.SCC_BUILD_DEDUP | capi.SCC_BUILD_NO_SELF_LOOPS


def _run(name, rmat_scale=0, edge_factor=0, grid_side=0, num_cycles=0, cycle_max=0, hubs=0, hub_deg=0, learned=False):
    """Decompose a resident graph: reset, method 2, canonical labels on the device."""
    c = {"kind": "run", "rmat_scale": rmat_scale, "edge_factor": edge_factor, "grid_side": grid_side,
         "num_cycles": num_cycles, "cycle_max": cycle_max, "hubs": hubs, "hub_deg": hub_deg, "learned": learned}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the smallest call: a graph of a few thousand vertices, where launches and host round trips count
        _run("run_s12_grid32", 12, 8, grid_side=32),
        # the small configuration: R-MAT scale 16, edge factor 8
        _run("run_s16", 16, 8),
        # the ordinary mixed graph (the benchmark's 1/16 sample): hubs and a long-diameter part together
        _run("run_s20_grid1024", 20, 16, grid_side=1024),
        # long diameters alone, a road-network or mesh shape of odd side
        _run("run_grid2501", grid_side=2501),
        # a sparse random digraph with hubs of mid degree: wide levels full of lists of 64 to 4,000 edges
        _run("run_hubs", 20, 2, hubs=7500, hub_deg=4000),
        # planted cycles with the learned pivot proposer switched on
        _run("run_s22_cycles_learned", 22, 16, num_cycles=250, cycle_max=100000, learned=True),
        # the large power-law graph
        _run("run_s24", 24, 16),
        # the headline configuration: R-MAT scale 24 and a 4096 x 4096 grid, 298.7 M edges
        _run("run_s24_grid4096", 24, 16, grid_side=4096),
        # 4,096 uneven graphs of 1,024 to 65,536 vertices in one launch
        {"name": "batch_4096", "kind": "batch", "graphs": 4096, "n_min": 1024, "n_max": 65536},
        # a streamed batch (70 % inserts, 30 % deletes, the configuration's geometric-mean size is 31,623 edges and
        # its mean 145,000) and then its inverse, on the served R-MAT s22 graph
        {"name": "update_s22", "kind": "update", "rmat_scale": 22, "edge_factor": 16, "edges": 100001},
        # end to end from pinned host memory: forward CSR in, labels out
        {"name": "e2e_s22_grid2048", "kind": "e2e", "rmat_scale": 22, "edge_factor": 16, "grid_side": 2048},
        # CSR and transpose from a device edge list, duplicates and self-loops dropped
        {"name": "build_s22", "kind": "build", "rmat_scale": 22, "edge_factor": 16, "grid_side": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rmat", "mixed", "mixed", "grid", "cycles", "hubs", "batch", "update", "e2e", "build"])
    ef = rng.randint(5, 16)
    if kind == "rmat":
        return _run(None, rng.randint(12, 24), ef)
    if kind == "mixed":
        return _run(None, rng.randint(12, 23), ef, grid_side=_log_int(rng, 32, 3000))
    if kind == "grid":
        return _run(None, grid_side=_log_int(rng, 64, 3500))
    if kind == "cycles":
        return _run(None, rng.randint(17, 23), ef, num_cycles=_log_int(rng, 10, 1000),
                    cycle_max=_log_int(rng, 1000, 100000), learned=rng.random() < 0.5)
    if kind == "hubs":
        return _run(None, rng.randint(16, 20), 2, hubs=_log_int(rng, 100, 7500), hub_deg=_log_int(rng, 400, 4000))
    if kind == "batch":
        return {"kind": "batch", "graphs": _log_int(rng, 32, 3000), "n_min": 1024, "n_max": _log_int(rng, 4096, 65536)}
    if kind == "update":
        return {"kind": "update", "rmat_scale": rng.randint(16, 22), "edge_factor": ef,
                "edges": _log_int(rng, 1000, 500000)}
    return {"kind": kind, "rmat_scale": rng.randint(14, 22), "edge_factor": ef, "grid_side": _log_int(rng, 32, 2048)}


# ---------------------------------------------------------------- inputs
class _Device:
    """A graph's device array as torch sees it (CUDA array interface); a tensor made from it
    holds on to this object and so keeps the graph alive."""

    def __init__(self, graph, ptr, n):
        self.graph = graph
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (ptr, False), "version": 3}


def _device_csr(g):
    """begin, node_idx, r_begin, r_node_idx of a graph as tensors over its own device arrays."""
    n, m = g.num_nodes(), g.num_edges()
    p = [C.c_void_p() for _ in range(4)]
    capi.call("scc_graph_device_csr", g.handle, *[C.byref(x) for x in p])
    return [torch.as_tensor(_Device(g, x.value, k), device="cuda") if k else torch.empty(0, dtype=torch.int32, device="cuda")
            for x, k in zip(p, (n + 1, m, n + 1, m))]


def _graph_from_device_edges(n, src, dst, flags=BUILD):
    h = C.c_void_p()
    torch.cuda.current_stream().synchronize()      # the edges were written on torch's stream
    capi.call("scc_graph_create_edges_device", n, src.numel(), src.data_ptr(), dst.data_ptr(), flags, 0, C.byref(h))
    return Graph(h)


def _generator_args(case, seed):
    kw = dict(rmat_scale=case["rmat_scale"], edge_factor=case["edge_factor"], grid_side=case.get("grid_side", 0),
              seed=seed + 1)
    if case.get("num_cycles"):
        kw.update(num_cycles=case["num_cycles"], cycle_min=3, cycle_max=case["cycle_max"])
    return kw


def _hub_graph(case, seed):
    """A random digraph of the given out-degree plus distinct vertices with extra out- and
    in-edges, each count uniform in [64, hub_deg), whose other ends lie in the lower half of the ids."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = 1 << case["rmat_scale"]
    k = case["hubs"]

    def ints(lo, hi, count):
        return torch.randint(lo, hi, (count,), generator=gen, device="cuda", dtype=torch.int32)

    hub = torch.randperm(n, generator=gen, device="cuda")[:k].to(torch.int32)
    deg_out, deg_in = ints(64, case["hub_deg"], k).long(), ints(64, case["hub_deg"], k).long()
    out, inn = torch.repeat_interleave(hub, deg_out), torch.repeat_interleave(hub, deg_in)
    tail = torch.arange(n, device="cuda", dtype=torch.int32).repeat_interleave(case["edge_factor"])
    src = torch.cat([tail, out, ints(0, n // 2, inn.numel())])
    dst = torch.cat([ints(0, n, tail.numel()), ints(0, n // 2, out.numel()), inn])
    return _graph_from_device_edges(n, src, dst)


def _batch_graph(case, seed):
    """Disjoint union of uneven graphs: sizes log-uniform in [n_min, n_max] (the case's own), out-degrees
    Poisson(6), targets inside the graph, 70 % uniform and 30 % as an R-MAT column falls (each id bit set
    with probability 0.24).  Returns (graph, offsets)."""
    k = case["graphs"]
    u = np.random.default_rng([k, case["n_min"], case["n_max"]]).random(k)
    sizes = np.floor(case["n_min"] * (case["n_max"] / case["n_min"]) ** u).astype(np.int64)
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    size = torch.from_numpy(sizes).cuda()
    base = torch.from_numpy(offsets[:-1]).cuda()
    n = int(offsets[-1])
    deg = torch.poisson(torch.full((n,), 6.0, device="cuda"), generator=gen).int()
    src = torch.repeat_interleave(torch.arange(n, device="cuda", dtype=torch.int32), deg)
    graph_of = torch.repeat_interleave(torch.arange(k, device="cuda", dtype=torch.int32), size)[src]
    m = src.numel()
    at = torch.zeros(m, device="cuda")                     # the target's place in its graph, in [0, 1)
    for bit in range(1, 17):
        at += (torch.rand(m, generator=gen, device="cuda") < 0.24) * 2.0 ** -bit
    uniform = torch.rand(m, generator=gen, device="cuda") < 0.7
    at = torch.where(uniform, torch.rand(m, generator=gen, device="cuda"), at)
    del uniform
    dst = base[graph_of] + torch.minimum((at * size[graph_of]).int(), (size[graph_of] - 1).int())
    return _graph_from_device_edges(n, src, dst), offsets


def _graph(case, seed):
    if case.get("hubs"):
        return _hub_graph(case, seed)
    return Graph.generate(**_generator_args(case, seed), flags=BUILD)


def _batch_edges(g, case, seed):
    """An update batch: inserts whose ends are ends of random edges (degree-proportional), new to
    the graph and distinct, and distinct existing edges to delete.  Host arrays."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = g.num_nodes()
    begin, adj, _, _ = _device_csr(g)
    src = torch.repeat_interleave(torch.arange(n, device="cuda"), (begin[1:] - begin[:-1]).long())
    keys = src * n + adj.long()                       # ascending: lists are sorted
    m = keys.numel()
    ki = max(1, int(round(0.7 * case["edges"])))
    kd = max(1, case["edges"] - ki)

    def pick(k):
        return torch.randint(0, m, (k,), generator=gen, device="cuda")

    s, d = src[pick(ki)], adj[pick(ki)].long()
    new = torch.unique((s * n + d)[s != d])
    at = torch.searchsorted(keys, new).clamp_(max=m - 1)
    new = new[keys[at] != new]
    gone = keys[torch.unique(pick(kd))]
    return [x.to(torch.int32).cpu().numpy() for x in (new // n, new % n, gone // n, gone % n)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "run":
        g = _graph(case, seed)
        st = State(g)
        s = {"kind": kind, "graph": g, "state": st, "pivot": PIVOT_DEGREE,
             "labels": torch.empty(g.num_nodes(), dtype=torch.int32, device="cuda")}
        if case["learned"]:
            s["model"] = PivotModel(seed=seed + 1)
            st.set_pivot_model(s["model"])
            s["pivot"] = PIVOT_LEARNED
        return s
    if kind == "batch":
        g, offsets = _batch_graph(case, seed)
        st = State(g)
        return {"kind": kind, "graph": g, "state": st, "plan": BatchPlan(g, st, offsets),
                "labels": torch.empty(g.num_nodes(), dtype=torch.int32, device="cuda")}
    if kind == "update":
        g = _graph(case, seed)
        st = State(g)
        st.run()
        ins_src, ins_dst, del_src, del_dst = _batch_edges(g, case, seed)
        return {"kind": kind, "graph": g, "state": st, "ins": (ins_src, ins_dst), "del": (del_src, del_dst),
                "labels": [torch.empty(g.num_nodes(), dtype=torch.int32, device="cuda") for _ in range(2)]}
    if kind == "e2e":
        g = _graph(case, seed)
        begin, adj, _, _ = _device_csr(g)
        host = [torch.empty(x.numel(), dtype=torch.int32, pin_memory=True).copy_(x) for x in (begin, adj)]
        labels = torch.empty(g.num_nodes(), dtype=torch.int32, pin_memory=True)
        return {"kind": kind, "graph": g, "state": State(g), "begin": host[0].numpy(), "adj": host[1].numpy(),
                "labels": labels.numpy(), "pinned": (host, labels)}
    # build: a fixed number of the graph's edges in a random order, 3 % of them twice, and a few self-loops
    g = _graph(case, seed)
    begin, adj, _, _ = _device_csr(g)
    n = g.num_nodes()
    src = torch.repeat_interleave(torch.arange(n, device="cuda", dtype=torch.int32), (begin[1:] - begin[:-1]).long())
    gen = torch.Generator(device="cuda").manual_seed(seed)
    keep = int(0.75 * _sizes(case)[1])
    order = torch.randperm(src.numel(), device="cuda", generator=gen)[:keep]
    again, loops = order[: int(0.03 * keep)], src[order[:: 4099]]
    src = torch.cat([src[order], src[again], loops])
    dst = torch.cat([adj[order], adj[again], loops])
    order = torch.randperm(src.numel(), device="cuda", generator=gen)
    return {"kind": kind, "n": n, "src": src[order], "dst": dst[order]}


# ---------------------------------------------------------------- one pass
def _labels_to(state, tensor):
    capi.call("scc_canonical_labels_device", state.handle, tensor.data_ptr())
    return tensor


def run(state):
    kind = state["kind"]
    if kind == "run":
        st = state["state"]
        st.reset()
        r = st.run(pivot_mode=state["pivot"])
        return {"labels": _labels_to(st, state["labels"]), "num_sccs": r["num_sccs"]}
    if kind == "batch":
        state["plan"].run()
        return {"labels": _labels_to(state["state"], state["labels"])}
    if kind == "update":
        # the batch, then its inverse, which brings the graph back to where it was
        st, ins, gone = state["state"], state["ins"], state["del"]
        a = st.update_batch(ins_src=ins[0], ins_dst=ins[1], del_src=gone[0], del_dst=gone[1])
        after = _labels_to(st, state["labels"][0])
        b = st.update_batch(ins_src=gone[0], ins_dst=gone[1], del_src=ins[0], del_dst=ins[1])
        back = _labels_to(st, state["labels"][1])
        return {"labels": after, "labels_back": back, "edges": [a["m_after"], b["m_after"]],
                "num_sccs": [a["num_sccs"], b["num_sccs"]]}
    if kind == "e2e":
        g, st, labels = state["graph"], state["state"], state["labels"]
        g.upload_csr(state["begin"], state["adj"], stream=st.stream())     # ordered before the run
        st.reset()
        r = st.run()
        capi.call("scc_canonical_labels", st.handle, capi.i32p(labels))
        return {"labels": labels, "num_sccs": r["num_sccs"]}
    g = _graph_from_device_edges(state["n"], state["src"], state["dst"])
    return dict(zip(("begin", "node_idx", "r_begin", "r_node_idx"), _device_csr(g)))


# ---------------------------------------------------------------- what a pass cannot do without
def _sizes(case):
    """Vertices and generated edges (before duplicates are dropped, a few percent)."""
    if case["kind"] == "batch":
        lo, hi = case["n_min"], case["n_max"]
        n = case["graphs"] * (hi - lo) / math.log(hi / lo)      # mean of a log-uniform size
        return n, 6.0 * n
    side = case.get("grid_side", 0)
    n = (1 << case["rmat_scale"] if case["rmat_scale"] else 0) + side * side
    m = (case["edge_factor"] << case["rmat_scale"] if case["rmat_scale"] else 0) + 2.1 * side * max(side - 1, 0)
    if case.get("num_cycles"):
        m += case["num_cycles"] * (case["cycle_max"] - 3) / math.log(case["cycle_max"] / 3)
    if case.get("hubs"):
        m += case["hubs"] * (64 + case["hub_deg"])
    return n, m


def work(case):
    n, m = _sizes(case)
    graph = 4.0 * (2 * m + 2 * n)              # CSR and transpose
    if case["kind"] == "update":               # twice: the graph read and written, the batch, the labels
        return {"bytes": 2 * (2 * graph + 8.0 * case["edges"] + 4 * n), "flops": 0}
    if case["kind"] == "build":                # the edge list read, the graph written
        return {"bytes": 8.0 * m + graph, "flops": 0}
    if case["kind"] == "e2e":                  # the forward CSR read, both written and read, the labels
        return {"bytes": 2.5 * graph + 4 * n, "flops": 0}
    return {"bytes": graph + 4 * n, "flops": 0}


def exact(case, seed):
    """Every output is a whole number."""
    return None
