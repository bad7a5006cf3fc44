"""The work a user of this framework has it do, as timed cases.

Graphs are the seeded synthetic workloads of the benchmark configurations
(Erdos-Renyi, R-MAT with edge factor 16, Chung-Lu with exponent 2.1 and mean
degree 40, batches of Barabasi-Albert graphs), from the smallest request to
the benchmark graph, through the public entry points: the whole-path calls,
the batched call, preprocessing and the drop-in operators.  Every result is a
whole number, so results are equal or they are wrong; there is no floating
output to compare with a 64-bit value.

A case names its graph ("graph" is the generator's seed).  The seed of
prepare() permutes the vertex ids, as R-MAT workloads do: ranks of vertices of
equal degree, edge positions and list contents all change with it, while the
sizes of the results stay those of the case.
"""
import math

import numpy as np
import torch

from tdtdecomposition_gb300 import CSRCOO, batch, generators as G, graph as GR, truss, trusstensor as tt
from tdtdecomposition_gb300 import workloads
from tdtdecomposition_gb300.preprocess import group_offsets, preprocess_edges

LIST_BUDGET = 24 << 30  # the fixed list tail a serving loop gives its requests


def _rmat(scale, draws):
    return {"gen": "rmat", "scale": scale, "draws": draws, "graph": 1}


def listed():
    return [
        # one small graph, the default call: latency of launches and of the
        # peel's sub-rounds
        dict(_er(4096, 65536), name="decompose_er_4096", op="decompose", lists="auto"),
        # a served request of ordinary size: the list tail is a fixed budget
        # (R-MAT scale 16, a draw count that is no power of two)
        dict(_rmat(16, 1000003), name="decompose_rmat_16_served", op="decompose", lists="budget"),
        # the largest served request
        dict(_rmat(20, 16 << 20), name="decompose_rmat_20", op="decompose", lists="auto"),
        # the single-graph benchmark workload, full peel to the maximum k
        dict(_rmat(22, 16 << 22), name="decompose_rmat_22", op="decompose", lists="auto"),
        # many small graphs of uneven size in one run
        {"name": "decompose_batch_ba_512", "op": "batch", "gen": "ba_batch", "graphs": 512, "graph": 1000},
        # a skewed graph whose triangle lists do not fit beside what the
        # program already holds: the peel searches the adjacency
        dict(_chung_lu(1000000), name="decompose_chung_lu_1m_search", op="decompose", lists="none"),
        # a served k-truss query: fixed-level search without lists
        dict(_rmat(18, 16 << 18), name="ktruss_rmat_18_k10", op="ktruss", k=10, lists="none"),
        # triangle count with per-edge support of a large graph
        dict(_rmat(21, 16 << 21), name="triangles_rmat_21", op="triangles"),
        # preprocessing of one small edge list, and of the benchmark graph
        dict(_er(4096, 65536), name="preprocess_er_4096", op="preprocess"),
        dict(_rmat(22, 16 << 22), name="preprocess_rmat_22", op="preprocess"),
        # the drop-in operators as the host-driven flow calls them (two tiles):
        # the support count, and the peel update of one sub-round
        dict(_rmat(18, 16 << 18), name="op_support_rmat_18", op="op_support", n_cut=2),
        dict(_rmat(17, 16 << 17), name="op_update_rmat_17", op="op_update", n_cut=2, share=0.1),
    ]


def _er(n, m):
    return {"gen": "er", "n": n, "draws": m, "graph": 1}


def _chung_lu(n):
    return {"gen": "chung_lu", "n": n, "draws": 20 * n, "graph": 2}


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["decompose", "decompose", "decompose", "batch", "ktruss", "ktruss", "triangles", "preprocess",
                     "preprocess", "op_support", "op_update"])
    if op == "batch":
        return {"op": op, "gen": "ba_batch", "graphs": _log_uniform(rng, 16, 512), "graph": rng.randrange(1 << 20)}
    # a k-truss query asks about a graph that has one
    gen = rng.choice(["rmat", "rmat", "chung_lu"] if op == "ktruss" else ["er", "rmat", "rmat", "chung_lu"])
    if gen == "er":
        n = _log_uniform(rng, 512, 1 << 15)
        c = _er(n, int(n * rng.uniform(4, 24)))
    elif gen == "rmat":
        scale = rng.randint(10, 20)
        c = _rmat(scale, int((1 << scale) * rng.uniform(8, 16)))
    else:
        c = _chung_lu(_log_uniform(rng, 1 << 10, 1 << 19))
    c["op"] = op
    c["graph"] = rng.randrange(1 << 20)
    if op == "decompose":
        c["lists"] = rng.choice(["auto", "auto", "budget", "none"])
    elif op == "ktruss":
        c["k"] = rng.randint(3, 10)
        c["lists"] = rng.choice(["auto", "none"])
    elif op == "op_support":
        c["n_cut"] = rng.randint(1, 4)
    elif op == "op_update":
        c["n_cut"] = rng.randint(1, 4)
        c["share"] = round(rng.uniform(0.01, 0.3), 3)
    return c


def _edges(case, seed):
    """Raw edge list (int32 CUDA tensors), before preprocessing, and for a
    batch the graph of each vertex id."""
    group = None
    if case["gen"] == "ba_batch":
        s, d, vg = workloads.ba_batch_edges(case["graphs"], seed=case["graph"])
        src, dst, group = (torch.from_numpy(x).cuda() for x in (s, d, vg))
        n = group.numel()
    elif case["gen"] == "er":
        n = case["n"]
        s, d = G.er_edges(n, case["draws"], seed=case["graph"])
        src, dst = torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda()
    elif case["gen"] == "rmat":
        n = 1 << case["scale"]
        src, dst = G.rmat_edges_device(case["scale"], case["draws"], seed=case["graph"])
    else:
        n = case["n"]
        src, dst = G.chung_lu_edges_device(n, seed=case["graph"], m=case["draws"])
    rnd = torch.rand(n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
    perm = torch.argsort(rnd if group is None else group + rnd).to(torch.int32)  # within each graph of a batch
    return perm[src.long()], perm[dst.long()], group


def prepare(case, seed):
    op = case["op"]
    src, dst, group = _edges(case, seed)
    if op == "batch":
        g, verts = preprocess_edges(src, dst, group)
        vo, eo = group_offsets(group, verts, g)
        return {"op": op, "batch": batch.batch_from_union(g, eo, vo)}
    if op == "preprocess":
        return {"op": op, "src": src, "dst": dst}
    g, _ = preprocess_edges(src, dst)
    st = {"op": op, "graph": g}
    if op == "decompose":
        st["kw"] = {"auto": {}, "none": {"lists": False}, "budget": {"list_budget": LIST_BUDGET}}[case["lists"]]
    elif op == "ktruss":
        st["k"] = case["k"]
        st["kw"] = {} if case["lists"] == "auto" else {"lists": False}
    elif op in ("op_support", "op_update"):
        n_cut = case["n_cut"]
        st["n_cut"] = n_cut
        st["graph"] = CSRCOO(columns=g.columns, rows=g.rows, row_ptr=GR.tiling_row_ptr(g, n_cut))
        if op == "op_update":
            # one sub-round: the `share` of the edges with the lowest support
            # is peeled; affected are the edges from or into their tails
            sup = torch.zeros_like(g.columns)
            tt.segment_isin2tile(g.rows, g.columns, st["graph"].row_ptr, n_cut, sup)
            l = int(torch.sort(sup).values[int(case["share"] * (sup.numel() - 1))])
            curr = sup <= l
            tails = torch.zeros(g.num_vertices, dtype=torch.bool, device=sup.device)
            tails[g.rows[curr].long()] = True
            st["affect"] = torch.where(tails[g.columns.long()] | tails[g.rows.long()])[0].to(torch.int32)
            st["alive"] = ~curr
            st["support"] = sup
            st["l"] = l
    return st


def run(st):
    op = st["op"]
    if op == "decompose":
        r = truss.truss_decompose(st["graph"], **st["kw"])
        return {"truss": r.truss, "e_truss": r.e_truss, "ptr_truss": r.ptr_truss, "kmax": r.kmax,
                "triangles": r.triangles, "rounds": r.rounds}
    if op == "batch":
        r = batch.decompose(st["batch"])
        return {"truss": r.truss, "kmax": r.kmax}
    if op == "ktruss":
        return truss.ktruss_search(st["graph"], st["k"], **st["kw"])
    if op == "triangles":
        t, sup = truss.triangle_count(st["graph"], return_support=True)
        return {"triangles": t, "support": sup}
    if op == "preprocess":
        g, verts = preprocess_edges(st["src"], st["dst"])
        return {"rows": g.rows, "columns": g.columns, "row_ptr": g.row_ptr, "vertices": verts}
    g = st["graph"]
    if op == "op_support":
        out = torch.zeros_like(g.columns)
        if st["n_cut"] > 1:
            tt.segment_isin2tile(g.rows, g.columns, g.row_ptr, st["n_cut"], out)
        else:
            tt.segment_isin2(g.rows, g.columns, g.row_ptr, out)
        return out
    sup = st["support"].clone()
    n_mark = torch.zeros_like(st["alive"])
    if st["n_cut"] > 1:
        tt.sub_AllAffectedSupport_tilenot(st["affect"], g.rows, g.columns, g.row_ptr, st["n_cut"], st["alive"],
                                          st["l"], n_mark, sup)
    else:
        tt.sub_AllAffectedSupport_not(st["affect"], g.rows, g.columns, g.row_ptr, st["alive"], st["l"], n_mark, sup)
    # how far below the level a support falls depends on the order of the
    # decrements; the flow only asks whether it is at or below it
    return {"support": sup.clamp_(min=st["l"]), "n_mark": n_mark}


def work(case):
    """Bytes of inputs read once and outputs written once (E edges after
    deduplication, about nine tenths of the draws; V vertices)."""
    if case["op"] == "batch":
        n, m = workloads.ba_batch_params(case["graphs"])
        draws, V = float(np.sum(n * m)), float(np.sum(n))
    else:
        draws, V = float(case["draws"]), float(case.get("n") or (1 << case["scale"]) * 0.6)
    E = 0.9 * draws
    csr = 8 * E + 8 * V  # rows, columns, row offsets
    return {"bytes": {"decompose": csr + 8 * E, "batch": csr + 4 * E, "ktruss": csr + E, "triangles": csr + 4 * E,
                      "preprocess": 8 * draws + csr + 4 * V, "op_support": csr + 4 * E,
                      "op_update": csr + 15 * E}[case["op"]], "flops": 0}
