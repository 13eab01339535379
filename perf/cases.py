"""What the speed of this framework is measured on.

Each case is one call (or the short run of calls) that a program using the
library makes, through kclistpp_gb300's public functions: k-clique degrees,
Seq- and Sim-kClist++ passes, the trim, the clique sample, a batch of graphs
and a whole Seq run with its reports.  Graphs are the seeded synthetic ones
of the library's generators, in the families and shapes that the tests, the
benchmark and the configurations use; the schedule is the library's default.

A case's "op" says which call it is:

  count     count_cliques: the k-clique degrees of every vertex
  seq       `passes` Seq passes on a host vector (deterministic streams)
  seq_dev   `passes` Seq passes on a device vector, enqueued on the program's
            stream; `det` chooses the streams or the wave ordering
  sim       `passes` Sim passes on a host vector
  sim_dev   `passes` Sim passes on a device vector
  trim      the k-clique core trim of an edge list, the first step of a run
  main      seq_main: passes 1 .. 2^j with a report at every power of two
  sample    Seq-Sampling++: draw the sample, `passes` passes, one report
  batch     many uneven graphs, k = 3 .. kmax, one captured CUDA graph

`start` passes have been run before the timed call on the pass cases, so that
the loads are those of a run in progress (0: the run's first pass, in which
every load ties).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import kclistpp_gb300 as K


def listed() -> list[dict]:
    return [
        # The smallest call: triangle counts of a 10,000-vertex power-law graph.
        {"name": "count-small-k3", "op": "count", "graph": "chung_lu", "n": 10000, "degree": 20.0, "gamma": 2.5,
         "k": 3},
        # The parity configuration: a short Seq run from zero on that graph.
        {"name": "seq-small-k4", "op": "seq", "graph": "chung_lu", "n": 10000, "degree": 20.0, "gamma": 2.5,
         "k": 4, "start": 0, "passes": 10},
        # The headline: a Seq pass and Sim passes over a trimmed RMAT core, in
        # the middle of a run that keeps its vector on the device.
        {"name": "seq-core-k4", "op": "seq_dev", "graph": "rmat_core", "scale": 18, "factor": 16, "k": 4,
         "start": 4, "passes": 1, "det": "streams"},
        {"name": "sim-core-k4", "op": "sim_dev", "graph": "rmat_core", "scale": 18, "factor": 16, "k": 4,
         "start": 4, "passes": 2},
        # The warm-start and convergence runs: k = 5 on RMAT with planted
        # communities, the run's first pass for Seq, a later one for Sim.
        {"name": "seq-planted-k5", "op": "seq", "graph": "rmat_planted", "scale": 15, "factor": 16,
         "communities": 6, "cmin": 100, "cmax": 300, "k": 5, "start": 0, "passes": 1},
        {"name": "sim-planted-k5", "op": "sim", "graph": "rmat_planted", "scale": 15, "factor": 16,
         "communities": 6, "cmin": 100, "cmax": 300, "k": 5, "start": 2, "passes": 1},
        # Clique degrees of a whole large graph, before any trim.
        {"name": "count-large-k4", "op": "count", "graph": "rmat", "scale": 18, "factor": 16, "k": 4},
        # Wave-ordered passes over a large sparse graph, triangles: many small roots.
        {"name": "waves-large-k3", "op": "seq_dev", "graph": "rmat", "scale": 17, "factor": 16, "k": 3, "start": 1,
         "passes": 2, "det": "waves"},
        # Many uneven graphs at once, k = 3 .. 7, as the batched configuration has them.
        {"name": "batch-k3-7", "op": "batch", "graphs": 24, "nmin": 1000, "nmax": 20000, "kmax": 7, "passes": 2},
        # A sampled run: 1e6 of the 4-cliques kept, 16 passes over them, the report.
        {"name": "sample-k4", "op": "sample", "graph": "rmat", "scale": 16, "factor": 16, "k": 4,
         "target": 1000000, "passes": 16},
        # The trim that comes before the passes, whole call on host edges.
        {"name": "trim-k4", "op": "trim", "graph": "rmat", "scale": 14, "factor": 16, "k": 4},
        # A whole Seq run: 16 passes from zero, a report after passes 1, 2, 4, 8, 16.
        {"name": "main-planted-k4", "op": "main", "graph": "planted", "n": 60000, "degree": 10.0, "gamma": 2.2,
         "communities": 10, "cmin": 100, "cmax": 300, "k": 4, "passes": 16},
    ]


def _log_int(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    op = rng.choice(["count", "count", "seq", "seq", "seq_dev", "seq_dev", "sim", "sim_dev", "batch", "sample",
                     "trim", "main"])
    if op == "batch":
        return {"op": op, "graphs": rng.randint(3, 24), "nmin": 1000, "nmax": _log_int(rng, 2000, 20000),
                "kmax": rng.randint(4, 7), "passes": rng.randint(1, 2)}
    k = rng.choice([3, 4, 4, 5])
    if op in ("sample", "trim"):
        g = {"graph": "rmat", "scale": rng.randint(11, 16 if op == "sample" else 14), "factor": rng.randint(6, 16)}
    elif op == "main":
        g = {"graph": "planted", "n": _log_int(rng, 3000, 60000), "degree": round(rng.uniform(6.0, 10.0), 1),
             "gamma": 2.2, "communities": rng.randint(1, 10), "cmin": rng.randint(40, 100),
             "cmax": rng.randint(101, 300)}
    else:
        kind = rng.choice(["chung_lu", "rmat", "rmat_core", "rmat_planted"])
        if kind == "chung_lu":
            g = {"graph": kind, "n": _log_int(rng, 2000, 100000), "degree": round(rng.uniform(8.0, 32.0), 1),
                 "gamma": round(rng.uniform(2.2, 2.8), 2)}
        elif kind == "rmat_planted":
            g = {"graph": kind, "scale": rng.randint(11, 15), "factor": rng.randint(6, 16),
                 "communities": rng.randint(1, 6), "cmin": rng.randint(40, 100), "cmax": rng.randint(101, 300)}
        else:
            g = {"graph": kind, "scale": rng.randint(12, 17 if op == "count" else 16),
                 "factor": rng.randint(6, 16)}
    if op == "main" or (k == 5 and g["graph"] in ("rmat", "rmat_core") and g["scale"] > 14):
        k = 4
    c = {"op": op, **g, "k": k}
    if op == "sample":
        c.update(target=_log_int(rng, 20000, 1000000), passes=rng.randint(1, 16))
    elif op == "main":
        c.update(passes=rng.randint(2, 16))
    elif op not in ("count", "trim"):
        c.update(start=rng.choice([0, 1, 3, 6]), passes=rng.randint(1, 3))
    if op == "seq_dev":
        c["det"] = rng.choice(["streams", "streams", "waves"])
    return c


def _edges(case: dict, seed: int) -> "K.EdgeList":
    s = seed + 1
    if case["graph"] == "chung_lu":
        return K.chung_lu(case["n"], case["degree"], case["gamma"], seed=s)
    if case["graph"] == "planted":
        return K.planted(case["n"], case["degree"], case["gamma"], case["communities"], case["cmin"], case["cmax"],
                         0.5, seed=s)
    if case["graph"] == "rmat_planted":
        return K.rmat_planted(case["scale"], case["factor"], case["communities"], case["cmin"], case["cmax"], 0.5,
                              seed=s)
    return K.rmat(case["scale"], case["factor"], seed=s)


def _graph(ctx: "K.Context", case: dict, seed: int) -> "K.Graph":
    el = _edges(case, seed)
    if case["graph"] == "rmat_core":
        # the k-clique core that the trim leaves, with its own vertex numbers
        p = K.trim(ctx, el, case["k"], K.TRIM_FAST).edges.pairs()
        el = K.EdgeList.from_pairs(np.unique(p, return_inverse=True)[1].reshape(-1, 2))
    # The relabelled graph ends at its last vertex with an edge; a program that
    # keeps its own vertex set (every seed's is the same) hands the rest over too.
    off, cols = K.build_graph(ctx, el).csr()
    n = {"rmat": 1 << case.get("scale", 0), "rmat_planted": 1 << case.get("scale", 0), "rmat_core": 2048}
    n = max(n.get(case["graph"], case.get("n", 0)), len(off) - 1)
    return K.graph_from_csr(ctx, np.pad(off, (0, n + 1 - len(off)), mode="edge"), cols)


def _whole(el: "K.EdgeList", n: int) -> "K.EdgeList":
    """el with an edge to its successor for every vertex without one, so that a
    graph of the batch keeps its n vertices."""
    p = el.pairs()
    alone = np.setdiff1d(np.arange(n, dtype=np.uint32), p)
    if not len(alone):
        return el
    return K.EdgeList.from_pairs(np.concatenate([p, np.stack([alone, (alone + 1) % n], axis=1).astype(np.uint32)]))


_DET = {"streams": K.SEQ_EDGE_STREAMS, "waves": K.SEQ_WAVES}


def prepare(case: dict, seed: int) -> dict:
    op = case["op"]
    stream = torch.cuda.Stream()
    ctx = K.Context(0, stream=stream.cuda_stream)
    st = {"case": case, "stream": stream, "ctx": ctx}
    if op == "trim":
        st["el"] = _edges(case, seed)
        return st
    if op == "batch":
        rng = np.random.default_rng(case["graphs"])  # sizes: the case's; edges: the seed's
        els = []
        for i in range(case["graphs"]):
            n = int(np.exp(rng.uniform(np.log(case["nmin"]), np.log(case["nmax"]))))
            d = float(rng.uniform(8, 64))
            s = 1000 * (seed + 1) + i
            els.append(_whole(K.erdos_renyi(n, d, seed=s) if i % 2 else K.chung_lu(n, d, 2.5, seed=s), n))
        st["batch"] = K.Batch(ctx, els)
        return st
    g = st["g"] = _graph(ctx, case, seed)
    st["seed"] = seed
    if op in ("seq", "seq_dev"):
        r = K.seq_passes(g, case["k"], case["start"]) if case["start"] else np.zeros(g.n, np.uint64)
        st["r"] = r
    elif op in ("sim", "sim_dev"):
        st["r"] = K.sim_passes(g, case["k"], case["start"]) if case["start"] else np.zeros(g.n)
    if op in ("seq_dev", "sim_dev"):
        st["start"] = torch.from_numpy(st["r"].view(np.int64) if op == "seq_dev" else st["r"]).cuda()
        st["vec"] = torch.empty_like(st["start"])
        torch.cuda.synchronize()
    return st


def _padded(a: np.ndarray, n: int) -> np.ndarray:
    """a with zeros behind it: the trim's arrays have as many entries as survive."""
    out = np.zeros(n, a.dtype)
    out[: len(a)] = a
    return out


def _info(i) -> list:
    return [int(i.n), int(i.m), int(i.cliques), float(i.density), float(i.ub)]


def run(st: dict):
    case, ctx = st["case"], st["ctx"]
    op, k = case["op"], case.get("k")
    if op == "count":
        total, per = K.count_cliques(st["g"], k)
        return [total, per]
    if op == "seq":
        return K.seq_passes(st["g"], k, case["passes"], st["r"])
    if op == "sim":
        return K.sim_passes(st["g"], k, case["passes"], st["r"], t_first=case["start"] + 1)
    if op in ("seq_dev", "sim_dev"):
        with torch.cuda.stream(st["stream"]):
            st["vec"].copy_(st["start"], non_blocking=True)
        if op == "seq_dev":
            K.seq_passes_dev(st["g"], k, case["passes"], st["vec"].data_ptr(), det_mode=_DET[case["det"]])
        else:
            K.sim_passes_dev(st["g"], k, case["start"] + 1, case["passes"], st["vec"].data_ptr())
        return st["vec"]
    if op == "trim":
        t = K.trim(ctx, st["el"], k)
        n = st["el"].n
        pairs = t.edges.pairs()
        whole = [_padded(a, n) for a in (t.map, t.nck, t.order, t.core_num)]
        return whole + [_padded(pairs.reshape(-1), 2 * case["factor"] << case["scale"]), int(t.info.ntrim),
                        int(t.info.mtrim), int(t.info.total), float(t.info.ckrho)]
    if op == "main":
        infos, r = K.seq_main(st["g"], k, case["passes"])
        return [r, [_info(i) for i in infos]]
    if op == "sample":
        s = K.Sampling(st["g"], k, case["target"], seed=st["seed"] + 1, waves=8)
        s.passes(case["passes"])
        rep, order = s.extract(case["passes"])
        rho = s.rho()
        s.close()
        return [rho, order, int(rep.n), int(rep.m), int(rep.sub_cliques), float(rep.density), float(rep.ub)]
    return st["batch"].run(K.KERNEL_SEQ, list(range(3, case["kmax"] + 1)), case["passes"])


def work(case: dict) -> dict:
    """The graph read once and the vectors read and written once, per pass and
    k: the sizes the generators give (duplicates in RMAT are about a tenth)."""
    if case["op"] == "batch":
        n = case["graphs"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
        m = 18.0 * n
    elif case["graph"] == "chung_lu":
        n, m = case["n"], 0.45 * case["n"] * case["degree"]
    elif case["graph"] == "planted":
        n, c = case["n"], math.sqrt(case["cmin"] * case["cmax"])
        m = 0.45 * n * case["degree"] + case["communities"] * c * c / 4
    elif case["graph"] == "rmat_core":
        n, m = 1351 * 2.0 ** (0.22 * (case["scale"] - 20)), 494283 * 2.0 ** (0.54 * (case["scale"] - 20))
    else:
        n, m = 2.0 ** case["scale"], 0.9 * case["factor"] * 2.0 ** case["scale"]
        if case["graph"] == "rmat_planted":
            m += case["communities"] * case["cmin"] * case["cmax"] / 4
    csr = 8.0 * n + 4.0 * m
    op = case["op"]
    if op == "count":
        return {"bytes": csr + 8 * n}
    if op == "trim":
        return {"bytes": 16 * m + 36 * n}
    if op == "sample":  # the graph, then every kept clique once per pass
        return {"bytes": csr + 8 * n + case["passes"] * 4.0 * case["k"] * case["target"]}
    runs = case["passes"] * (case["kmax"] - 2 if op == "batch" else 1)
    return {"bytes": runs * (csr + 16 * n)}


def exact(case: dict, seed: int):
    """Sim's rho in 64 bits, from the definition: each 4-clique gives its unit
    to its member of smallest (rho, id), then rho = (t rho + 2 add) / (t + 2).
    Other outputs are whole numbers or follow from them."""
    if case["op"] not in ("sim", "sim_dev") or case["k"] != 4 or case["graph"] != "rmat_core":
        return None
    st = prepare(case, seed)
    off, cols = st["g"].csr()
    n = st["g"].n
    src = np.repeat(np.arange(n), np.diff(off.astype(np.int64)))
    dev = torch.device("cuda")
    A = torch.zeros((n, n), dtype=torch.float64, device=dev)
    A[torch.from_numpy(src).to(dev), torch.from_numpy(cols.astype(np.int64)).to(dev)] = 1.0
    A = A + A.T
    rho = st["r"].copy()
    for t in range(case["start"] + 1, case["start"] + 1 + case["passes"]):
        order = torch.from_numpy(np.lexsort((np.arange(n), rho))).to(dev)
        U = torch.triu(A[order][:, order], diagonal=1)
        add = torch.zeros(n, dtype=torch.float64, device=dev)
        for p in range(n):
            q = torch.nonzero(U[p]).reshape(-1)
            if len(q) >= 3:
                S = U[q][:, q]
                add[order[p]] = ((S @ S) * S).sum()
        rho = (t * rho + 2.0 * add.cpu().numpy()) / (t + 2.0)
    rho = torch.from_numpy(rho)
    return rho if case["op"] == "sim" else rho.to(dev)
