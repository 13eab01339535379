"""Benchmark: k-cliques/s of the KClist++ "++" pass on one GB300.

Workload (the headline configuration): RMAT scale 20, (a, b, c, d) =
(0.57, 0.19, 0.19, 0.05), edge factor 16, symmetrised and deduplicated
(15.7 M edges), k-clique core trimmed at k first; then the degeneracy DAG of
the trimmed graph.  One step = one Seq-kClist++ pass (per-root-edge streams)
plus one Sim-kClist++ pass at k (default 4), i.e. every k-clique of the graph
is processed twice.  Inputs are resident in HBM when the timed region starts;
the trimmed graph fits in L2, so L2 is flushed (a 256 MiB write) before every
timed step.

    python bench.py [--gpus N --steps K --warmup W] [--impl reference] [--k 4]

`--impl reference` times the reference algorithm on the host cores instead:
the CPU port of kCDensestNoAtom's and kCDensestCmpSync's passes (the oracle,
with the reference's own p-thread schedule), each step a bounded sample of
root edges of the same workload.

The graph preparation (generation, trim, DAG) is not timed; the trim counts
cliques on the GPU in both arms.

The JSON line also carries: the pass-level roofline (warp instructions of the
Seq pass over its time, against the issue peak; beside it the reference's
per-root-edge gather bytes over the same time), the host-buffer run through the C ABI (`e2e`, the same
passes from the same state), the CPU port's rate (`cpu_baseline`), clocks
sampled during the timed region, and `convergence`: wall time to a certified
1 % density gap on a held-out RMAT-16 graph with planted communities (k = 5)
for the zero start, the learned warm start and the wave ordering
(`--no-convergence` skips it).  `--workload batch` measures the batched
configuration instead (many uneven graphs x k = 3..7 in one captured CUDA
graph) and prints its own line; `--workload sampling` times Seq-Sampling++
(count, 10^7-clique sample, "++" passes over it, one report) on the untrimmed
RMAT graph of `--scale`.
"""
from __future__ import annotations

import argparse
import json
import math
import os
import statistics
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "k-cliques/sec"
UNIT = "k-cliques/s"
L2_FLUSH_BYTES = 256 << 20


def log(*a):
    print(*a, file=sys.stderr, flush=True)


# ---------------------------------------------------------------------------
# workload
GOLDEN_TRIM = os.path.join(ROOT, "tests", "golden", "rmat20_trim.json")


def golden_trim(scale: int, k: int, seed: int) -> dict | None:
    """The reference program's trim of this graph (kClistCoreTrim run on it,
    tests/golden/make_golden_rmat20.py), where one was recorded."""
    if scale != 20 or seed != 1 or not os.path.exists(GOLDEN_TRIM):
        return None
    return json.load(open(GOLDEN_TRIM)).get(str(k))


def induce_kept(pairs: np.ndarray, kept_in_label_order: list) -> np.ndarray:
    """The reference's trimmed edge list from the input pairs and its kept
    vertices in the order of its new labels: the input edges with both ends
    kept, in input order, each with its end of larger label first
    (relabelnodes and printdensest, kClistCoreTrim.c:274-294, 686-699)."""
    n = int(pairs.max()) + 1 if len(pairs) else 1
    lab = np.full(n, -1, dtype=np.int64)
    lab[np.asarray(kept_in_label_order, dtype=np.int64)] = np.arange(len(kept_in_label_order))
    sel = pairs[(lab[pairs[:, 0]] >= 0) & (lab[pairs[:, 1]] >= 0)]
    swap = lab[sel[:, 0]] < lab[sel[:, 1]]
    out = sel.copy()
    out[swap] = sel[swap][:, ::-1]
    return np.ascontiguousarray(out, dtype=np.uint32)


def prepare_workload(K, ctx, scale: int, k: int, seed: int, cache_dir: str) -> dict:
    """RMAT -> the exact k-clique-core trim (the reference's peel, GPU recounts)
    -> trimmed edge list (cached on disk), checked against the reference
    program's own trim of the same graph where it was recorded."""
    os.makedirs(cache_dir, exist_ok=True)
    path = os.path.join(cache_dir, f"rmat{scale}_ef16_s{seed}_k{k}_trim_exact.npz")
    if os.path.exists(path):
        z = np.load(path, allow_pickle=False)
        return {"pairs": z["pairs"], "meta": json.loads(str(z["meta"]))}
    t0 = time.time()
    el = K.rmat(scale, 16, 0.57, 0.19, 0.19, seed=seed)
    tg = time.time() - t0
    t0 = time.time()
    tr = K.trim(ctx, el, k, K.TRIM_EXACT)
    tt = time.time() - t0
    pairs = tr.edges.pairs()
    i = tr.info
    meta = dict(rmat_vertices=int(el.n), rmat_edges=int(el.e), k_core_vertices=int(i.n2), k_core_edges=int(i.e2),
                cliques_before_trim=int(i.total), trimmed_vertices=int(i.ntrim), trimmed_edges=int(i.mtrim),
                trimmed_cliques=int(i.ncktrim), trim_density=float(i.ckrho), k_clique_core_number=int(i.ckcore),
                gen_s=round(tg, 2), trim_s=round(tt, 2), trim_mode="exact (the reference's heap peel, GPU recounts)",
                peel=tr.peel.as_dict())
    gold = golden_trim(scale, k, seed)
    if gold is not None:
        meta["trim_matches_reference"] = bool(
            (i.n2, i.e2, i.total, i.ckcore, i.ntrim, i.mtrim, i.ncktrim) ==
            (gold["n2"], gold["e2"], gold["total"], gold["ckcore"], gold["ntrim"], gold["mtrim"], gold["ncktrim"])
            and "%f" % i.ckrho == gold["ckrho"]
            and np.array_equal(pairs, induce_kept(el.pairs(), gold["kept_in_label_order"])))
        meta["reference_trim_seconds"] = gold.get("reference_seconds")
    tmp = path + ".tmp.npz"
    np.savez(tmp, pairs=pairs, meta=np.array(json.dumps(meta)))
    os.replace(tmp, path)
    return {"pairs": pairs, "meta": meta}


def reference_workload(scale: int, k: int, seed: int) -> dict | None:
    """The same trimmed edge list for the reference arm, built without the
    library: the oracle's restatement of the RMAT generator and the reference
    program's recorded kept set (tests/golden/rmat20_trim.json)."""
    from oracle import oracle as O

    gold = golden_trim(scale, k, seed)
    if gold is None:
        return None
    t0 = time.time()
    P = O.rmat(scale, 16, 0.57, 0.19, 0.19, seed=seed)
    pairs = induce_kept(P, gold["kept_in_label_order"])
    meta = dict(rmat_vertices=int(P.max()) + 1, rmat_edges=int(len(P)), k_core_vertices=gold["n2"],
                k_core_edges=gold["e2"], cliques_before_trim=gold["total"], trimmed_vertices=gold["ntrim"],
                trimmed_edges=gold["mtrim"], trimmed_cliques=gold["ncktrim"], trim_density=float(gold["ckrho"]),
                k_clique_core_number=gold["ckcore"], gen_s=round(time.time() - t0, 2),
                trim_mode="the reference program's own trim of this graph (recorded kept set)")
    return {"pairs": pairs, "meta": meta}


def dag_stats(off: np.ndarray, cols: np.ndarray, k: int, s_max: int = 64, split1: int = 256,
              split2: int = 512) -> dict:
    """Algorithmic bytes by tier.

    "bytes" is the per-root-edge figure of the reference's MakeSubgraph
    (kCDensestNoAtom.c:86-113) summed over the root edges of every root in the
    tier: 8 + 4(d+s + d+t) + 4 sum_{x in C(s,t)} d+x + 8(|C(s,t)| + 2) per root
    edge (the root edge, both root lists, the induced-subgraph gathers, the r
    gathers of the candidates and of s, t).  "impl_bytes" is what this
    implementation's per-root induction needs at least: every out-list of
    N+(s) once per root, plus r of {s} and N+(s) read and written.
    s_max, split1 and split2 are the schedule's tier bounds (kclpp_schedule)."""
    n = len(off) - 1
    deg = np.diff(off).astype(np.int64)
    src = np.repeat(np.arange(n, dtype=np.int64), deg)
    dst = cols.astype(np.int64)
    out_bytes_sum = np.zeros(n, dtype=np.int64)  # sum_{x in N+(s)} (16 + 4 d+(x))
    np.add.at(out_bytes_sum, src, 16 + 4 * deg[dst])
    impl_root = 16 + 4 * deg + out_bytes_sum + 8 * (deg + 1) + 8 * (deg + 1)
    active = deg >= max(1, k - 1)
    edge_root = None
    ref_equiv = None
    if n <= 30000:
        A = np.zeros((n, n), dtype=np.float32)
        A[src, dst] = 1.0
        C = np.einsum("ij,ij->i", A[src], A[dst]).astype(np.int64)           # |N+(s) ∩ N+(t)|
        Ad = A * deg[None, :].astype(np.float32)
        SD = np.einsum("ij,ij->i", Ad[src], A[dst]).astype(np.int64)          # sum_{x in C(s,t)} d+(x)
        per_edge = 8 + 4 * (deg[src] + deg[dst]) + 4 * SD + 8 * (C + 2)
        edge_root = np.zeros(n, dtype=np.int64)
        np.add.at(edge_root, src, per_edge)
        ref_equiv = int(8 * (n + 1) + per_edge.sum() + 16 * n)

    def bucket(d):
        if d <= s_max:
            return ("S", 0)
        if d <= split1:
            return ("M", split1)
        if d <= split2:
            return ("M", split2)
        if d <= 1024:
            return ("M", 1024)
        return ("L", 2048)

    tiers = {}
    for s in np.nonzero(deg > 0)[0]:
        key = bucket(int(deg[s]))
        t = tiers.setdefault(key, {"roots": 0, "bytes": 0, "impl_bytes": 0, "dmax": 0})
        t["roots"] += 1
        t["dmax"] = max(t["dmax"], int(deg[s]))
        if active[s]:
            t["impl_bytes"] += int(impl_root[s])
        if edge_root is not None:
            t["bytes"] += int(edge_root[s])
    return {"tiers": tiers, "ref_equiv_bytes_per_pass": ref_equiv, "n": n, "m": int(len(cols))}


PASS_COUNTERS = os.path.join(ROOT, "profiles", "seq_sim_pass_rmat20_k4_counters.txt")


def profiled(counter: str, kernel: str, a=None):
    """A per-pass counter of `kernel` ("seq" or "sim") on this workload, read
    from the committed ncu summary (a "<counter> <kernel> <value>" line):
    dram_bytes_per_pass, l2_bytes_per_pass, warp_inst_per_pass.  The summary
    was measured on the default workload (RMAT scale 20, seed 1, k = 4); for
    any other (`a`, the parsed arguments) there is no counter (None)."""
    if a is not None and (a.scale, a.seed, a.k) != (20, 1, 4):
        return None
    try:
        with open(PASS_COUNTERS) as f:
            for line in f:
                p = line.split()
                if len(p) == 3 and p[0] == counter and p[1] == kernel:
                    return int(p[2])
    except OSError:
        pass
    return None


# ---------------------------------------------------------------------------
# clocks during the timed region
class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.file = None

    def start(self):
        try:
            self.file = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=self.file, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self) -> dict:
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        time.sleep(0.25)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        self.file.flush()
        self.file.seek(0)
        rows = [r.split(",") for r in self.file.read().strip().splitlines() if r.strip()]
        os.unlink(self.file.name)
        sm, mx, reasons, power = [], [], set(), []
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in rows:
            r = [x.strip() for x in r]
            if len(r) < 9:
                continue
            try:
                sm.append(float(r[1]))
                mx.append(float(r[2]))
                power.append(float(r[3]))
            except ValueError:
                continue
            for nm, v in zip(names, r[5:9]):
                if v.lower() == "active":
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(sm),
                "power_w_max": max(power) if power else None}


def measured_peaks() -> tuple[float, str]:
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(p) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


# ---------------------------------------------------------------------------
# CPU legs (the oracle: the reference algorithm ported to a C library)
def cpu_sample(pairs: np.ndarray, k: int, modes: list[str], seconds: float, threads: int) -> dict:
    """Time the reference algorithm on a bounded sample of root edges."""
    from oracle import oracle as O

    og = O.Graph(pairs)
    r = np.zeros(og.n, dtype=np.uint64)
    rho = np.zeros(og.n, dtype=np.float64)

    def run(stride):
        cl, t = 0, 0.0
        for md in modes:
            t0 = O.wtime()
            if md == "seq":
                cl += og.seq_pass_sample(k, r.copy(), O.SEQ_THREADS, threads, stride)
            else:
                cl += og.sim_counts_sample(k, rho, threads, stride)
            t += O.wtime() - t0
        return cl, t

    stride = max(1, og.m // 64)
    cl, t = run(stride)
    while t < seconds / 8 and stride > 1:
        stride = max(1, int(stride * max(0.1, t / (seconds / 2))) if t > 0 else stride // 8)
        cl, t = run(stride)
    return {"cliques": cl, "seconds": t, "stride": stride, "edges": (og.m + stride - 1) // stride,
            "m": og.m, "threads": threads}


# ---------------------------------------------------------------------------
def convergence(ctx, gap: float = 0.01, max_passes: int = 400, scale: int = 16, train_graphs: int = 16,
                labels: tuple = ("zero", "warm", "waves", "shared", "warm_shared")) -> dict:
    """Wall time to a certified density gap on a held-out graph: the zero-start
    Seq run (per-root-edge streams) against the learned warm start, the
    wave-ordered passes, the shared-load passes (KCLPP_SEQ_SHARED) and the
    warm start with shared-load passes.  The network is trained here on
    zero-start runs of `train_graphs` seeded graphs of the same families
    (planted Chung-Lu and RMAT with planted communities, k = 5, half each);
    evaluation is on an RMAT graph of `scale` with planted communities that
    the training never saw.  Every pass is followed by the extraction (sort,
    PAVA pass, upper bound) that certifies the gap, inside the timed region."""
    import kclistpp_gb300 as K
    from kclistpp_gb300 import warm as W

    k = 5
    t0 = time.perf_counter()
    half = max(1, train_graphs // 2)
    train = [K.planted(6000 + 1000 * (i % 8), 8.0, 2.2, 3, 60, 160, 0.6, seed=100 + i) for i in range(half)]
    train += [K.rmat_planted(13 + (i % 3), 16, 4, 60, 300, 0.5, seed=200 + i) for i in range(train_graphs - half)]
    X, Y = W.training_set(ctx, train, k, passes=64)
    model = W.WarmModel(ctx, seed=5)
    loss = model.train(X, Y, steps=800, lr=1e-2)
    train_s = time.perf_counter() - t0
    comms = 8 << max(0, scale - 16)  # the held-out graph's planted communities grow with it
    g = K.build_graph(ctx, K.rmat_planted(scale, 16, comms, 100, 400, 0.5, seed=79))
    runs = {}
    for label, kw in (("zero", {}), ("warm", {"model": model}), ("waves", {"det_mode": K.SEQ_WAVES}),
                      ("shared", {"det_mode": K.SEQ_SHARED}),
                      ("warm_shared", {"model": model, "det_mode": K.SEQ_SHARED})):
        if label in labels:
            runs[label] = W.time_to_gap(g, k, gap, max_passes, trace=True, **kw)
    D = runs["zero"]["density"]
    out = {"graph": {"kind": f"rmat scale {scale}, edge factor 16, {comms} planted G(n_c, 0.5), n_c in [100, 400]",
                     "n": g.n, "m": g.m}, "k": k, "gap": gap,
           "train": {"graphs": len(train), "vertices": int(X.shape[0]), "loss": loss, "seconds": train_s},
           "warm_t0": W.DEFAULT_T0}
    for label, r in runs.items():
        to_d = W.passes_to_density(r["trace"], D * (1 - 1e-12))
        out[label] = {"passes": r["passes"], "seconds": r["seconds"], "reached": r["reached"],
                      "density": r["density"], "ub": r["ub"],
                      "passes_to_zero_density": to_d[0], "seconds_to_zero_density": to_d[1]}
    z = runs["zero"]["seconds"]
    fin = lambda x: x if math.isfinite(x) else None  # noqa: E731
    for lb in runs:
        out[lb]["seconds_to_zero_density"] = fin(out[lb]["seconds_to_zero_density"])
    others = [lb for lb in runs if lb != "zero"]
    out["speedup_certified"] = {lb: z / runs[lb]["seconds"] for lb in others}
    out["speedup_to_zero_density"] = {lb: (z / out[lb]["seconds_to_zero_density"]
                                           if out[lb]["seconds_to_zero_density"] else None)
                                      for lb in others}
    g.close()
    return out


def batch_workload(K, ctx, a) -> dict:
    """Many graphs of uneven size, k = 3..7, `batch_passes` Seq passes each, all
    in one persistent replay of a captured CUDA graph (kclpp_batch_run): the
    batched configuration with n log-uniform in [1e3, batch_nmax] (the
    configuration's 1e6 would need ~1.3e9 edges of host-side generation)."""
    rng = np.random.default_rng(a.seed)
    t0 = time.perf_counter()
    els = []
    for i in range(a.batch_graphs):
        n = int(np.exp(rng.uniform(np.log(1e3), np.log(a.batch_nmax))))
        d = float(rng.uniform(8, 64))
        els.append(K.erdos_renyi(n, d, seed=1000 + i) if i % 2 else K.chung_lu(n, d, 2.5, seed=1000 + i))
    gen_s = time.perf_counter() - t0
    print(f"batch: generated {len(els)} graphs in {gen_s:.1f} s", file=sys.stderr, flush=True)
    t0 = time.perf_counter()
    b = K.Batch(ctx, els)
    build_s = time.perf_counter() - t0
    print(f"batch: union of {b.n} vertices, {b.m} edges built in {build_s:.1f} s", file=sys.stderr, flush=True)
    ks = [3, 4, 5, 6, 7]
    T = a.batch_passes
    tuned = None
    if not a.no_autotune:
        # Untimed setup: the union's schedule tuned at the largest k, whose
        # passes take most of the replay (one schedule serves every k).
        t0 = time.perf_counter()
        res = K.autotune(b.union_graph(), max(ks), K.KERNEL_SEQ)
        tuned = {"k": max(ks), "schedule": res.best.as_dict(), "pass_ms": res.best_ms, "default_pass_ms": res.default_ms,
                 "seconds": round(time.perf_counter() - t0, 1)}
        print(f"batch: tuned at k = {max(ks)} in {tuned['seconds']} s", file=sys.stderr, flush=True)
    t0 = time.perf_counter()
    out = b.run(K.KERNEL_SEQ, ks, T)  # captures the CUDA graph
    first_s = time.perf_counter() - t0
    print(f"batch: first run (capture + replay) {first_s:.1f} s", file=sys.stderr, flush=True)
    # every pass gives each k-clique one unit: the r vectors sum to T x the count
    visits = int(sum(int(out[i].sum()) for i in range(len(ks))))
    times = []
    for _ in range(max(1, a.steps)):
        t0 = time.perf_counter()
        out2 = b.run(K.KERNEL_SEQ, ks, T)
        ctx.synchronize()
        times.append(time.perf_counter() - t0)
    same = bool(np.array_equal(out, out2))
    sec = statistics.median(times)
    return {"metric": METRIC, "value": visits / sec, "unit": UNIT, "n_gpus": 1, "steps": len(times),
            "ms_per_step": 1000 * sec, "higher_is_better": True, "dtype": "u64", "data": "synthetic",
            "config": {"workload": f"batch: {a.batch_graphs} graphs (Erdos-Renyi / Chung-Lu 2.5, n log-uniform in "
                                   f"[1e3, {a.batch_nmax:.0e}], average degree uniform in [8, 64]), k = 3..7, "
                                   f"{T} Seq passes each, one captured CUDA graph per run",
                       "graphs": a.batch_graphs, "total_n": b.n, "total_m": b.m, "k": ks, "passes": T},
            "clique_visits_per_step": visits, "first_run_s": first_s, "gen_s": gen_s, "build_s": build_s,
            "autotune": tuned,
            "replay_identical": same,
            "note": "one step = one kclpp_batch_run replay (all graphs x all k x all passes) plus the "
                    "download of the r vectors"}


def sampling_workload(K, ctx, a) -> dict:
    """Seq-Sampling++ (kCDensestSamplingKclistpp.c) on the RMAT graph of
    --scale (untrimmed, seeded), k = --k: the exact clique count, the sample
    of 10^7 cliques kept on the device, one "++" pass over the sample per
    step (8 waves), and one report (densest prefix, exact count of its
    subgraph, bound)."""
    t0 = time.perf_counter()
    el = K.rmat(a.scale, 16, seed=a.seed)
    g = K.build_graph(ctx, el)
    prep_s = time.perf_counter() - t0
    K.count_cliques(g, a.k)  # warm-up
    t0 = time.perf_counter()
    total, _ = K.count_cliques(g, a.k)
    count_s = time.perf_counter() - t0
    t0 = time.perf_counter()
    smp = K.Sampling(g, a.k, K.SAMPLE_TARGET, a.seed, 8)
    create_s = time.perf_counter() - t0
    info = smp.info()
    for _ in range(max(3, a.warmup)):
        smp.passes(1)
    times = []
    for _ in range(max(1, a.steps)):
        t0 = time.perf_counter()
        smp.passes(1)
        times.append(time.perf_counter() - t0)
    T = smp.info().passes
    t0 = time.perf_counter()
    rep, _ = smp.extract(T)
    extract_s = time.perf_counter() - t0
    sec = statistics.median(times)
    out = {"metric": "sampled k-cliques/s (Seq-Sampling++ pass)", "value": info.sampled / sec,
           "unit": "k-cliques/s", "n_gpus": 1, "steps": len(times), "warmup": max(3, a.warmup),
           "ms_per_step": 1000 * sec, "higher_is_better": True, "dtype": "u32", "data": "synthetic",
           "config": {"workload": f"sampling: rmat{a.scale}-ef16 (0.57,0.19,0.19,0.05), untrimmed, k={a.k}, "
                                  f"target {K.SAMPLE_TARGET} cliques, 8 waves", "n": g.n, "m": g.m,
                      "core": g.core, "k": a.k},
           "cliques_total": total, "sampled": info.sampled, "prob": info.prob, "count_ms": 1000 * count_s,
           "create_ms": 1000 * create_s, "extract_ms": 1000 * extract_s, "prep_s": prep_s,
           "report": {"T": rep.T, "sub_n": rep.sub_n, "sub_e": rep.sub_e, "sub_cliques": rep.sub_cliques,
                      "clique_density": rep.clique_density, "upper_bound": rep.upper_bound},
           "note": "one step = one kclpp_sampling_passes(1) call (8 waves, synchronised); create_ms is the "
                   "count plus the sampling pass"}
    smp.close()
    return out


def convergence_workload(K, ctx, a) -> dict:
    """The learned warm start's configuration towards its stated scale: the
    time-to-gap comparison of the default line on a held-out RMAT graph of
    --conv-scale with --conv-train training graphs (the configuration names
    RMAT scale 22 and 2,000 training runs)."""
    labels = tuple(x for x in a.conv_modes.split(",") if x)
    if "zero" not in labels:
        labels = ("zero",) + labels
    conv = convergence(ctx, scale=a.conv_scale, train_graphs=a.conv_train, labels=labels)
    z = conv["zero"]["seconds"]
    best = min((lb for lb in labels if lb != "zero"), key=lambda lb: conv[lb]["seconds"], default="zero")
    return {"metric": "time to a certified 1% density gap (k = 5)", "value": conv[best]["seconds"], "unit": "s",
            "n_gpus": 1, "higher_is_better": False, "dtype": "u64", "data": "synthetic",
            "config": {"workload": f"convergence: held-out RMAT scale {a.conv_scale} with planted communities, "
                                   f"{a.conv_train} training graphs, modes {','.join(labels)}"},
            "best": best, "zero_seconds": z, "convergence": conv}


def large_workload(K, ctx, a) -> dict:
    """The large configuration's shape -- Chung-Lu n = 4M, exponent 2.1,
    average degree 50, 50 planted G(n_c, 0.5) communities -- at k = --large-k
    (default 4) for --large-passes passes, the communities' sizes set by
    --large-nc.  The configuration's k = 6 is beyond a run here: the Chung-Lu
    background alone has degeneracy ~770, and its 6-clique count did not
    finish in 25 minutes on a GB300 even with communities of 100-250.  Times
    the core order, the count, T Seq and T Sim passes on the whole graph (on
    device buffers), the exact k-clique core trim, and on the trimmed core T
    Seq passes, the extraction and the certificate; checks the count, the
    trim's core against the oracle's count and one Seq and one Sim pass on
    the trimmed core against the oracle bit for bit."""
    import torch
    from oracle import oracle as O

    lo_c, hi_c = (int(x) for x in a.large_nc.split(","))
    k, T = a.large_k, a.large_passes
    out = {"metric": METRIC, "unit": UNIT, "n_gpus": 1, "higher_is_better": True, "dtype": "u64+f64",
           "data": "synthetic"}
    cfg = {"workload": f"large: Chung-Lu n = 4M, exponent 2.1, average degree 50, 50 planted G(n_c, 0.5) "
                       f"communities, n_c in [{lo_c}, {hi_c}], k = {k}, T = {T}",
           "k": k, "passes": T}
    t0 = time.perf_counter()
    el = K.planted(4_000_000, 50.0, 2.1, 50, lo_c, hi_c, 0.5, seed=a.seed)
    cfg["gen_s"] = round(time.perf_counter() - t0, 2)
    t0 = time.perf_counter()
    g = K.build_graph(ctx, el)
    cfg["build_s"] = round(time.perf_counter() - t0, 2)
    cfg.update(n=g.n, m=g.m, core=g.core)
    print(f"large: n {g.n} m {g.m} core {g.core}, generated in {cfg['gen_s']} s, ordered in {cfg['build_s']} s",
          file=sys.stderr, flush=True)
    K.count_cliques(g, k)  # warm-up
    t0 = time.perf_counter()
    total, per = K.count_cliques(g, k)
    count_s = time.perf_counter() - t0
    out["count"] = {"cliques": total, "seconds": round(count_s, 3), "k_cliques_per_s": total / count_s,
                    "per_vertex_sums_to_k_times_total": int(per.sum()) == k * total}
    print(f"large: {total} {k}-cliques in {count_s:.2f} s", file=sys.stderr, flush=True)
    stream = torch.cuda.current_stream()
    r = torch.zeros(g.n, dtype=torch.int64, device="cuda")
    rho = torch.zeros(g.n, dtype=torch.float64, device="cuda")
    K.seq_passes_dev(g, k, 1, r.data_ptr())  # warm-up (and the first pass's ties)
    K.sim_passes_dev(g, k, 1, 1, rho.data_ptr())
    ctx.synchronize()
    r.zero_()
    rho.zero_()
    torch.cuda.synchronize()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(3)]
    ev[0].record(stream)
    K.seq_passes_dev(g, k, T, r.data_ptr())
    ev[1].record(stream)
    K.sim_passes_dev(g, k, 1, T, rho.data_ptr())
    ev[2].record(stream)
    torch.cuda.synchronize()
    seq_ms = ev[0].elapsed_time(ev[1]) / T
    sim_ms = ev[1].elapsed_time(ev[2]) / T
    rh = r.cpu().numpy().view(np.uint64)
    info, _ = K.extract_densest_seq(g, k, T, rh.copy())
    out["value"] = 2 * total / ((seq_ms + sim_ms) / 1000.0)
    out["ms_per_step"] = seq_ms + sim_ms
    out["steps"] = T
    out["passes"] = {"seq_ms": seq_ms, "sim_ms": sim_ms, "seq_k_cliques_per_s": total / (seq_ms / 1000.0),
                     "sim_k_cliques_per_s": total / (sim_ms / 1000.0),
                     "seq_conserves": int(rh.sum()) == T * total,
                     "densest": {"n": info.n, "m": info.m, "cliques": info.cliques, "density": info.density,
                                 "ub": info.ub}}
    print(f"large: Seq {seq_ms:.1f} ms, Sim {sim_ms:.1f} ms per pass", file=sys.stderr, flush=True)
    g.close()
    t0 = time.perf_counter()
    tr = K.trim(ctx, el, k, K.TRIM_EXACT)
    trim_s = time.perf_counter() - t0
    ti = tr.info
    P = tr.edges.pairs()
    out["trim"] = {"seconds": round(trim_s, 2), "k_core_vertices": ti.n2, "cliques_in_k_core": ti.total,
                   "core_number": ti.ckcore, "density": ti.ckrho, "trimmed_vertices": ti.ntrim,
                   "trimmed_edges": ti.mtrim, "trimmed_cliques": ti.ncktrim, "peel": tr.peel.as_dict()}
    print(f"large: trim {trim_s:.1f} s -> {ti.ntrim} vertices, {ti.ncktrim} cliques", file=sys.stderr, flush=True)
    gt = K.build_graph(ctx, K.EdgeList.from_pairs(P))
    og = O.Graph(P)
    threads = os.cpu_count() or 1
    ct, _ = K.count_cliques(gt, k)
    rt = K.seq_passes(gt, k, T)
    infot, _ = K.extract_densest_seq(gt, k, T, rt)
    want = og.seq_pass(k, rt, O.SEQ_EDGE_STREAMS, threads)
    got = K.seq_passes(gt, k, 1, rt.copy())
    rho_t = K.sim_passes(gt, k, 1)
    want_sim = og.sim_pass(k, 1, np.zeros(gt.n), threads)
    t0 = time.perf_counter()
    cert, _ = K.certify_densest(gt, k, rt, 256)
    cert_s = time.perf_counter() - t0
    out["trimmed_core"] = {
        "cliques": ct, "count_matches_oracle": ct == og.count_cliques(k)[0] == ti.ncktrim,
        "seq_pass_matches_oracle": bool(np.array_equal(got, want)),
        "sim_pass_matches_oracle": bool(np.array_equal(rho_t.view(np.uint64), want_sim.view(np.uint64))),
        "densest": {"n": infot.n, "m": infot.m, "cliques": infot.cliques, "density": infot.density, "ub": infot.ub},
        "certificate": {"certified": bool(cert.certified), "inside": bool(cert.inside),
                        "inside_method": cert.inside_method, "outside": bool(cert.outside), "n": cert.n,
                        "cliques": cert.cliques, "density": cert.density, "seconds": round(cert_s, 2)}}
    gt.close()
    out["config"] = cfg
    out["note"] = ("value: (Seq + Sim) k-cliques per second over the whole graph, passes on device buffers; "
                   "one step = one Seq pass + one Sim pass")
    return out


def parity_check(K, ctx, a, g, pairs, r_start, rho_start, t_start, el_full=None) -> dict:
    """Outside the timed region, with the oracle as the checker: one Seq pass
    (per-root-edge streams) and one Sim pass on the bench graph from the state
    the timed passes started from, bit for bit, and the extraction of the Seq
    result; at k = 4 also k = 5 on the graph trimmed at 5, on two root shards
    of the library's partition (a whole k = 5 pass takes minutes on the host)."""
    from oracle import oracle as O

    threads = os.cpu_count() or 1
    t0 = time.time()
    og = O.Graph(pairs)
    out = {"k": [a.k]}
    r = K.seq_passes(g, a.k, 1, r_start.copy())
    want = og.seq_pass(a.k, r_start, O.SEQ_EDGE_STREAMS, threads)
    out["seq"] = bool(np.array_equal(r, want))
    info, re = K.extract_densest_seq(g, a.k, t_start, r)
    oinfo, ore = og.seq_find_densest(a.k, t_start, want, threads)
    out["extract"] = bool(np.array_equal(re, ore) and (info.n, info.m, info.cliques) == (oinfo.n, oinfo.m, oinfo.cliques)
                          and info.density == oinfo.density and info.ub == oinfo.ub)
    rho = K.sim_passes(g, a.k, 1, rho_start.copy(), t_first=t_start)
    want = og.sim_pass(a.k, t_start, rho_start, threads)
    out["sim"] = bool(np.array_equal(rho.view(np.uint64), want.view(np.uint64)))
    if a.k == 4 and el_full is not None:
        import torch

        k5 = K.trim(ctx, el_full, 5, K.TRIM_EXACT)
        gold5 = golden_trim(a.scale, 5, a.seed)
        if gold5 is not None:
            out["trim5_matches_reference"] = bool(
                k5.info.ncktrim == gold5["ncktrim"] and k5.info.ckcore == gold5["ckcore"]
                and np.array_equal(k5.edges.pairs(), induce_kept(el_full.pairs(), gold5["kept_in_label_order"])))
        P5 = k5.edges.pairs()
        g5 = K.build_graph(ctx, K.EdgeList.from_pairs(P5))
        og5 = O.Graph(P5)
        off5, _ = g5.csr()
        world = 48
        owner = K.shard_plan(off5, world)
        r0 = np.zeros(g5.n, np.uint64)
        rho0 = np.zeros(g5.n)
        r_d = torch.from_numpy(r0.view(np.int64).copy()).cuda()
        rho_d = torch.from_numpy(rho0.copy()).cuda()
        part = torch.empty(g5.n, dtype=torch.int64, device="cuda")
        ok_s = ok_o = True
        for rank in (0, 29):
            mask = (owner == rank).astype(np.uint8)
            torch.cuda.synchronize()
            K.graph_shard(g5, rank, world)
            K.seq_delta_dev(g5, 5, r_d.data_ptr(), part.data_ptr())
            ctx.synchronize()
            ok_s &= bool(np.array_equal(part.cpu().numpy().view(np.uint64), og5.seq_delta_masked(5, r0, mask, threads)))
            K.sim_counts_dev(g5, 5, rho_d.data_ptr(), part.data_ptr())
            ctx.synchronize()
            ok_o &= bool(np.array_equal(part.cpu().numpy().view(np.uint64), og5.sim_counts_masked(5, rho0, mask, threads)))
            K.graph_shard(g5, 0, 1)
        g5.close()
        out["k"] = [4, 5]
        out["k5"] = {"seq": ok_s, "sim": ok_o, "how": "2 of 48 root shards of the k = 5 trimmed core, from zero"}
        out["seq"] = out["seq"] and ok_s
        out["sim"] = out["sim"] and ok_o
    out["seconds"] = round(time.time() - t0, 1)
    return out


def reference_arm(a, modes: list[str], world: int) -> None:
    """`--impl reference`: the reference algorithm (the oracle, a C port of
    kCDensestNoAtom's and kCDensestCmpSync's passes with the reference's own
    p-thread schedule) on all host cores, each step a bounded sample of root
    edges of the same trimmed graph."""
    wl = reference_workload(a.scale, a.k, a.seed)
    if wl is None:
        print(json.dumps({"impl": "reference", "unavailable": f"no recorded reference trim for rmat{a.scale} seed "
                                                              f"{a.seed} k={a.k} (tests/golden/rmat20_trim.json)"}),
              flush=True)
        return
    pairs, meta = wl["pairs"], wl["meta"]
    config = workload_config(a, modes, meta, world)
    threads = os.cpu_count() or 1
    for _ in range(a.warmup):
        cpu_sample(pairs, a.k, modes, a.cpu_seconds / 4, threads)
    res = [cpu_sample(pairs, a.k, modes, a.cpu_seconds, threads) for _ in range(a.steps)]
    cl = sum(x["cliques"] for x in res)
    sec = sum(x["seconds"] for x in res)
    v = cl / sec
    samp = res[-1]
    line = {"impl": "reference", "metric": METRIC, "value": v, "unit": UNIT, "n_gpus": world, "steps": a.steps,
            "warmup": a.warmup, "ms_per_step": 1000 * sec / a.steps, "higher_is_better": True,
            "scaling": "strong", "vs_baseline": None, "dtype": "u64+f64", "data": "synthetic", "config": config,
            "cpu_baseline": {"value": v, "unit": UNIT, "cores": threads, "kind": "port",
                             "sample": f"every {samp['stride']}th root edge ({samp['edges']} of {samp['m']}) "
                                       f"per mode per step, {', '.join(modes)}; reference p-thread schedule"},
            "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def workload_config(a, modes: list[str], meta: dict, world: int) -> dict:
    return {"workload": f"rmat{a.scale}-ef16 (0.57,0.19,0.19,0.05) k-clique-core-trimmed, k={a.k}; "
                        f"one step = one {' + one '.join(m.capitalize() + '-kClist++ pass' for m in modes)}",
            "k": a.k, "graph": meta, "l2": "flushed before every timed step (256 MiB write)",
            "seq_order": "per-root-edge streams",
            "parallelism": f"roots split over {world} GPUs, per-pass all-reduce" if world > 1 else "1 GPU"}


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--k", type=int, default=4)
    ap.add_argument("--scale", type=int, default=20)
    ap.add_argument("--seed", type=int, default=1)
    ap.add_argument("--modes", default="seq,sim")
    ap.add_argument("--workload", default="rmat", choices=["rmat", "batch", "sampling", "large", "convergence"],
                    help="rmat: the default line (RMAT-20 trimmed core); batch: many uneven graphs x k = 3..7 "
                         "in one captured CUDA graph; sampling: Seq-Sampling++ on the untrimmed RMAT graph; "
                         "large: the large configuration's graph (Chung-Lu 4M, exponent 2.1, planted communities); "
                         "convergence: the time-to-gap comparison at --conv-scale")
    ap.add_argument("--conv-scale", type=int, default=18)
    ap.add_argument("--conv-train", type=int, default=128)
    ap.add_argument("--conv-modes", default="zero,warm,shared,warm_shared")
    ap.add_argument("--large-nc", default="200,2000", help="planted community sizes of --workload large")
    ap.add_argument("--large-k", type=int, default=4)
    ap.add_argument("--large-passes", type=int, default=10)
    ap.add_argument("--batch-graphs", type=int, default=512)
    ap.add_argument("--batch-nmax", type=float, default=1e5)
    ap.add_argument("--batch-passes", type=int, default=20)
    ap.add_argument("--cpu-seconds", type=float, default=12.0)
    ap.add_argument("--e2e-steps", type=int, default=-1,
                    help="steps of the host-buffer run (default: --steps, replaying the timed passes)")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-autotune", action="store_true")
    ap.add_argument("--no-parity", action="store_true",
                    help="skip the oracle check of one Seq and one Sim pass (k and, at k = 4, k = 5)")
    ap.add_argument("--no-convergence", action="store_true",
                    help="skip the time-to-1%%-gap comparison (learned warm start, waves, zero start)")
    ap.add_argument("--cache", default=os.path.join(tempfile.gettempdir(), "kclpp_bench_cache"))
    a = ap.parse_args()
    modes = [m for m in a.modes.split(",") if m]
    if a.impl == "reference" and a.workload != "rmat":
        if int(os.environ.get("RANK", "0")) == 0:
            print(json.dumps({"impl": "reference", "unavailable": f"the reference arm times the default workload "
                                                                  f"only, not --workload {a.workload}"}), flush=True)
        return

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))

    if a.impl == "reference":
        # The reference algorithm on the host cores: only the oracle's library
        # is loaded in this process (no torch, no kclistpp_gb300).  Under
        # torchrun, rank 0 alone runs it.
        if rank == 0:
            reference_arm(a, modes, world)
        return

    import torch

    dist = None
    if world > 1:
        import torch.distributed as dist

        dist.init_process_group("nccl")
    torch.cuda.set_device(local)
    import kclistpp_gb300 as K

    # A dedicated stream: the library launches on it and the timing events are
    # recorded on it (torch's default stream has the handle 0, which the
    # library would read as "make your own stream").
    stream = torch.cuda.Stream()
    torch.cuda.set_stream(stream)
    ctx = K.Context(local, stream=stream.cuda_stream)
    if a.workload in ("batch", "sampling", "large", "convergence"):
        if rank == 0:
            fn = {"batch": batch_workload, "sampling": sampling_workload, "large": large_workload,
                  "convergence": convergence_workload}[a.workload]
            print(json.dumps(fn(K, ctx, a)), flush=True)
        ctx.close()
        if dist:
            dist.destroy_process_group()
        return
    wl = prepare_workload(K, ctx, a.scale, a.k, a.seed, a.cache)
    pairs, meta = wl["pairs"], wl["meta"]
    config = workload_config(a, modes, meta, world)

    # ---- GB300 arm -----------------------------------------------------------------
    el = K.EdgeList.from_pairs(pairs)
    g = K.build_graph(ctx, el)
    off, cols = g.csr()
    tuned = {}
    if not a.no_autotune:
        # Untimed setup: pick the fastest schedule for each kernel of the step.
        for md, kern in (("seq", K.KERNEL_SEQ), ("sim", K.KERNEL_ORDER)):
            if md in modes:
                t = K.autotune(g, a.k, kern)
                tuned[md] = {"schedule": t.best.as_dict(), "pass_ms": t.best_ms, "default_pass_ms": t.default_ms,
                             "candidates": t.candidates}
    cliques_per_pass, _ = K.count_cliques(g, a.k)
    sp_c = K.Schedule(**tuned["sim"]["schedule"]) if "sim" in tuned else K.get_schedule(g)
    sp_s = K.Schedule(**tuned["seq"]["schedule"]) if "seq" in tuned else K.get_schedule(g)
    stats = dag_stats(off, cols, a.k, sp_c.tier_s_max, sp_c.m_split1, sp_c.m_split2)
    stats_seq = dag_stats(off, cols, a.k, sp_s.tier_s_max_seq, sp_s.seq_split1, sp_s.seq_split2)
    config["autotune"] = tuned
    config["dag"] = {"n": g.n, "m": g.m, "max_out_degree": g.core, "cliques_per_pass": int(cliques_per_pass),
                     "tiers": {f"{t}{d}": v for (t, d), v in stats["tiers"].items()},
                     "seq_tiers": {f"{t}{d}": v for (t, d), v in stats_seq["tiers"].items()}}
    n = g.n
    r_dev = torch.zeros(n, dtype=torch.int64, device="cuda")
    rho_dev = torch.zeros(n, dtype=torch.float64, device="cuda")
    flush = torch.empty(L2_FLUSH_BYTES, dtype=torch.uint8, device="cuda")
    t_sim = [1]

    if world > 1:
        # Split every pass over the ranks by root (the library's partition);
        # the ranks sum the per-pass n-vectors with an all-reduce.
        K.graph_shard(g, rank, world)
        part = torch.empty(n, dtype=torch.int64, device="cuda")

    def step(marks=None):
        for md in modes:
            if md == "seq":
                if world > 1:
                    K.seq_delta_dev(g, a.k, r_dev.data_ptr(), part.data_ptr())
                    dist.all_reduce(part)
                    r_dev.add_(part)
                else:
                    K.seq_passes_dev(g, a.k, 1, r_dev.data_ptr())
            else:
                if world > 1:
                    K.sim_counts_dev(g, a.k, rho_dev.data_ptr(), part.data_ptr())
                    dist.all_reduce(part)
                    K.sim_update_dev(ctx, n, t_sim[0], rho_dev.data_ptr(), part.data_ptr())
                else:
                    K.sim_passes_dev(g, a.k, t_sim[0], 1, rho_dev.data_ptr())
                t_sim[0] += 1
            if marks is not None:
                ev = torch.cuda.Event(enable_timing=True)
                ev.record(stream)
                marks.append((md, ev))

    for _ in range(max(3, a.warmup)):
        flush.fill_(1)
        step()
    ctx.synchronize()
    torch.cuda.synchronize()
    # the state the timed passes start from (the host-buffer run replays them)
    r_start = r_dev.cpu().numpy().view(np.uint64).copy()
    rho_start = rho_dev.cpu().numpy().copy()
    t_start = t_sim[0]
    if dist:
        dist.barrier()
    clocks = ClockSampler(local)
    clocks.start()
    time.sleep(0.3)
    ctx.profile(True)
    ctx.profile_read()
    launches0 = ctx.launches()
    evs = []
    torch.cuda.synchronize()
    if dist:
        dist.barrier()
    nvtx = getattr(torch.cuda, "nvtx", None)
    if nvtx is not None:
        nvtx.range_push("kclpp_timed")  # lets a profiler select the timed launches
    wall0 = time.perf_counter()
    for i in range(a.steps):
        flush.fill_(i & 0xFF)
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        marks = []
        step(marks)
        e1.record(stream)
        evs.append((e0, e1, marks))
    torch.cuda.synchronize()
    if nvtx is not None:
        nvtx.range_pop()
    if dist:
        dist.barrier()
    wall = time.perf_counter() - wall0
    launches = ctx.launches() - launches0
    prof = ctx.profile_read()
    ctx.profile(False)
    clk = clocks.stop()
    ctx.synchronize()
    step_ms = [x.elapsed_time(y) for x, y, _ in evs]
    ms = sum(step_ms) / len(step_ms)
    # per pass of each mode: from the previous mark (or the step's start) to its own
    pass_ms = {md: [] for md in modes}
    for e0, _, marks in evs:
        prev = e0
        for md, ev in marks:
            pass_ms[md].append(prev.elapsed_time(ev))
            prev = ev
    pass_ms = {md: sum(v) / len(v) for md, v in pass_ms.items()}
    if dist:
        t = torch.tensor([ms], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    per_step = cliques_per_pass * len(modes)
    value = per_step / (ms / 1000.0)

    # Roofline of the dominant kernel: one pass of the mode that takes the most
    # time (its root groups run as concurrent launches of one kernel, so the
    # pass, timed on the launching stream, is the unit).  The dense core is L2-
    # resident and every scheduler issues most cycles, so the roof is instruction
    # issue: SMs x 4 schedulers x one warp instruction per cycle at the sampled
    # SM clock; the instructions are the committed counters of this workload
    # (without them there is no fraction).  Beside it, as a measure of work and
    # not of traffic, the reference's per-root-edge gathers of MakeSubgraph.
    peak, peak_kind = measured_peaks()
    roofline = None
    if pass_ms and stats["ref_equiv_bytes_per_pass"]:
        md = max(pass_ms, key=pass_ms.get)
        st = stats_seq if md == "seq" else stats
        mhz = (clk or {}).get("sm_mhz") or 2070.0
        sms = torch.cuda.get_device_properties(local).multi_processor_count
        ipeak = sms * 4 * mhz * 1e6
        wi = profiled("warp_inst_per_pass", md, a)
        iach = wi / (pass_ms[md] / 1000.0) if wi else None
        bpp = stats["ref_equiv_bytes_per_pass"]
        achieved = bpp / (pass_ms[md] / 1000.0) / 1e9
        roofline = {"bound": "issue", "achieved": iach, "peak": ipeak, "unit": "warp inst/s",
                    "frac": iach / ipeak if wi else None, "warp_inst_per_pass": wi, "sm_mhz": mhz, "sms": sms,
                    "kernel": f"{'seq' if md == 'seq' else 'order'} pass "
                    f"(tier_m_kernel/tier_s_kernel, {len(st['tiers'])} concurrent root groups)",
                    "avg_launch_ms": pass_ms[md], "pass_ms": pass_ms,
                    "l2_bytes_per_pass": profiled("l2_bytes_per_pass", md, a),
                    "traffic": profiled("dram_bytes_per_pass", md, a),
                    "source": os.path.relpath(PASS_COUNTERS, ROOT) if wi else None,
                    "reference_bytes": {
                        "bytes_per_pass": bpp, "rate": achieved, "step_rate": bpp * len(modes) / (ms / 1000.0) / 1e9,
                        "unit": "GB/s", "hbm_gbs": peak, "hbm_source": f"{peak_kind} hbm_gbs",
                        "impl_bytes_per_pass": sum(v["impl_bytes"] for v in st["tiers"].values()),
                        "note": "the reference's per-root-edge gathers (MakeSubgraph, kCDensestNoAtom.c:86-113) "
                                "over every root edge, by the pass time: the rate of the work those bytes stand "
                                "for, above the HBM rate because they are not moved (one induction per root "
                                "vertex, the DAG in L2)"}}
    kernels = [{**p, "avg_ms": p["ms"] / max(1, p["launches"])} for p in prof]

    # ---- end to end through the C ABI with host buffers -------------------------------
    e2e = None
    e2e_steps = a.steps if a.e2e_steps < 0 else a.e2e_steps
    if e2e_steps > 0 and world == 1:
        off_h = torch.empty(len(off), dtype=torch.int64, pin_memory=True).numpy().view(np.uint64)
        off_h[:] = off
        cols_h = torch.empty(len(cols), dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
        cols_h[:] = cols
        r_h = torch.zeros(n, dtype=torch.int64, pin_memory=True).numpy().view(np.uint64)
        rho_h = torch.zeros(n, dtype=torch.float64, pin_memory=True).numpy()
        import ctypes as C

        sched = K.get_schedule(g)  # the tuned schedule of both kernels

        def e2e_step(tt):
            # The public host-buffer path: upload the DAG, choose the schedule,
            # run one pass of each kernel on host r / rho, download them.
            g2 = K.graph_from_csr(ctx, off_h, cols_h)
            K.set_schedule(g2, sched)
            for md in modes:
                if md == "seq":
                    K._check(K._lib.kclpp_seq_passes(ctx.handle, g2._h, a.k, 1, K.SEQ_EDGE_STREAMS,
                                                     r_h.ctypes.data_as(C.POINTER(C.c_uint64))))
                else:
                    K._check(K._lib.kclpp_sim_passes(ctx.handle, g2._h, a.k, tt, 1,
                                                     rho_h.ctypes.data_as(C.POINTER(C.c_double))))
            g2.close()

        r_h[:] = r_start
        rho_h[:] = rho_start
        e2e_step(t_start)  # warm
        # the same passes as the timed region: from the same r / rho and pass index
        r_h[:] = r_start
        rho_h[:] = rho_start
        e2e_t = []
        tt = t_start
        for _ in range(e2e_steps):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            e2e_step(tt)
            tt += 1
            e2e_t.append(time.perf_counter() - t0)
        roots = int(np.count_nonzero(np.diff(off)))
        # offsets, columns, edge sources, the root lists (counting, Seq and
        # wave schedules, u32 each, built at upload and again by
        # set_schedule), and r / rho
        graph_bytes = 8 * (n + 1) + 4 * g.m + 4 * g.m + 2 * 3 * 4 * roots
        h2d = graph_bytes + 8 * n * len(modes)
        d2h = (8 * n + 4) * len(modes)
        e2e = {"value": per_step / (sum(e2e_t) / len(e2e_t)), "unit": UNIT, "h2d_bytes_per_step": h2d,
               "d2h_bytes_per_step": d2h, "steps": e2e_steps,
               "api": "kclpp_graph_from_csr + kclpp_graph_set_schedule + kclpp_seq_passes / kclpp_sim_passes "
                      "(host CSR + host r / rho, pinned)"}

    cpu = None
    if rank == 0 and world == 1 and not a.no_cpu:
        threads = os.cpu_count() or 1
        s = cpu_sample(pairs, a.k, modes, a.cpu_seconds, threads)
        cpu = {"value": s["cliques"] / s["seconds"], "unit": UNIT, "cores": threads, "kind": "port",
               "sample": f"every {s['stride']}th root edge ({s['edges']} of {s['m']}) per mode, "
                         f"{', '.join(modes)}; {s['seconds']:.1f} s of CPU wall time"}

    parity = None
    if rank == 0 and world == 1 and not a.no_parity:
        el_full = K.rmat(a.scale, 16, 0.57, 0.19, 0.19, seed=a.seed) if a.k == 4 else None
        parity = parity_check(K, ctx, a, g, pairs, r_start, rho_start, t_start, el_full)
        parity["trim"] = meta.get("trim_matches_reference")

    cert = None
    if rank == 0 and world == 1 and not a.no_parity:
        # The exact certificate of the densest prefix (kCDensestMem.c:329-467,
        # restated with GPU passes), from the loads of 64 shared-load passes.
        t0 = time.time()
        _, r_c = K.seq_main(g, a.k, 64, K.SEQ_SHARED)
        ci, _ = K.certify_densest(g, a.k, r_c, 128)
        cert = {**ci.as_dict(), "seconds": round(time.time() - t0, 2),
                "note": "inside needs loads uniform on S to 1/(n j) or a max-flow on G[S] (at most 2e7 k-cliques)"}

    conv = None
    if rank == 0 and world == 1 and not a.no_convergence:
        conv = convergence(ctx)

    if rank == 0:
        line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": a.steps,
                "warmup": max(3, a.warmup), "ms_per_step": ms, "higher_is_better": True,
                "scaling": "strong",
                "vs_baseline": None, "dtype": "u64+f64", "data": "synthetic", "config": config,
                "roofline": roofline, "cpu_baseline": cpu, "e2e": e2e, "gpu_launches": launches,
                "clocks": clk, "kernels": kernels, "step_ms": step_ms, "wall_s": wall, "parity": parity,
                "certificate": cert, "convergence": conv}
        print(json.dumps(line), flush=True)
    g.close()
    ctx.close()
    if dist:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
