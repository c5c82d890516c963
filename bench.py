#!/usr/bin/env python3
"""Benchmark of the edgemap/vertexmap hot path on one B200 (or N replicas).

Workload (the large single-GPU configuration): R-MAT scale 24, edge factor 16
(2^28 generated edges, a,b,c,d = .57,.19,.19,.05, seed 1), symmetrised, self
loops and duplicate edges removed, uint32 vertex ids / uint64 offsets, built on
the device.  One step = one BFSLVLv run (BFS levels, sparse push / dense pull
switched by the m/20 threshold) from the next of 64 seeded non-isolated
roots.  The graph (2.3 GB) is far larger than the 126 MB L2, so no flush is
needed between steps.

Headline `value`: BFS GTEPS over the timed steps, Graph500 convention
(m_c/2 per run, m_c = directed edges incident to the reached vertices),
inputs resident in HBM.  The same JSON line also carries CC (CCv to
convergence) and PageRank (PRv, 20 iterations) throughput, the reduced
precision PageRank speed-ups, `e2e` (the public C-ABI call returning levels
to pinned host memory), the roofline of the dominant kernel, and the
reference CPU build timed on this host (`cpu_baseline`).

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference]

With --gpus N under torchrun every rank runs its own replica on its own
roots (no collective on the data path; "replicas only"); time is the max
over ranks.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "BFS/CC GTEPS, PR GEdges/s/iter @RMAT-24, %HBM peak; BF16/learned vs plain"
# Output checks that need the oracle / the reference build, queued by the
# measurement sections as (check(O, result_dict), result_dict) and run by the
# reference leg (the only part of the GPU arm that executes oracle/)
REF_CHECKS = []
SCALE, EDGE_FACTOR, GRAPH_SEED, ROOT_SEED, NROOTS = 24, 16, 1, 12345, 64
WORKLOAD = ("BFSLVLv levels from 64 seeded non-isolated roots, R-MAT scale 24 edge factor 16 "
            "(a,b,c=.57,.19,.19, seed 1), symmetrised, deduplicated, no self-loops")


# ---------------------------------------------------------------------------
# helpers
# ---------------------------------------------------------------------------
def peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(p) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


class ClockSampler:
    """SM clocks and clock-event (throttle) reasons sampled during the timed
    region: NVML polled every 5 ms from a thread (read-only queries), or
    nvidia-smi at 200 ms when NVML is unavailable."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
    REASONS = {"hw_slowdown": 0x8, "sw_thermal_slowdown": 0x20, "hw_thermal_slowdown": 0x40,
               "sw_power_cap": 0x4}

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.rows = []
        self.proc = None
        self.thread = None
        self.nvml = None
        self.stop_flag = threading.Event()
        try:
            import pynvml
            import torch
            pynvml.nvmlInit()
            p = torch.cuda.get_device_properties(gpu_index)
            bus = f"{p.pci_domain_id:08x}:{p.pci_bus_id:02x}:{p.pci_device_id:02x}.0"
            try:
                self.handle = pynvml.nvmlDeviceGetHandleByPciBusId(bus.encode())
            except Exception:
                self.handle = pynvml.nvmlDeviceGetHandleByIndex(gpu_index)
            self.max_mhz = float(pynvml.nvmlDeviceGetMaxClockInfo(self.handle, pynvml.NVML_CLOCK_SM))
            self.nvml = pynvml
        except Exception:
            self.nvml = None

    def _poll(self):
        nv = self.nvml
        while not self.stop_flag.is_set():
            try:
                sm = nv.nvmlDeviceGetClockInfo(self.handle, nv.NVML_CLOCK_SM)
                rs = nv.nvmlDeviceGetCurrentClocksEventReasons(self.handle)
                self.rows.append((float(sm), int(rs)))
            except Exception:
                pass
            self.stop_flag.wait(0.005)

    def start(self):
        if self.nvml is not None:
            self.thread = threading.Thread(target=self._poll, daemon=True)
            self.thread.start()
            return
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.proc = None
            return
        self.thread = threading.Thread(target=self._read, daemon=True)
        self.thread.start()

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append([x.strip() for x in line.split(",")])

    def stop(self):
        self.stop_flag.set()
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
        if self.thread is not None:
            self.thread.join(timeout=5)
        sm, mx, reasons = [], None, set()
        if self.nvml is not None:
            mx = self.max_mhz
            for clk, rs in self.rows:
                sm.append(clk)
                for nm, bit in self.REASONS.items():
                    if rs & bit:
                        reasons.add(nm)
            src = "nvml 5 ms"
        else:
            names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
            for r in self.rows:
                try:
                    sm.append(float(r[1]))
                    mx = float(r[2])
                except (ValueError, IndexError):
                    continue
                for i, nm in enumerate(names):
                    if len(r) > 5 + i and r[5 + i].lower() == "active":
                        reasons.add(nm)
            src = "nvidia-smi 200 ms"
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": mx,
                "reasons": sorted(reasons), "samples": len(sm), "source": src}


def dist_setup(args, backend: str = "nccl"):
    """One process per GPU (torchrun's RANK / LOCAL_RANK / WORLD_SIZE); the
    replicas share nothing on the data path, the process group only carries
    the barrier and the max / sum of the timing scalars."""
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if ws > 1:
        import datetime
        import torch
        import torch.distributed as dist
        if backend == "nccl":
            torch.cuda.set_device(local)
            dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600),
                                    device_id=torch.device("cuda", local))
        else:
            dist.init_process_group(backend, timeout=datetime.timedelta(seconds=60))
    return ws, rank, local


def barrier(ws):
    if ws > 1:
        import torch.distributed as dist
        dist.barrier()


def _reduce(x: float, ws: int, op: str) -> float:
    if ws == 1:
        return x
    import torch
    import torch.distributed as dist
    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([x], dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX if op == "max" else dist.ReduceOp.SUM)
    return float(t.item())


def max_over_ranks(x: float, ws: int) -> float:
    return _reduce(x, ws, "max")


def sum_over_ranks(x: float, ws: int) -> float:
    return _reduce(x, ws, "sum")


def replica_roots(roots, ws: int, rank: int, count: int):
    """Rank `rank`'s sequence of `count` roots: the 64 roots dealt round-robin
    over the ranks (step k of rank r takes root (k * ws + r) mod 64)."""
    return [int(roots[(k * ws + rank) % len(roots)]) for k in range(count)]


def pick_roots(deg: np.ndarray) -> np.ndarray:
    nz = np.flatnonzero(deg)
    rng = np.random.default_rng(ROOT_SEED)
    return rng.choice(nz, size=NROOTS, replace=False).astype(np.uint32)


# DRAM bytes (read + write) of one resident BFS (k_bfs_run) from ncu captures
# at R-MAT scale 23 (two roots, 734 and 374 MB), their mean scaled by the
# vertex count to scale 24
K_BFS_TRAFFIC_PER_RUN = 1.108e9
# DRAM bytes of one 128-seed PPR iteration (k_ppr_wide) at R-MAT 22
# (m = 128,311,324) from ncu: 8.58 GB read, 1.20 GB written
PPR_DRAM_BYTES_PER_ITER = 9.78e9


def bfs_bytes(n: int, st, it: int) -> float:
    """Algorithmic bytes of BFS iteration `it` (per-unit figures: 8-byte
    offsets, 4-byte ids and levels).  Sparse push: 4F + 16F + 4E + 4E + 4N.
    Dense pull: 8(n+1) + 4n + 4S + 4N + 2n/8."""
    from graptor_b200 import gg
    F, E, S = st.nactv[it], st.nacte[it], st.scanned[it]
    N = st.nactv[it + 1] if it + 1 < st.iterations else 0
    if st.variant[it] == gg.VAR_PULL_DENSE:
        return 8.0 * (n + 1) + 4.0 * n + 4.0 * S + 4.0 * N + 2.0 * n / 8
    return 20.0 * F + 8.0 * E + 4.0 * N


def cc_bytes(n: int, m: int, st, it: int) -> float:
    """Algorithmic bytes of CC iteration `it`: a dense pull reads offsets,
    labels, the scanned in-edges and their sources' labels (8(n+1) + 4n + 8S
    + 4N + 2n/8); a sparse push 4F + 16F + 4E + 4E + 4N; the hooking step
    (road-like graphs) offsets, labels and the scanned edges' ids (8(n+1) + 4S + 8n).
    The default run's two records, the search and the hooks, count as pulls."""
    from graptor_b200 import gg
    F, E, S = st.nactv[it], st.nacte[it], st.scanned[it]
    N = st.nactv[it + 1] if it + 1 < st.iterations else 0
    v = st.variant[it]
    if v == gg.VAR_PULL_DENSE:
        return 8.0 * (n + 1) + 4.0 * n + 8.0 * S + 4.0 * N + 2.0 * n / 8
    if v == gg.VAR_HOOK:
        return 8.0 * (n + 1) + 4.0 * S + 8.0 * n
    return 20.0 * F + 8.0 * E + 4.0 * N


# ---------------------------------------------------------------------------
# reference CPU arm / baseline
# ---------------------------------------------------------------------------
def reference_bfs(bin_path: str, roots, threads: int):
    from oracle import oracle as O
    return O.ref_bfs(bin_path, [int(r) for r in roots], threads=threads)


def cpu_info():
    cores = os.cpu_count() or 1
    model = ""
    try:
        with open("/proc/cpuinfo") as f:
            for line in f:
                if line.startswith("model name"):
                    model = line.split(":", 1)[1].strip()
                    break
    except OSError:
        pass
    return cores, model


def run_reference_arm(args, ws, rank):
    """The reference's own BFSLVLv (compiled from its sources, OpenMP backend)
    on this host's cores, same graph, roots, metric and unit."""
    if rank != 0:
        return 0
    from oracle import oracle as O
    if not O.ref_available("ref_bfslvl"):
        print(json.dumps({"impl": "reference", "unavailable":
                          "reference build oracle/_ref missing (needs the reference sources to compile)"}))
        return 0
    cores, model = cpu_info()
    t0 = time.time()
    g = O.rmat(args.scale, EDGE_FACTOR << args.scale, GRAPH_SEED)
    roots = pick_roots(g.outdeg())
    with tempfile.TemporaryDirectory() as tmp:
        path = os.path.join(tmp, "rmat.bin")
        O.write_bin(g, path)
        prep = time.time() - t0
        seq = [roots[i % NROOTS] for i in range(args.warmup + args.steps)]
        res = reference_bfs(path, seq, cores)
    res = res[args.warmup:]
    tot_t, tot_e = 0.0, 0.0
    gteps = []
    for r, t, _, _ in res:
        lv = O.bfs_level(g, int(r))
        mc = O.reached_edges(g, lv)
        tot_t += t
        tot_e += mc / 2
        gteps.append(mc / 2 / t / 1e9)
    val = tot_e / tot_t / 1e9
    line = {
        "impl": "reference", "metric": METRIC, "value": round(val, 4), "unit": "GTEPS",
        "n_gpus": ws, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": round(tot_t / len(res) * 1e3, 3), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "int32", "data": "synthetic",
        "config": {"workload": WORKLOAD, "scale": args.scale, "edge_factor": EDGE_FACTOR,
                   "n": g.n, "m": g.m, "roots": NROOTS},
        "cpu_baseline": {"value": round(val, 4), "unit": "GTEPS", "cores": cores, "kind": "reference",
                         "sample": f"{len(res)} BFSLVLv runs, reference build (OpenMP, {model})"},
        "e2e": {"value": round(val, 4), "unit": "GTEPS", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "bfs": {"gteps_mean": round(float(np.mean(gteps)), 4),
                "gteps_hmean": round(float(len(gteps) / np.sum(1.0 / np.array(gteps))), 4)},
        "input_prep_s": round(prep, 1),
    }
    print(json.dumps(line))
    return 0


def reference_leg(g, roots, args, lvl):
    """The reference build (oracle/_ref, compiled from the reference sources)
    on this host's cores, on the benchmarked graph written out as a Graptor
    .bin file: its BFSLVLv from the bench's roots is the CPU baseline (one
    process, one graph load, each run timed like the reference driver's
    "Running" bracket), and its outputs check the GPU's at this size -- BFS
    levels by a pair of 64-bit checksums per root (bit-exact or not), CCv
    labels in full (-cc:outfile), PRv ranks after 20 iterations in full
    (-pr:outfile, L1)."""
    from graptor_b200 import gg
    from oracle import oracle as O
    for check, res in REF_CHECKS:
        try:
            check(O, res)
        except Exception as e:  # recorded, never fatal
            res["check_failed"] = f"{e}"[:300]
    REF_CHECKS.clear()
    if not O.ref_available("ref_bfslvl"):
        return None, None
    cores, model = cpu_info()
    sample_roots = [int(r) for r in roots[: args.cpu_roots]]
    par = {"graph": f"rmat{args.scale} ef{EDGE_FACTOR}", "reference": "oracle/_ref build of the reference sources"}
    with tempfile.TemporaryDirectory() as tmp:
        path = os.path.join(tmp, "rmat.bin")
        g.write_bin(path)
        tc = time.time()
        res = O.ref_bfs(path, sample_roots, threads=cores, checksums=True)
        wall = time.time() - tc
        tt, ee, exact = 0.0, 0.0, 0
        for r, t, _, h in res:
            st = gg.RunStats()
            lv = g.bfs_level(int(r), level=lvl, stats=st)
            tt += t
            ee += st.edges_reached / 2.0
            exact += int(O.level_checksums(lv) == h)
        cpu = {"value": round(ee / tt / 1e9, 4), "unit": "GTEPS", "cores": cores, "kind": "reference",
               "sample": f"{len(res)} BFSLVLv runs (the first {len(res)} of the 64 roots) of the reference "
                         f"build, OpenMP, {model}; load+VEBO+runs wall {wall:.0f} s"}
        par["bfs_roots_checked"] = len(res)
        par["bfs_roots_bitexact"] = exact
        if not args.no_parity_cc_pr:
            tc = time.time()
            lab_ref, cc_t = O.ref_cc(path, os.path.join(tmp, "cc.txt"), threads=cores)
            lab = g.cc()
            par["cc_bitexact"] = bool(np.array_equal(lab, lab_ref))
            par["cc_reference_ms"] = round(min(cc_t) * 1e3, 2) if cc_t else None
            x_ref, pr_t = O.ref_pr(path, os.path.join(tmp, "pr.txt"), maxiter=20, threads=cores)
            x = g.pagerank(maxiter=20, tol=1e-7, contrib=gg.F32, accum_f64=True, renorm_f32=True)
            par["pr_iters"] = 20
            par["pr_l1_vs_ref"] = float(np.abs(x.astype(np.float64) - x_ref).sum())
            par["pr_max_rel_vs_ref"] = float((np.abs(x.astype(np.float64) - x_ref) /
                                              np.maximum(x_ref, 1e-30)).max())
            par["pr_reference_ms_per_iter"] = round(min(pr_t) * 1e3 / 20, 2) if pr_t else None
            par["cc_pr_wall_s"] = round(time.time() - tc, 1)
            if O.ref_available("KC_bucket"):
                tc = time.time()
                try:
                    core_ref, kc_t = O.ref_kc(path, os.path.join(tmp, "kc.txt"), threads=cores)
                    core, largest = g.kcore()
                    par["kc_bitexact"] = bool(np.array_equal(core, core_ref))
                    par["kc_largest"] = largest
                    par["kc_reference_ms"] = round(kc_t * 1e3, 2) if kc_t else None
                except Exception as e:  # recorded, never fatal
                    par["kc_check_failed"] = f"{e}"[:300]
                par["kc_wall_s"] = round(time.time() - tc, 1)
    return cpu, par


# ---------------------------------------------------------------------------
# learned selector evaluation (held-out graphs)
# ---------------------------------------------------------------------------
def deviation_oracle(g, analytic, root, thr_variant, t_thr, max_iters=64):
    """Oracle-best time of one run from forced timings on the threshold run's
    own state (gg_selector_collect: the run follows the threshold except at
    one iteration, which takes each of the four variants in turn).  BFS: every
    variant leaves the same next frontier, so the per-iteration gains over the
    threshold's own choice add up, oracle = T_thr - sum_i (t_i(thr) - min_v
    t_i(v)); CC: a step's choice changes what follows, so the best single
    deviation counts, oracle = T_thr - max_i (rest_i(thr) - min_v rest_i(v)).
    Returns (oracle ms, iterations covered) or (None, 0) for runs longer than
    max_iters iterations."""
    from graptor_b200 import gg
    T = len(thr_variant)
    if T > max_iters:
        return None, 0
    if gg.VAR_HOOK in thr_variant:
        # a CC run that finished by hooking: the forced runs could only
        # deviate before the hook, and each would then propagate labels to
        # convergence (minutes on the 2896^2 grid) without a sample to show
        return t_thr, 0
    X, Y = gg.selector_collect(g, 0 if analytic == "bfs" else 1, root, max_samples=max_iters, cap=max_iters)
    gains = []
    for x, y in zip(X, Y):
        it = int(round(2.0 ** (8.0 * float(x[3])) - 1.0))  # the iteration feature, log2(1 + it) / 8
        # (an iteration the threshold run took as CC's hooking step has no
        # traversal variant to deviate from)
        if it >= T or not np.all(np.isfinite(y)) or not 0 <= thr_variant[it] < len(y):
            continue
        t = 2.0 ** y.astype(np.float64) / 1e3  # ms
        gains.append(max(0.0, t[thr_variant[it]] - t.min()))
    if not gains:
        return t_thr, 0
    g_all = sum(gains) if analytic == "bfs" else max(gains)
    return t_thr - g_all, len(gains)


def selector_eval(ctx, graphs):
    """Device-driven BFS / CC with the density threshold, the learned selector
    and each fixed variant, medians of three runs; oracle-best from forced
    one-iteration deviations of the threshold run (deviation_oracle)."""
    from graptor_b200 import gg
    from graptor_b200.selector_train import load_selector
    sel = load_selector(ctx)
    old = {k: gg.tuning_get(k) for k in ("persistent", "resident")}
    gg.tuning_set("persistent", 7)
    gg.tuning_set("resident", 0)  # (the resident CC makes no choice: not for one policy only)
    out = {"weights": "graptor_b200/data/selector.npz" if sel else None,
           "oracle": "per root, the smaller of: the threshold run with one iteration forced to each variant "
                     "in turn on the same state (BFS sums the per-iteration gains, CC takes the best single "
                     "deviation), and every measured policy's time"}
    try:
        for name, g, roots in graphs:
            if sel:
                gg.attach_selector(g, sel)
            res = {}
            for analytic in ("bfs", "cc"):
                def run(opts, r):
                    st = gg.RunStats()
                    if analytic == "bfs":
                        g.bfs_level(r, host=False, opts=opts, stats=st)
                    else:
                        g.cc(host=False, opts=opts, stats=st)
                    return st
                rs = roots if analytic == "bfs" else [0]
                thr_opts = gg.default_opts(gg.THRESH_DEFAULT if analytic == "bfs" else gg.THRESH_FRAC,
                                           0 if analytic == "bfs" else 5)
                modes = {"threshold": thr_opts}
                if sel:
                    modes["learned"] = gg.default_opts(gg.THRESH_LEARNED)
                for v, vn in gg.VARIANT_NAMES.items():
                    modes["fixed_" + vn] = gg.default_opts(variant=v)
                tot = {k: 0.0 for k in modes}
                oracle, covered, dev_total = 0.0, 0, 0.0
                for r in rs:
                    per = {}
                    for k, o in modes.items():
                        run(o, r)  # warm
                        per[k] = float(np.median([run(o, r).total_ms for _ in range(3)]))
                        tot[k] += per[k]
                    rec = run(gg.default_opts(gg.THRESH_DEFAULT if analytic == "bfs" else gg.THRESH_FRAC,
                                              0 if analytic == "bfs" else 5, collect=True), r)
                    thr_var = [rec.variant[i] for i in range(min(rec.iterations, gg.MAX_ITERS))]
                    o_ms, cov = deviation_oracle(g, analytic, r, thr_var, per["threshold"])
                    if o_ms is None or oracle is None:
                        oracle = None
                    else:
                        # the oracle-best is a lower bound on every policy measured
                        # on this root: no measured run beats it by construction
                        # (the deviation estimate alone can miss gains that
                        # combine across iterations)
                        dev_total += o_ms
                        oracle += min(o_ms, min(per.values()))
                        covered += cov
                best_fixed = min(v for k, v in tot.items() if k.startswith("fixed_"))
                d = {k: round(v / len(rs), 4) for k, v in tot.items()}
                d["oracle_best_ms"] = round(oracle / len(rs), 4) if oracle is not None else None
                d["deviation_estimate_ms"] = round(dev_total / len(rs), 4) if oracle is not None else None
                d["oracle_iterations_covered"] = covered
                d["best_fixed_ms"] = round(best_fixed / len(rs), 4)
                if sel:
                    d["learned_vs_threshold"] = round(tot["threshold"] / tot["learned"], 3)
                    if oracle is not None:
                        d["learned_over_oracle"] = round(tot["learned"] / oracle, 3)
                if oracle is not None:
                    d["threshold_over_oracle"] = round(tot["threshold"] / oracle, 3)
                res[analytic] = d
            out[name] = res
            if sel:
                gg.attach_selector(g, None)
    finally:
        for k, v in old.items():
            gg.tuning_set(k, v)
    # the default BFS driver (one resident launch per run): the network picks
    # between its push and pull
    if sel:
        for name, g, roots in graphs:
            gg.attach_selector(g, sel)
            tot = {}
            for mode, opts in (("threshold", gg.default_opts(gg.THRESH_DEFAULT, collect=True)),
                               ("learned", gg.default_opts(gg.THRESH_LEARNED, collect=True))):
                t = 0.0
                for r in roots:
                    g.bfs_level(r, host=False, opts=opts)
                    st = gg.RunStats()
                    g.bfs_level(r, host=False, opts=opts, stats=st)
                    t += st.total_ms
                tot[mode] = t / len(roots)
            out[name]["bfs_default_driver"] = {k: round(v, 4) for k, v in tot.items()}
            out[name]["bfs_default_driver"]["learned_vs_threshold"] = round(tot["threshold"] / tot["learned"], 3)
            gg.attach_selector(g, None)
    return out


# ---------------------------------------------------------------------------
# PageRank precision (R-MAT 25 ef16; directed ER 2^25 avg degree 32, 1% sinks)
# ---------------------------------------------------------------------------
def reference_f64_check(O, path, x64, tmpd, res):
    """PR_vary VARIANT 11 of the reference build (FP64 ranks, contributions
    and sums, to the 1e-7 residual) on the graph file `path` against the
    FP64 variant's ranks x64: L1, max relative difference, iterations."""
    import shutil
    try:
        if not O.ref_available("PR_vary_11"):
            res["reference"] = "unavailable (reference build missing)"
            return
        cores, _ = cpu_info()
        t0 = time.time()
        xr, ts, its = O.ref_pr(path, os.path.join(tmpd, "x.txt"), maxiter=100, threads=cores,
                               prog_name="PR_vary_11", iterations=True)
        d = np.abs(x64 - xr)
        res.update({"l1_vs_reference_f64": float(d.sum()),
                    "max_rel_vs_reference_f64": float((d / np.maximum(xr, 1e-300)).max()),
                    "reference_iterations": its, "reference_wall_s": round(time.time() - t0, 1),
                    "reference_ms_per_iter": round(min(ts) * 1e3 / max(its or 1, 1), 1) if ts else None})
    finally:
        shutil.rmtree(tmpd, ignore_errors=True)


def precision_eval(ctx, hbm_peak, with_ref=True):
    """Each storage format run until the L1 residual <= 1e-7 or 100 iterations,
    timed per iteration, its ranks compared with the FP64 variant's (double
    ranks, sums and contributions; checked against the CPU FP64 oracle by the
    parity tests)."""
    from graptor_b200 import gg
    out = {}
    fmts = [("f32", gg.F32, True), ("bf16", gg.BF16, False), ("f16", gg.F16, False),
            ("fp8e4m3", gg.FP8E4M3, False), ("cfp_6_10", gg.CFP_6_10, False),
            ("bf16_sr_avg50", gg.BF16, False)]
    # BF16 with stochastic rounding of the contributions and the mean of the
    # last 50 of the 100 iterations' ranks
    extra = {"bf16_sr_avg50": dict(stochastic=True, average_last=50)}
    for name, make in (("rmat25", lambda: ctx.rmat(25, 16 << 25, GRAPH_SEED)),
                       ("er25_directed_1pct_sinks",
                        lambda: ctx.er(1 << 25, 32.0, GRAPH_SEED, dangling_bp=100, symmetric=False))):
        g = make()
        n, m = g.n, g.m
        x64 = g.pagerank(maxiter=100, tol=1e-7, contrib=gg.F64)
        st = gg.RunStats()
        g.pagerank(maxiter=100, tol=1e-7, contrib=gg.F64, host=False, stats=st)
        res = {"n": n, "m": m, "f64": {"iterations": st.iterations,
                                       "ms_per_iter": round(st.total_ms / max(st.iterations, 1), 4)}}
        # the reference's own FP64 run (PR_vary VARIANT 11) checks the FP64
        # variant on the symmetric graph (the reference build computes a
        # different iteration on directed graphs, so ER is not compared)
        if with_ref and name == "rmat25":
            tmpd = tempfile.mkdtemp(prefix="gg_pr25_")
            path = os.path.join(tmpd, "g.bin")
            g.write_bin(path)
            REF_CHECKS.append((lambda O, r, path=path, x64=x64, tmpd=tmpd: reference_f64_check(O, path, x64, tmpd, r),
                               res["f64"]))
        for fname, fmt, acc64 in fmts:
            kw = extra.get(fname, {})
            x = g.pagerank(maxiter=100, tol=1e-7, contrib=fmt, accum_f64=acc64, renorm_f32=(fname == "f32"), **kw)
            ts, its = [], 0
            for _ in range(2):
                st = gg.RunStats()
                g.pagerank(maxiter=100, tol=1e-7, contrib=fmt, accum_f64=acc64, renorm_f32=(fname == "f32"),
                           host=False, stats=st, **kw)
                ts.append(st.total_ms / max(st.iterations, 1))
                its = st.iterations
            err = np.abs(x.astype(np.float64) - x64)
            nz = x64 > 0
            res[fname] = {"iterations": its, "ms_per_iter": round(float(np.median(ts)), 4),
                          "l1_vs_f64": float(err.sum()),
                          "max_rel_vs_f64": float((err[nz] / x64[nz]).max())}
        base = res["f32"]["ms_per_iter"]
        for fname, _, _ in fmts:
            res[fname]["speedup_vs_f32_per_iter"] = round(base / res[fname]["ms_per_iter"], 3)
        # the BF16 target: >= 1.7x the FP32 path per iteration at <= 1e-4 L1 against FP64
        for fname in ("bf16", "bf16_sr_avg50"):
            r = res[fname]
            r["target_1.7x_at_1e-4"] = {"speed_met": r["speedup_vs_f32_per_iter"] >= 1.7,
                                         "l1_met": r["l1_vs_f64"] <= 1e-4}
        # staged precision (the switch taken on the device): time to the 1e-7 residual
        t_f32 = res["f32"]["ms_per_iter"] * res["f32"]["iterations"]
        for sname, stages in (("staged_f16_f32", [(gg.F16, False, 1e-3), (gg.F32, True, 0.0)]),
                              ("staged_bf16_f32", [(gg.BF16, False, 1e-3), (gg.F32, True, 0.0)]),
                              ("pr_vary_4620", [(gg.CFP_6_10, False, 1e-3), (gg.F32, True, 0.0)])):
            x = g.pagerank(maxiter=100, tol=1e-7, renorm_f32=False, stages=stages)
            ts = []
            for _ in range(2):
                st = gg.RunStats()
                g.pagerank(maxiter=100, tol=1e-7, renorm_f32=False, stages=stages, host=False, stats=st)
                ts.append(st.total_ms)
            err = np.abs(x.astype(np.float64) - x64)
            nz = x64 > 0
            res[sname] = {"iterations": st.iterations, "total_ms": round(float(np.median(ts)), 3),
                          "speedup_vs_f32_to_1e-7": round(t_f32 / float(np.median(ts)), 3),
                          "l1_vs_f64": float(err.sum()), "max_rel_vs_f64": float((err[nz] / x64[nz]).max())}
        res["f32"]["total_ms"] = round(t_f32, 3)
        out[name] = res
        g.close()
    return out


# ---------------------------------------------------------------------------
# batched traversals
# ---------------------------------------------------------------------------
def small_graph_batch(ctx, count, seed=2000):
    """`count` graphs, vertex counts log-uniform in [2^10, 2^18]: R-MAT with
    edge factor 8-32 (vertex count rounded to a power of two) and 2-D grids
    with 4-neighbour edges, alternating."""
    rng = np.random.default_rng(seed)
    parts = []
    for i in range(count):
        lg = rng.uniform(10, 18)
        if i % 2 == 0:
            scale = int(round(lg))
            parts.append(ctx.rmat(scale, int(rng.integers(8, 33)) << scale, seed + i))
        else:
            side = int(2 ** (lg / 2))
            parts.append(ctx.grid(side, max(1, int(2 ** lg) // side), seed + i))
    return parts


def batch_eval(ctx, g, roots, hbm_peak, n_small):
    """(a) 64-root multi-source BFS and 128-seed PPR on R-MAT 22 ef 16;
    (b) BFS from vertex 0 and CC of `n_small` small graphs as one union."""
    from graptor_b200 import gg
    out = {}
    n, m = g.n, g.m
    r64 = [int(r) for r in roots[:64]]
    gg.msbfs(g, r64, host=False)
    ms = []
    edges = 0
    for _ in range(3):
        st = gg.RunStats()
        gg.msbfs(g, r64, host=False, stats=st)
        ms.append(st.total_ms)
        edges = st.edges_reached
    t = float(np.median(ms))
    seq = 0.0
    for r in r64:
        st = gg.RunStats()
        g.bfs_level(r, host=False, stats=st)
        seq += st.total_ms
    out["msbfs64"] = {"ms": round(t, 3), "gteps": round(edges / 2.0 / (t / 1e3) / 1e9, 2),
                      "sequential_64_bfs_ms": round(seq, 3), "speedup_vs_sequential": round(seq / t, 2)}
    seeds = [int(r) for r in roots[:64]] + [int(r) for r in roots[:64][::-1]]
    seeds = seeds[:128]
    gg.ppr(g, seeds, iters=2, host=False)
    ms = []
    for _ in range(3):
        st = gg.RunStats()
        gg.ppr(g, seeds, alpha=0.15, iters=20, host=False, stats=st)
        ms.append(st.total_ms / 20)
    t = float(np.median(ms))
    # per iteration: ids + one 256-byte bf16 row per edge, offsets, the new
    # contribution rows (the ranks are written by the last iteration only).
    # Most of those row reads hit L2 (R-MAT hubs' rows are read again and
    # again), so this is a work figure, not DRAM traffic; the DRAM fraction
    # uses the bytes ncu counted for one iteration's launch at this size
    ppr_bytes = m * (256.0 + 4.0) + 8.0 * (n + 1) + n * 256.0
    ppr_dram = PPR_DRAM_BYTES_PER_ITER * m / 128311324.0
    out["ppr128"] = {"ms_per_iter": round(t, 3), "gedges_per_s_per_iter": round(m / (t / 1e3) / 1e9, 3),
                     "seed_edges_per_s": round(128 * m / (t / 1e3) / 1e9, 1),
                     "dram_frac_of_hbm": round(ppr_dram / (t / 1e3) / 1e9 / hbm_peak, 4),
                     "dram_bytes_per_iter": ppr_dram,
                     "dram_bytes_source": "ncu dram__bytes_read+write of k_ppr_wide at R-MAT 22, scaled by m",
                     "work_bytes_per_iter": ppr_bytes,
                     "work_bytes_over_time_frac": round(ppr_bytes / (t / 1e3) / 1e9 / hbm_peak, 4),
                     "storage": "bf16 rows of 128 seeds, fp32 sums"}
    # (b) many small graphs: one union; BFS from every part's vertex 0 plus CC,
    # submitted as one CUDA graph launch (gg_batch_bfs_cc), with the knobs the
    # autotuner picks on a 200-graph union of the same family
    from graptor_b200 import autotune as AT
    t0 = time.time()
    parts = small_graph_batch(ctx, n_small)
    U, base = gg.graph_union(ctx, parts)
    for p in parts:
        p.close()
    build_s = time.time() - t0

    def batch_runs(reps=3):
        gg.batch_bfs_cc(U, base[:-1], host=False)
        runs = []
        for _ in range(reps):
            bs, cs = gg.RunStats(), gg.RunStats()
            w0 = time.perf_counter()
            _, _, glaunch, kernels = gg.batch_bfs_cc(U, base[:-1], host=False, bfs_stats=bs, cc_stats=cs)
            runs.append((bs.total_ms, (time.perf_counter() - w0) * 1e3, bs, cs, glaunch, kernels))
        runs.sort(key=lambda r: r[0])
        return runs[len(runs) // 2]

    t_def = batch_runs()
    knob_names = ["bin_small_max", "bin_medium_max", "pull_k", "push_k", "large_chunk", "blocks_per_sm",
                  "heavy_deg", "heavy_chunk", "persistent", "cc_hook"]
    defaults = {k: gg.tuning_get(k) for k in knob_names}
    try:
        tparts = small_graph_batch(ctx, 200, seed=7000)
        TU, tbase = gg.graph_union(ctx, tparts)
        for p in tparts:
            p.close()
        ta = time.time()
        tuned = AT.tune_graph(TU, gg.TUNE_BFS | gg.TUNE_CC, nroots=4, passes=1, reps=2)
        tune_s = time.time() - ta
        TU.close()
        gg.graph_retune(U)  # heavy-row tables with the tuned cut
        t_tun = batch_runs()
    except Exception:
        AT.apply(defaults)  # later measurements run with the default knobs
        gg.graph_retune(U)
        raise
    use_tuned = t_tun[0] <= t_def[0]
    if not use_tuned:
        AT.apply(defaults)
        gg.graph_retune(U)
    tb, wall, bst, cst, glaunch, kernels = t_tun if use_tuned else t_def
    # parity on every part: the checker (the reference leg) runs the oracle's
    # multi-root BFS and CC over the union and compares
    lv, lb, _, _ = gg.batch_bfs_cc(U, base[:-1])
    uoff, uadj = U.download()
    roots0 = base[:-1].copy()
    union_n = U.n

    def check_union(O, res):
        p0 = time.time()
        OU = O.Graph(union_n, uoff, uadj)
        res["bfs_levels_bitexact"] = bool(np.array_equal(lv, O.bfs_level_multi(OU, roots0)))
        res["cc_labels_bitexact"] = bool(np.array_equal(lb, O.cc(OU)))
        res["wall_s"] = round(time.time() - p0, 1)

    sg_parity = {"parts": n_small, "checked_against": "oracle multi-root BFS and CC over the union"}
    REF_CHECKS.append((check_union, sg_parity))
    out["small_graphs"] = {"graphs": n_small, "n": U.n, "m": U.m, "build_s": round(build_s, 1),
                           "bfs_cc_ms": round(tb, 3), "bfs_cc_wall_ms": round(wall, 3),
                           "bfs_iterations": bst.iterations, "cc_iterations": cst.iterations,
                           "graph_launches": glaunch, "kernels_in_launch": int(kernels),
                           "bfs_gteps": round(bst.edges_reached / 2.0 / (tb / 1e3) / 1e9, 2),
                           "graphs_per_s": round(n_small / (tb / 1e3), 1),
                           "default_knobs_ms": round(t_def[0], 3), "tuned_knobs_ms": round(t_tun[0], 3),
                           "knobs": tuned["knobs"] if use_tuned else "defaults (the tuned ones were slower)",
                           "tuned_on": "a 200-graph union of the same family (BFS from 4 part roots + CC)",
                           "tune_s": round(tune_s, 1),
                           "parity": sg_parity}
    AT.apply(defaults)
    gg.graph_retune(U)
    U.close()
    return out


# ---------------------------------------------------------------------------
# our arm
# ---------------------------------------------------------------------------
def run_ours(args, ws, rank, local):
    from graptor_b200 import gg
    import torch

    hbm_peak, peak_kind = peaks()
    ctx = gg.Context(local)
    t0 = time.time()
    g = ctx.rmat(args.scale, EDGE_FACTOR << args.scale, GRAPH_SEED)
    gen_s = time.time() - t0
    off, adj = g.download()
    deg = np.diff(off).astype(np.int64)
    roots = pick_roots(deg)
    n, m = g.n, g.m

    lvl = g.prop(gg.I32)
    # variant choice per step: the learned selector (trained on other graphs:
    # R-MAT scales 18-22, ER, grids), the density threshold as its fallback;
    # the levels do not depend on the choice
    sel = None
    if args.select == "learned":
        from graptor_b200.selector_train import load_selector
        sel = load_selector(ctx)
    if sel is not None:
        gg.attach_selector(g, sel)
        opts = gg.default_opts(gg.THRESH_LEARNED, collect=True)
        select_desc = ("learned selector (graptor_b200/data/selector.npz, trained on R-MAT scales 18-22, ER and "
                       "grids, not on this graph), density threshold m/20 as its fallback")
    else:
        opts = gg.default_opts(collect=True)
        select_desc = "density threshold m/20"
    seq = replica_roots(roots, ws, rank, args.warmup + args.steps)

    # ---- warm-up ----
    for k in range(args.warmup):
        g.bfs_level(seq[k], level=lvl, host=False, opts=opts)
    ctx.sync()

    # ---- timed BFS steps (device time, CUDA events on the library's stream) ----
    stream = torch.cuda.ExternalStream(ctx.stream())
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    sampler = ClockSampler(local)
    stats = [gg.RunStats() for _ in range(args.steps)]
    launches0 = ctx.launches
    barrier(ws)
    torch.cuda.synchronize()
    sampler.start()
    ev0.record(stream)
    for k in range(args.steps):
        g.bfs_level(seq[args.warmup + k], level=lvl, host=False, opts=opts, stats=stats[k])
    ev1.record(stream)
    torch.cuda.synchronize()
    clocks = sampler.stop()
    launches = ctx.launches - launches0
    t_ms = ev0.elapsed_time(ev1)
    t_ms_max = max_over_ranks(t_ms, ws)
    barrier(ws)

    half_edges = sum(st.edges_reached for st in stats) / 2.0
    total_half_edges = sum_over_ranks(half_edges, ws)
    value = total_half_edges / (t_ms_max / 1e3) / 1e9
    # the same steps with the density threshold alone, timed the same way
    value_threshold = None
    if sel is not None:
        topts = gg.default_opts(collect=True)
        barrier(ws)
        torch.cuda.synchronize()
        ev0.record(stream)
        for k in range(args.steps):
            g.bfs_level(seq[args.warmup + k], level=lvl, host=False, opts=topts)
        ev1.record(stream)
        torch.cuda.synchronize()
        t_thr = max_over_ranks(ev0.elapsed_time(ev1), ws)
        value_threshold = total_half_edges / (t_thr / 1e3) / 1e9
    per_root = [st.edges_reached / 2.0 / (st.total_ms / 1e3) / 1e9 for st in stats]

    # roofline of the traversal kernel.  By default a BFS is one launch of
    # k_bfs_run, whose steps (their barrier and the next step's decision
    # included) are listed by kind beside it; other drivers launch a kernel per
    # step, whose span (first CTA start to last CTA end) is stamped by the
    # kernel, and the dominant one by summed time is taken
    ktime = {}
    kbytes = {}
    stime = {}
    for st in stats:
        for it in range(st.iterations):
            v = st.variant[it]
            ktime[v] = ktime.get(v, 0.0) + st.kernel_ms[it]
            stime[v] = stime.get(v, 0.0) + st.iter_ms[it]
            kbytes[v] = kbytes.get(v, 0.0) + bfs_bytes(n, st, it)
    resident = all(st.kernels == 2 for st in stats)  # k_bfs_start and k_bfs_run
    if resident:
        dom_name, nlaunch = "k_bfs_run", len(stats)
        dom_ms, dom_bytes = sum(ktime.values()), sum(kbytes.values())
        kernel_names = {gg.VAR_PULL_DENSE: "k_bfs_run: pull steps", gg.VAR_PUSH_SPARSE: "k_bfs_run: push steps"}
    else:
        kernel_names = {gg.VAR_PULL_DENSE: "k_pull", gg.VAR_PUSH_SPARSE: "k_push_binned",
                        gg.VAR_PUSH_MERGE: "k_push_merge", gg.VAR_PUSH_DENSE: "k_push_dense"}
        dom = max(ktime, key=ktime.get)
        nlaunch = sum(1 for st in stats for it in range(st.iterations) if st.variant[it] == dom)
        dom_name, dom_ms, dom_bytes = kernel_names[dom], ktime[dom], kbytes[dom]
    achieved = dom_bytes / (dom_ms / 1e3) / 1e9
    bfs_iter_total_ms = sum(ktime.values())
    bfs_pass_bytes = 8.0 * (n + 1) + 4.0 * m + 8.0 * n
    # whole-run roofline: the algorithmic bytes of every iteration of every
    # timed step over the whole timed region (launch gaps and decisions included)
    bfs_all_bytes = sum(kbytes.values())
    kernel_roofline = {}
    for v, t in ktime.items():
        nl = sum(1 for st in stats for it in range(st.iterations) if st.variant[it] == v)
        a = kbytes[v] / (t / 1e3) / 1e9
        kernel_roofline[kernel_names[v]] = {"launches": nl, "ms_per_launch": round(t / max(nl, 1), 4),
                                            "step_ms_per_launch": round(stime[v] / max(nl, 1), 4),
                                            "bytes_per_launch": round(kbytes[v] / max(nl, 1)),
                                            "achieved_gbs": round(a, 1), "frac": round(a / hbm_peak, 4)}

    out = {}
    wall = {"graph_build_and_bfs": round(time.time() - t0, 1)}  # wall seconds per part of this run
    if rank == 0:
        out["bfs"] = {
            "variant_selection": select_desc,
            "value_threshold_gteps": round(value_threshold, 3) if value_threshold is not None else None,
            "gteps_mean": round(float(np.mean(per_root)), 3),
            "gteps_hmean": round(float(len(per_root) / np.sum(1.0 / np.array(per_root))), 3),
            "ms_per_root_mean": round(float(np.mean([st.total_ms for st in stats])), 4),
            "iterations_mean": round(float(np.mean([st.iterations for st in stats])), 2),
            "kernel_share": {kernel_names[v]: round(t / bfs_iter_total_ms, 3) for v, t in ktime.items()},
            "kernel_ms_per_root": round(bfs_iter_total_ms / args.steps, 4),
            "step_ms_per_root": round(sum(stime.values()) / args.steps, 4),
            "kernel_roofline": kernel_roofline,
            "whole_run_bytes_per_step": round(bfs_all_bytes / args.steps),
            "whole_run_frac_of_hbm": round(bfs_all_bytes / (t_ms / 1e3) / 1e9 / hbm_peak, 4),
            "one_pass_frac_of_hbm": round(bfs_pass_bytes / (np.mean([st.total_ms for st in stats]) / 1e3)
                                          / 1e9 / hbm_peak, 4),
        }

    tw = time.time()
    # ---- CC (CCv to convergence) ----
    if not args.quick:
        lab = g.prop(gg.U32)
        g.cc(label=lab, host=False)
        cc_ms = []
        cst = gg.RunStats()
        for _ in range(3):
            st = gg.RunStats()
            g.cc(label=lab, host=False, opts=gg.default_opts(gg.THRESH_FRAC, 5), stats=st)
            cc_ms.append(st.total_ms)
            cst = st
        cc_best = float(np.median(cc_ms))
        # one pass over the CSC and the labels, as the BFS line's one-pass fraction
        cc_pass = 8.0 * (n + 1) + 4.0 * m + 8.0 * n
        cc_all = sum(cc_bytes(n, m, cst, it) for it in range(min(cst.iterations, gg.MAX_ITERS)))
        out["cc"] = {"ms": round(cc_best, 3), "gedges_per_s": round(m / (cc_best / 1e3) / 1e9, 3),
                     "iterations": cst.iterations,
                     "variants": [gg.VARIANT_NAMES.get(cst.variant[i], "hook")
                                  for i in range(min(cst.iterations, gg.MAX_ITERS))],
                     "whole_run_bytes": round(cc_all),
                     "whole_run_frac_of_hbm": round(cc_all / (cc_best / 1e3) / 1e9 / hbm_peak, 4),
                     "one_pass_frac_of_hbm": round(cc_pass / (cc_best / 1e3) / 1e9 / hbm_peak, 4)}

        # ---- k-core (KC_bucket: peel floors with count-down pushes) ----
        core = g.prop(gg.U32)
        g.kcore(coreness=core, host=False)
        kc_ms = []
        for _ in range(3):
            st = gg.RunStats()
            _, kc_largest = g.kcore(coreness=core, host=False, stats=st)
            kc_ms.append(st.total_ms)
        kc_best = float(np.median(kc_ms))
        # one count-down per edge end (every edge is pushed from both ends)
        out["kcore"] = {"ms": round(kc_best, 3), "gedges_per_s": round(m / (kc_best / 1e3) / 1e9, 3),
                        "largest_core": kc_largest, "peel_steps": st.iterations,
                        "floors": int(st.vertices_reached), "kernels": int(st.kernels)}
        core.close()

        # ---- PageRank (PRv: FP32 storage, double gather accumulation, 20 iterations) ----
        x = g.prop(gg.F32)
        prs = {}
        for name, fmt, acc64 in [("f32", gg.F32, True), ("f32_accf32", gg.F32, False), ("bf16", gg.BF16, False),
                                 ("f16", gg.F16, False), ("fp8e4m3", gg.FP8E4M3, False),
                                 ("cfp_6_10", gg.CFP_6_10, False)]:
            g.pagerank(maxiter=3, tol=0, contrib=fmt, accum_f64=acc64, x=x, host=False)
            ts = []
            for _ in range(3):
                st = gg.RunStats()
                # tol < 0: exactly 20 iterations (a low-precision run can reach
                # an exact fixed point, delta = 0, before that)
                g.pagerank(maxiter=20, tol=-1.0, contrib=fmt, accum_f64=acc64, renorm_f32=(name == "f32"),
                           x=x, host=False, stats=st)
                assert st.iterations == 20
                ts.append(st.total_ms / st.iterations)
            t_it = float(np.median(ts))
            prs[name] = {"ms_per_iter": round(t_it, 4), "gedges_per_s_per_iter": round(m / (t_it / 1e3) / 1e9, 3)}
        base = prs["f32"]["ms_per_iter"]
        for k, v in prs.items():
            v["speedup_vs_f32"] = round(base / v["ms_per_iter"], 3)
        pr_bytes_f32 = 8.0 * (n + 1) + 4.0 * m + 4.0 * m + n * (4 + 4 + 4 + 4)
        prs["f32"]["frac_of_hbm"] = round(pr_bytes_f32 / (base / 1e3) / 1e9 / hbm_peak, 4)
        out["pr"] = prs

    # The secondary measurements below run after the headline BFS timing; a
    # failure in one of them is recorded in its entry and the others still run.
    def section(name, fn):
        ts = time.time()
        try:
            out[name] = fn()
        except Exception as e:  # noqa: BLE001 -- reported in the JSON line
            import traceback
            out[name] = {"error": f"{type(e).__name__}: {e}"[:400],
                         "where": traceback.format_exc().strip().splitlines()[-3:]}
        wall[name] = round(time.time() - ts, 1)

    wall["cc_kcore_pagerank"] = round(time.time() - tw, 1)

    # ---- learned selector vs threshold vs oracle-best (held-out RMAT-24 and a road-like grid) ----
    if not args.quick and not args.no_selector and rank == 0:
        def sel_section():
            grid = ctx.grid(2896, 2896, seed=77, del_bp=100)  # 2^23 vertices, 1% edges deleted
            try:
                return selector_eval(ctx, [("rmat24", g, [int(r) for r in roots[:4]]), ("grid2896", grid, [0])])
            finally:
                grid.close()
        section("selector", sel_section)

    # ---- PageRank precision workloads ----
    if not args.quick and not args.no_precision and rank == 0:
        section("pr_precision", lambda: precision_eval(ctx, hbm_peak, with_ref=not args.no_cpu_baseline))

    # ---- batching: multi-source BFS, 128-seed PPR (R-MAT 22), many small graphs ----
    if not args.quick and not args.no_batch and rank == 0:
        def batch_section():
            g22 = ctx.rmat(22, EDGE_FACTOR << 22, GRAPH_SEED)
            try:
                off22, _ = g22.download()
                b = batch_eval(ctx, g22, pick_roots(np.diff(off22).astype(np.int64)), hbm_peak, args.batch_graphs)
                b["graph"] = "rmat22 ef16 seed 1 (msbfs64, ppr128)"
                return b
            finally:
                g22.close()
        section("batch", batch_section)

    # ---- e2e: public C-ABI call, graph uploaded from host memory, every step's
    # levels delivered to page-locked host memory (gg_bfs_level_host_async: the
    # copy of step k runs behind the BFS of step k+1; the last one is waited
    # for inside the timed region) ----
    e2e = None
    te = time.time()
    if not args.quick:
        pins = [torch.empty(n, dtype=torch.int32, pin_memory=True).numpy() for _ in range(2)]
        t_up = time.time()
        gh = ctx.upload(off, adj, symmetric=True)
        upload_s = time.time() - t_up
        eopts = None
        if sel is not None:
            gg.attach_selector(gh, sel)
            eopts = gg.default_opts(gg.THRESH_LEARNED)
        for k in range(min(args.warmup, 3)):
            gh.bfs_level_host_async(seq[k], out=pins[k % 2], opts=eopts)
        gh.bfs_level_host_wait()
        barrier(ws)
        t1 = time.perf_counter()
        e2e_edges = 0.0
        for k in range(args.steps):
            st = gg.RunStats()
            gh.bfs_level_host_async(seq[args.warmup + k], out=pins[k % 2], opts=eopts, stats=st)
            e2e_edges += st.edges_reached / 2.0
        gh.bfs_level_host_wait()
        e2e_s = max_over_ranks(time.perf_counter() - t1, ws)
        e2e_val = sum_over_ranks(e2e_edges, ws) / e2e_s / 1e9
        # the last step's levels, checked against the device-resident run of the same root
        last_ok = bool(np.array_equal(pins[(args.steps - 1) % 2], g.bfs_level(seq[args.warmup + args.steps - 1])))
        e2e = {"value": round(e2e_val, 4), "unit": "GTEPS", "h2d_bytes_per_step": 4,
               "d2h_bytes_per_step": 4 * n, "graph_upload_s": round(upload_s, 3),
               "api": "gg_bfs_level_host_async (levels to page-locked host memory, copy behind the next BFS)",
               "last_step_levels_match": last_ok}
        gh.close()
        del gh
    wall["e2e"] = round(time.time() - te, 1)

    # ---- CPU baseline and parity: the reference build on this host, same graph ----
    cpu, parity = None, None
    if rank == 0 and ws == 1 and not args.no_cpu_baseline:
        tr = time.time()
        try:
            cpu, parity = reference_leg(g, roots, args, lvl)
        except Exception as e:  # the baseline is reported, never required
            cpu = {"value": None, "unit": "GTEPS", "cores": os.cpu_count(), "kind": "reference",
                   "sample": f"failed: {e}"[:300]}
        wall["reference_leg"] = round(time.time() - tr, 1)

    if rank == 0:
        line = {
            "metric": METRIC, "value": round(value, 4), "unit": "GTEPS", "n_gpus": ws,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(t_ms_max / args.steps, 4),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "int32",
            "data": "synthetic",
            "config": {"workload": WORKLOAD, "scale": args.scale, "edge_factor": EDGE_FACTOR, "n": n, "m": m,
                       "roots": NROOTS, "parallelism": f"replicas{ws}" if ws > 1 else "single",
                       "variant_selection": "learned" if sel is not None else "threshold",
                       "l2": "graph 2.3 GB > 126 MB L2, no flush between steps",
                       "graph_build_s": round(gen_s, 2)},
            "roofline": {"bound": "hbm", "kernel": dom_name, "achieved": round(achieved, 1),
                         "peak": hbm_peak, "unit": "GB/s", "frac": round(achieved / hbm_peak, 4),
                         "traffic": K_BFS_TRAFFIC_PER_RUN * n / (1 << 24) if resident else None,
                         "traffic_source": "ncu dram__bytes_read+write of k_bfs_run, scale-23 capture scaled by n",
                         "peak_kind": peak_kind, "launches": nlaunch,
                         "bytes_per_launch": round(dom_bytes / max(nlaunch, 1)),
                         "ms_per_launch": round(dom_ms / max(nlaunch, 1), 4),
                         "duration": "from the run's first step to its end, stamped by the kernel" if resident else
                                     "kernel span per launch (first CTA start to last CTA end, stamped by the "
                                     "kernel)"},
            "clocks": clocks, "gpu_launches": launches,
            "e2e": e2e, "cpu_baseline": cpu, "parity": parity, "wall_s": wall,
        }
        line.update(out)
        print(json.dumps(line))
    return 0


# ---------------------------------------------------------------------------
# single workloads for profilers (--case): one JSON line with device times and
# the per-iteration variant / frontier / kernel-time table of the last run
#
#   python bench.py --case bfs   --scale 24 --roots 4
#   python bench.py --case pr    --scale 24 --format bf16 --iters 5
#   python bench.py --case cc    --graph grid --side 2896
#   python bench.py --case kc    --scale 24
#   python bench.py --case msbfs --scale 22
#   python bench.py --case ppr   --scale 22 --iters 5
# ---------------------------------------------------------------------------
def case_formats():
    from graptor_b200 import gg
    return {"f32": gg.F32, "bf16": gg.BF16, "f16": gg.F16, "fp8": gg.FP8E4M3, "cfp": gg.CFP_6_10,
            "bf16t": gg.BF16_TRUNC, "f64": gg.F64}


def case_roots(g, k: int, seed: int = 12345):
    off, _ = g.download()
    nz = np.flatnonzero(np.diff(off))
    return [int(r) for r in np.random.default_rng(seed).choice(nz, size=k, replace=False)]


def iter_table(st):
    from graptor_b200 import gg
    t = min(st.iterations, gg.MAX_ITERS)
    return [[i, st.variant[i], int(st.nactv[i]), int(st.nacte[i]), round(st.iter_ms[i], 4), round(st.kernel_ms[i], 4)]
            for i in range(t)]


def run_case(a):
    from graptor_b200 import gg
    for kv in a.knob:
        name, val = kv.split("=")
        gg.tuning_set(name, int(val))
    if a.persistent is not None:
        gg.tuning_set("persistent", a.persistent)
    if a.graph_mode is not None:
        gg.tuning_set("graph", a.graph_mode)
    ctx = gg.Context(0)
    if a.graph == "grid":
        g = ctx.grid(a.side, a.side, 77, del_bp=100)
    elif a.graph == "er":
        g = ctx.er(1 << a.scale, 32.0, 1, dangling_bp=100, symmetric=False)
    else:
        g = ctx.rmat(a.scale, 16 << a.scale, 1)
    out = {"case": a.case, "graph": a.graph, "n": g.n, "m": g.m, "persistent": gg.tuning_get("persistent"),
           "knobs": a.knob}
    opts = gg.default_opts(gg.THRESH_LEARNED if a.threshold == "learned" else gg.THRESH_DEFAULT, collect=True)
    if a.threshold == "learned":
        from graptor_b200.selector_train import load_selector
        gg.attach_selector(g, load_selector(ctx))  # (the graph keeps its copy of the weights)
    if a.case == "bfs":
        rs = case_roots(g, a.roots)
        for r in rs[: a.warmup]:
            g.bfs_level(r, host=False)
        tot, ker, last, worst = [], [], None, None
        for _ in range(a.reps):
            for r in rs:
                st = gg.RunStats()
                g.bfs_level(r, host=False, opts=opts, stats=st)
                tot.append(st.total_ms)
                ker.append(sum(st.kernel_ms[i] for i in range(min(st.iterations, gg.MAX_ITERS))))
                last = st
                if worst is None or st.total_ms > worst[1]:
                    worst = (r, st.total_ms, iter_table(st))
        out.update(ms_per_bfs=round(float(np.mean(tot)), 4), kernel_ms_per_bfs=round(float(np.mean(ker)), 4),
                   ms_per_bfs_median=round(float(np.median(tot)), 4),
                   per_root_ms=[round(x, 3) for x in tot[: len(rs)]], iterations=iter_table(last),
                   worst_root=worst[0], worst_ms=round(worst[1], 3), worst_iterations=worst[2])
    elif a.case == "cc":
        for _ in range(a.warmup):
            g.cc(host=False)
        ts = []
        for _ in range(a.reps):
            st = gg.RunStats()
            g.cc(host=False, opts=gg.default_opts(gg.THRESH_FRAC, 5), stats=st)
            ts.append(st.total_ms)
        out.update(ms=round(float(np.median(ts)), 4), iterations=iter_table(st))
    elif a.case == "kc":
        for _ in range(a.warmup):
            g.kcore(host=False)
        ts = []
        for _ in range(a.reps):
            st = gg.RunStats()
            # (records per step: the host-driven peel)
            opts = gg.default_opts(gg.THRESH_ALWAYS_SPARSE, collect=True) if a.reps == 1 else None
            _, largest = g.kcore(host=False, opts=opts, stats=st)
            ts.append(st.total_ms)
        out.update(ms=round(float(np.median(ts)), 4), largest_core=largest, peel_steps=st.iterations,
                   floors=int(st.vertices_reached), kernels=int(st.kernels),
                   iterations=iter_table(st) if a.reps == 1 else None)
    elif a.case == "pr":
        fmt = case_formats()[a.format]
        for _ in range(a.warmup):
            g.pagerank(maxiter=2, tol=-1.0, contrib=fmt, host=False)
        ts = []
        for _ in range(a.reps):
            st = gg.RunStats()
            g.pagerank(maxiter=a.iters, tol=-1.0, contrib=fmt, accum_f64=fmt in (gg.F32, gg.F64), host=False,
                       stats=st)
            ts.append(st.total_ms / max(st.iterations, 1))
        out.update(format=a.format, ms_per_iter=round(float(np.median(ts)), 4))
    elif a.case == "msbfs":
        rs = case_roots(g, 64)
        for _ in range(a.warmup):
            gg.msbfs(g, rs, host=False)
        ts = []
        for _ in range(a.reps):
            st = gg.RunStats()
            gg.msbfs(g, rs, host=False, stats=st)
            ts.append(st.total_ms)
        out.update(ms=round(float(np.median(ts)), 4), edges_reached=int(st.edges_reached),
                   iterations=[[i, st.variant[i], round(st.iter_ms[i], 4)] for i in range(st.iterations)])
    else:
        rs = case_roots(g, min(a.seeds, gg.PPR_MAX_SEEDS))
        for _ in range(a.warmup):
            gg.ppr(g, rs, iters=1, host=False)
        ts = []
        for _ in range(a.reps):
            st = gg.RunStats()
            gg.ppr(g, rs, iters=a.iters, host=False, stats=st)
            ts.append(st.total_ms / max(a.iters, 1))
        out.update(seeds=len(rs), ms_per_iter=round(float(np.median(ts)), 4))
    print(json.dumps(out))
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=64)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--scale", type=int, default=SCALE)
    ap.add_argument("--cpu-roots", type=int, default=NROOTS,
                    help="roots of the reference's BFS runs (CPU baseline and level parity)")
    ap.add_argument("--no-cpu-baseline", action="store_true", help="skip the reference leg (baseline and parity)")
    ap.add_argument("--no-parity-cc-pr", action="store_true", help="reference leg: BFS only")
    ap.add_argument("--quick", action="store_true", help="BFS only (no CC/PR/e2e)")
    ap.add_argument("--no-selector", action="store_true", help="skip the learned-selector evaluation")
    ap.add_argument("--select", default="learned", choices=["learned", "threshold"],
                    help="variant choice of the timed BFS steps (levels are the same either way)")
    ap.add_argument("--no-batch", action="store_true", help="skip the batched-traversal measurements")
    ap.add_argument("--no-precision", action="store_true", help="skip the PageRank precision workloads")
    ap.add_argument("--batch-graphs", type=int, default=2000, help="small graphs in the union workload")
    # single workloads for profilers
    ap.add_argument("--case", default=None, choices=["bfs", "pr", "cc", "kc", "msbfs", "ppr"],
                    help="run one workload for a profiler instead of the benchmark")
    ap.add_argument("--graph", default="rmat", choices=["rmat", "grid", "er"])
    ap.add_argument("--side", type=int, default=2048)
    ap.add_argument("--roots", type=int, default=4)
    ap.add_argument("--format", default="f32", choices=["f32", "bf16", "f16", "fp8", "cfp", "bf16t", "f64"])
    ap.add_argument("--iters", type=int, default=5)
    ap.add_argument("--reps", type=int, default=2)
    ap.add_argument("--seeds", type=int, default=128)
    ap.add_argument("--persistent", type=int, default=None, help="tuning knob: device-driven analytics mask")
    ap.add_argument("--threshold", default="default", choices=["default", "learned"])
    ap.add_argument("--graph-mode", type=int, default=None, help="tuning knob: graph-driven BFS levels (0/1)")
    ap.add_argument("--knob", action="append", default=[], help="name=value of a tuning knob (repeatable)")
    args = ap.parse_args()
    if args.case:
        return run_case(args)
    args.warmup = max(args.warmup, 3) if args.impl == "ours" else args.warmup
    ws, rank, local = dist_setup(args)
    try:
        if args.impl == "reference":
            rc = run_reference_arm(args, ws, rank)
        else:
            rc = run_ours(args, ws, rank, local)
    finally:
        if ws > 1:
            import torch.distributed as dist
            dist.destroy_process_group()
    return rc


if __name__ == "__main__":
    sys.exit(main())
