"""Benchmark: uv Newton solves/s of the SSA (SSTREAM) diagnostic solve on B200,
mixed precision vs plain FP64, batched and served.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Headline workload (one "step" = one batched uv Newton solve of 256 meshes):
256 independent ice-stream/ice-shelf problems on 100 km x 50 km rectangles,
P1 triangles, sizes log-uniform in 2k-200k elements (10.56M elements, 5.35M
nodes in total, seeded synthetic fields: bed, thickness with bumps, smoothed
Glen A and Weertman C, n=m=3; u=v=0 at x=0, free-slip sides, calving front),
each solved from u=v=0 to rForce<1e-20.  The inputs (~0.5 GB) exceed the
126 MB L2; a 512 MB buffer is also written between timed steps.

Reported:
  value         solves/s of the batched mixed-precision form (FP32 tangents
                and PCG, FP64 residual/line search/update), inputs resident in HBM
  plain_fp64    the plain form: one mesh at a time, all FP64, on a size-stratified
                sample of 64 of the 256 meshes
  batched_fp64  the batched form in FP64
  e2e           the batched mixed form through the public API with host arrays
                (host->device copies and the device->host read of every solution
                inside the timed region)
  serving       the served form: Poisson arrivals (200 req/s) over 16 resident
                templates of 5k-500k elements, lognormal C perturbations, warm
                starts; p50/p99 latency and solves/s
  roofline      the dominant kernel by measured device time (CUDA events)
  cpu_baseline  the CPU restatement of the reference (oracle/ua_ref.py with its
                element loop compiled, oracle/ua_ref_asm.cpp) on every host core over
                16 meshes spanning the batch's size range; the GPU's FP64 and mixed
                solutions of those meshes against the oracle's (rel_err_vs_oracle)

Multi-GPU: independent replicas (whole meshes are the independent units; one
solve of one mesh does not shard), one process per GPU, time = max over ranks.
``--impl reference`` times the CPU restatement on the host cores: step k of K
solves the meshes of size rank k mod K, the K steps back to back on a process
pool (one oracle process per core), so the timed steps solve the whole batch once.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

BATCH = 256
CPU_SAMPLE = 16  # meshes of the CPU baseline (one per size stratum) and of the error against the oracle
METRIC = "uv Newton solves/s (batched, mixed FP32/FP64, <=1e-8 rel err vs FP64)"


def _workload(count):
    return (f"batched uv diagnostic Newton solves (SSTREAM2dNR2): {count} independent ice stream/shelf meshes "
            f"100x50 km, P1, log-uniform 2k-200k elements (seed 12345), u=v=0 start, rForce<1e-20")


# ----------------------------------------------------------------------------- CPU reference arm

def _oracle_solve(k, count, return_solution=False):
    """One full oracle solve of batch problem k (child process): the numpy/scipy restatement with
    its element loop in the compiled C++ restatement (one thread); returns
    (seconds, converged, Nele, k, solution or None)."""
    sys.path.insert(0, ROOT)
    from oracle import ua_ref as R
    from uasource_b200 import synth
    R.use_compiled_element_loop(True, 1)
    P = synth.batch_problem(k, count)
    mua = R.create_mua(P.coordinates, P.connectivity)
    p = R.Params()
    p.set_force_tolerance(1e-20)
    F = R.Fields(h=P.h, S=P.S, B=P.B, rho=P.rho, AGlen=P.AGlen, n=P.n, C=P.C, m=P.m, ub=P.ub, vb=P.vb)
    bcs = R.BCs(ubFixedNode=P.ubFixedNode, ubFixedValue=P.ubFixedValue, vbFixedNode=P.vbFixedNode,
                vbFixedValue=P.vbFixedValue)
    t = time.perf_counter()
    res = R.uv(p, mua, bcs, F)
    dt = time.perf_counter() - t
    sol = None
    if return_solution:
        import numpy as np
        sol = np.concatenate([res.ub, res.vb])
    return dt, bool(res.converged), int(P.Nele), int(k), sol


def _oracle_solve_args(a):
    return _oracle_solve(*a)


def _size_ranks(count):
    from uasource_b200 import synth
    import numpy as np
    return np.argsort(synth.batch_sizes(count), kind="stable")


def _stratified(count, n, offset):
    """n batch indices, one per size stratum (strata of equal count), at a fractional offset."""
    order = _size_ranks(count)
    return [int(order[min(count - 1, int((j + offset) * count / n))]) for j in range(n)]


def _host_cpu():
    """Host core count and CPU model (from /proc/cpuinfo)."""
    model = None
    try:
        for ln in open("/proc/cpuinfo"):
            if ln.startswith("model name"):
                model = ln.split(":", 1)[1].strip()
                break
    except OSError:
        pass
    return os.cpu_count() or 1, model


def _pool(workers):
    import multiprocessing as mp
    for v in ("OMP_NUM_THREADS", "OPENBLAS_NUM_THREADS", "MKL_NUM_THREADS"):
        os.environ[v] = "1"
    return mp.get_context("spawn").Pool(workers)


def run_reference(args):
    """The reference's CPU algorithm on the host cores (the oracle port: MATLAB cannot run on
    this machine).  Step k of K solves the meshes whose size rank is k modulo K, a stratified
    1/K share of the batch; the K timed steps run back to back on a process pool with one
    oracle process per core, largest meshes first, so together they solve each mesh of the
    batch exactly once and the value is the batch throughput of the host."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return 0
    count = args.batch
    cores, model = _host_cpu()
    workers = max(1, min(cores, 64))
    order = _size_ranks(count)
    K = max(1, args.steps)
    steps = [[int(order[r]) for r in range(k, count, K)] for k in range(K)]
    size_rank = {int(i): r for r, i in enumerate(order)}
    tasks = sorted((i for st in steps for i in st), key=lambda i: -size_rank[i])
    with _pool(workers) as pool:
        for _ in range(args.warmup):  # imports, page cache, the compiled loop: the smallest mesh per worker
            pool.map(_oracle_solve_args, [(int(order[0]), count)] * workers)
        t0 = time.perf_counter()
        res = list(pool.imap_unordered(_oracle_solve_args, [(i, count) for i in tasks]))
        el = time.perf_counter() - t0
    value = len(res) / el
    sizes = sorted(r[2] for r in res)
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": "solves/s", "n_gpus": args.gpus,
        "steps": K, "warmup": args.warmup, "ms_per_step": 1000 * el / K,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": _workload(count), "l2": "n/a (CPU)",
                   "step_rule": f"step k solves the meshes of size rank k mod {K} (stratified 1/{K} of the batch); "
                                f"the {K} steps run back to back on the pool, largest first, covering the "
                                f"{count} meshes once"},
        "cpu_baseline": {"value": value, "unit": "solves/s", "cores": workers, "kind": "port",
                         "nproc": cores, "cpu_model": model,
                         "sample": f"all {len(res)} meshes of the batch ({sizes[0]}-{sizes[-1]} elements), one "
                                   f"oracle process per core (numpy/scipy restatement, element loop in C++, "
                                   f"SuperLU with UMFPACK's symmetric strategy)"},
        "e2e": {"value": value, "unit": "solves/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "converged": int(sum(r[1] for r in res)),
    }
    print(json.dumps(line), flush=True)
    return 0


def _cpu_baseline_pool(count, n):
    """The oracle on every host core over a stratified sample of n meshes spanning the whole size
    range (one per size stratum, the stratum's middle mesh); returns the line's cpu_baseline and
    the oracle's solutions by batch index (for the GPU's error against the oracle)."""
    cores, model = _host_cpu()
    workers = max(1, min(cores, n))
    picks = _stratified(count, n, 0.5)
    t0 = time.perf_counter()
    with _pool(workers) as pool:
        res = pool.map(_oracle_solve_args, [(i, count, True) for i in sorted(picks, key=lambda i: -i)])
    el = time.perf_counter() - t0
    ns = [r[2] for r in res]
    out = {"value": len(res) / el, "unit": "solves/s", "cores": workers, "kind": "port", "nproc": cores,
           "cpu_model": model,
           "sample": f"{len(res)} full oracle solves, one per size stratum of the batch ({min(ns)}-{max(ns)} "
                     f"elements), in parallel on {workers} processes; solves/s over the sample's wall time",
           "core_seconds": sum(r[0] for r in res)}
    return out, {r[3]: r[4] for r in res}


# ----------------------------------------------------------------------------- GPU arm

class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.path = None

    def start(self):
        import tempfile
        try:
            fd, self.path = tempfile.mkstemp(prefix=f"ua_clocks_gpu{self.index}_", suffix=".csv")
            self.f = os.fdopen(fd, "w")
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "200"], stdout=self.f,
                                         stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(5)
        except Exception:
            self.proc.kill()
        self.f.close()
        sm, smax, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        with open(self.path) as fh:
            rows = fh.readlines()
        os.unlink(self.path)
        for ln in rows:
            parts = [x.strip() for x in ln.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1])); smax = float(parts[2])
            except ValueError:
                continue
            for nm, v in zip(names, parts[5:9]):
                if v.lower() == "active":
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": smax,
                "reasons": sorted(reasons), "samples": len(sm)}


NAMES = ("h", "S", "B", "rho", "AGlen", "n", "C", "m")


# ----------------------------------------------------------------------------- replicas over ranks

def rank_barrier(world):
    if world > 1:
        import torch.distributed as dist
        dist.barrier()


def max_over_ranks_on(x, world, device):
    """Max of a per-rank time over all ranks (an all-reduce on `device`; identity at world 1)."""
    if world == 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return t.item()


def replica_throughput(world, solves_per_rank, t_max_ms):
    """Whole-job solves/s of `world` independent replicas that each ran `solves_per_rank`
    solves, timed as the slowest rank."""
    return world * solves_per_rank / (t_max_ms / 1000.0)


def run_ours(args):
    import numpy as np
    import torch
    import torch.distributed as dist
    import uasource_b200 as ua
    from uasource_b200 import lib as L, synth

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if world > 1:
        from datetime import timedelta
        dist.init_process_group("nccl", timeout=timedelta(seconds=300), device_id=dev)

    def barrier():
        rank_barrier(world)

    def max_over_ranks(x):
        return max_over_ranks_on(x, world, dev)

    count = args.batch
    # weak scaling over replicas: every rank solves its own batch of the same size distribution
    # (rank 0 the seeded headline batch, rank r the batch of seed + 1000 r)
    probs = synth.batch_problems(count, seed=12345 + 1000 * rank)
    node_off = np.concatenate([[0], np.cumsum([P.Nnodes for P in probs])])
    Nn_tot = int(node_off[-1])
    mua = ua.CreateMUABatch([(P.coordinates, P.connectivity) for P in probs], device=local)
    bcss = [ua.BCs.from_problem(P) for P in probs]
    # resident inputs: one concatenated float64 tensor per field, system-major
    dev_in = {k: torch.tensor(np.concatenate([getattr(P, k) for P in probs]), dtype=torch.float64, device=dev)
              for k in NAMES}
    ub = torch.zeros(Nn_tot, dtype=torch.float64, device=dev)
    vb = torch.zeros_like(ub)

    def ptrs(s):
        o = 8 * int(node_off[s])
        d = {k: v.data_ptr() + o for k, v in dev_in.items()}
        d["ub"] = ub.data_ptr() + o
        d["vb"] = vb.data_ptr() + o
        return d

    F_devs = [ptrs(s) for s in range(count)]
    flush = torch.zeros(64 * 1024 * 1024, dtype=torch.float64, device=dev)  # 512 MB > L2

    def ctrl_of(prec, **kw):
        c = ua.CtrlVar(precision=prec, krylov_rtol=1e-12 if prec == L.UA_PREC_FP64 else 1e-6, **kw)
        return c.set_force_tolerance(1e-20)

    ctrlmx = ctrl_of(L.UA_PREC_MIXED)
    ctrl64 = ctrl_of(L.UA_PREC_FP64)
    # the assembly schedule (patch shape, CTA size) tuned on this batch at its start state, before
    # any timing; every handle of this process then uses it (results do not depend on it)
    tune = None
    if not args.no_autotune:
        tune = ua.autotune(ctrlmx, mua, [ua.Fields.from_problem(P) for P in probs])

    def solve_batch(ctrl):
        ub.zero_(); vb.zero_()
        torch.cuda.synchronize()
        return ua.uv_batch_resident(ctrl, mua, F_devs, bcss, rhow=probs[0].rhow, g=probs[0].g)

    def timed(fn, steps, warmup, sampler=None):
        for _ in range(warmup):
            fn()
        barrier()
        torch.cuda.synchronize()
        if sampler:
            sampler.start()
        per, out = [], []
        e0 = torch.cuda.Event(enable_timing=True); e1 = torch.cuda.Event(enable_timing=True)
        for _ in range(steps):
            flush.add_(1.0)
            torch.cuda.synchronize()
            e0.record()
            r = fn()
            e1.record()
            torch.cuda.synchronize()
            per.append(e0.elapsed_time(e1))
            out.append(r)
        clocks = sampler.stop() if sampler else None
        barrier()
        return per, out, clocks

    if args.legs == "mixed":  # profiling runs: the timed batched mixed-precision solves only
        timed(lambda: solve_batch(ctrlmx), args.steps, args.warmup)
        mua.close()
        if world > 1:
            dist.destroy_process_group()
        return 0

    # FP64 batched solution: the reference for the error report
    infos64 = solve_batch(ctrl64)
    u64 = [torch.cat([ub[node_off[s]:node_off[s + 1]], vb[node_off[s]:node_off[s + 1]]]).cpu().numpy()
           for s in range(count)]

    # headline: batched mixed precision, resident inputs
    sampler = ClockSampler(local)
    per_mx, outs_mx, clocks = timed(lambda: solve_batch(ctrlmx), args.steps, args.warmup, sampler)
    infos_mx = outs_mx[-1]
    errs = []
    cpu_picks = set(_stratified(count, CPU_SAMPLE, 0.5))
    u_mx = {}
    for s in range(count):
        u = torch.cat([ub[node_off[s]:node_off[s + 1]], vb[node_off[s]:node_off[s + 1]]]).cpu().numpy()
        errs.append(float(np.linalg.norm(u - u64[s]) / np.linalg.norm(u64[s])))
        if s in cpu_picks:
            u_mx[s] = u
    launches_mx = sum(o[0].gpu_launches for o in outs_mx)

    # batched FP64
    per_b64, outs_b64, _ = timed(lambda: solve_batch(ctrl64), max(1, args.steps // 2), 1)

    # plain FP64: one mesh at a time on a size-stratified sample
    sample = _stratified(count, min(64, count), 0.5)
    singles = [(s, ua.CreateMUA(probs[s].coordinates, probs[s].connectivity, device=local)) for s in sample]

    def plain_pass():
        its = 0
        for s, m1 in singles:
            ub[node_off[s]:node_off[s + 1]] = 0; vb[node_off[s]:node_off[s + 1]] = 0
            _, info = ua.uv_resident(ctrl64, m1, bcss[s], F_devs[s], rhow=probs[s].rhow, g=probs[s].g)
            its += info.krylov_its_total
        return its

    per_plain, _, _ = timed(plain_pass, 1, 1)
    for _, m1 in singles:
        m1.close()

    # e2e: public API with host arrays in pinned memory
    pin = {k: torch.tensor(np.concatenate([getattr(P, k) for P in probs]), dtype=torch.float64).pin_memory()
           for k in NAMES}
    pin_u = torch.zeros(Nn_tot, dtype=torch.float64).pin_memory()
    # the solutions go to pinned output arrays; the start velocities (zeros) stay untouched
    pin_ou = torch.zeros(Nn_tot, dtype=torch.float64).pin_memory()
    pin_ov = torch.zeros(Nn_tot, dtype=torch.float64).pin_memory()
    Fh, outh = [], []
    for s, P in enumerate(probs):
        a, b = int(node_off[s]), int(node_off[s + 1])
        Fh.append(ua.Fields(**{k: pin[k].numpy()[a:b] for k in NAMES}, ub=pin_u.numpy()[a:b],
                            vb=pin_u.numpy()[a:b], rhow=P.rhow, g=P.g))
        outh.append((pin_ou.numpy()[a:b], pin_ov.numpy()[a:b]))
    per_e2e, _, _ = timed(lambda: ua.uv_batch(ctrlmx, mua, Fh, bcss, out=outh), args.steps, 1)
    ncon = sum(len(b.ubFixedNode) + len(b.vbFixedNode) for b in bcss)
    h2d = 8 * Nn_tot * (len(NAMES) + 2) + 12 * ncon
    d2h = 8 * 2 * Nn_tot

    # per-kernel device time (a profiled batched mixed solve: CUDA events on the library's stream)
    prof_info = solve_batch(ctrl_of(L.UA_PREC_MIXED, profile=1))[0]
    prof = prof_info.kernels

    # served form
    serving = None
    if not args.skip_serve:
        serving = _serve_leg(args, ua, L, synth, np, local)

    # P2 legs: the implicit uvh step and the mixed uv solve against the oracle
    p2 = None
    if not args.skip_p2 and rank == 0 and world == 1:
        p2 = _p2_legs(args, ua, L, synth, np)

    t_mx = max_over_ranks(sum(per_mx))
    t_b64 = max_over_ranks(sum(per_b64))
    t_plain = max_over_ranks(sum(per_plain))
    t_e2e = max_over_ranks(sum(per_e2e))
    value = replica_throughput(world, count * args.steps, t_mx)
    value_b64 = replica_throughput(world, count * len(per_b64), t_b64)
    value_plain = replica_throughput(world, len(sample), t_plain)
    e2e_value = replica_throughput(world, count * args.steps, t_e2e)

    # roofline of the dominant kernel class (by measured device time).  Algorithmic bytes of each
    # timed launch follow from the tangent non-zeros and dof rows of the systems it processed
    # (counted on the device per launch; converged systems drop out of the Krylov kernels);
    # FP32 values and vectors, 4-byte indices.
    nnz = sum(mua.nnz(s) for s in range(count))
    Ne = sum(P.Nele for P in probs)
    rows = 2 * Nn_tot
    peaks = {}
    try:
        peaks = json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))
    except Exception:
        pass
    hbm_peak = float(peaks.get("hbm_gbs", 6650.0))
    wn, wr = prof["work_nnz"], prof["work_rows"]
    ele_per_row = Ne / rows
    # per class: (ms, launches, algorithmic bytes summed over the launches, bytes per non-zero / row)
    cand = {
        "uv_p1_kernel<K,float> (tangent+residual assembly)":
            (prof["asmK_ms"], prof["asmK_n"], 4 * wn["asmK"] + (12 * ele_per_row + 48 + 8) * wr["asmK"],
             "4 B/nnz (K write) + per row: 12*Ne/rows connectivity + 48 nodal fields + 8 R"),
        "uv_p1_kernel<K off> (residual-only assembly)":
            (prof["asmR_ms"], prof["asmR_n"], (12 * ele_per_row + 48 + 8) * wr["asmR"],
             "per row: 12*Ne/rows connectivity + 48 nodal fields + 8 R"),
        # The finest-level passes of the resident PCG: times inside the kernel, one pass per system and
        # step, team barriers included, weighted with the team's share of the GPU.  Node-sliced tangent
        # copies: four values per column index, so 1 B of index per non-zero; the quads of the transfer
        # Q and padding slots are not counted.
        "k_pcg_team: p, q = A p and p.q (FP32 node slices)":
            (prof["spmv_ms"], prof["spmv_n"], 5 * wn["spmv"] + 20 * wr["spmv"],
             "5 B/nnz (FP32 value + 1/4 column) + per row: 4 z + 8 p + 8 q"),
        "k_pcg_team: x, r update and finest restriction":
            (prof["amgR_ms"], prof["amgR_n"], 36 * wr["amgR"],
             "per row: 16 x + 8 r + 4 p + 4 q + 4 D (the transfer's quads not counted)"),
        "k_pcg_team: finest up pass z = 2 r - A r + Q z_c and r.z (BF16 node slices)":
            (prof["amgP_ms"], prof["amgP_n"], 3 * wn["amgP"] + 8 * wr["amgP"],
             "3 B/nnz (BF16 value + 1/4 column) + per row: 4 r + 4 z (the transfer's quads not counted)"),
    }
    dom = max(cand, key=lambda c: cand[c][0])
    ms, n, alg_total, rule = cand[dom]
    avg_ms = ms / max(n, 1)
    achieved = alg_total / (ms / 1000) / 1e9 if ms > 0 else 0.0
    total_k = sum(v[0] for v in cand.values())
    # DRAM traffic per launch: ncu dram__bytes_read.sum + dram__bytes_write.sum (MB) of the first
    # launch of each class over its algorithmic bytes (MB), captured with
    # `bench.py --batch 32 --legs mixed --steps 1 --warmup 1` (every system active), scaled to this
    # launch size
    traffic_ratio = {"uv_p1_kernel<K,": (133.05 + 48.05) / 145.44, "uv_p1_kernel<K off": None,
                     "k_pcg_team": None}
    tr = next((v for k, v in traffic_ratio.items() if dom.startswith(k)), None)
    # The assembly is bound by latency and FP64 issue, not HBM: its FP64 roofline beside the HBM one.
    # Executed FP64 operations per P1 element of the tangent+residual pass (2 DFMA + DADD + DMUL,
    # ncu per-cycle instruction sums x cycles of the 32-mesh batch: 4.82e9 over 1,162,956 elements,
    # patch halos included) over the measured launch time; peak 148 SMs x 64 DFMA/clock x 2 x 1965
    # MHz = 37.2 TFLOP/s (nominal, no measured FP64 figure in MEASURED_PEAKS.json).
    fp64_peak = 148 * 64 * 2 * float(peaks.get("sm_max_mhz", 1965.0)) * 1e6 / 1e12
    fp64 = {}
    for key, fpe in (("uv_p1_kernel<K,float> (tangent+residual assembly)", 4146.0),):
        cms, cn, _, _ = cand[key]
        cls_rows = wr["asmK"]
        if cms > 0:
            tf = fpe * ele_per_row * cls_rows / (cms / 1000) / 1e12
            fp64[key] = {"achieved": tf, "peak": fp64_peak, "unit": "TFLOP/s", "frac": tf / fp64_peak,
                         "flops_per_element": fpe}
    roof = {"bound": "hbm", "kernel": dom, "achieved": achieved, "peak": hbm_peak, "unit": "GB/s",
            "frac": achieved / hbm_peak,
            "traffic": (tr * alg_total / max(n, 1)) if tr else None,
            "traffic_source": ("ncu dram__bytes_read.sum + dram__bytes_write.sum on the 32-mesh batch, scaled by "
                               "algorithmic bytes to this launch size") if tr else None,
            "alg_bytes_per_launch": alg_total / max(n, 1), "alg_bytes_rule": rule,
            "avg_launch_ms": avg_ms, "launches": n,
            "peak_source": ("MEASURED_PEAKS.json hbm_gbs (burst copy), of measured" if "hbm_gbs" in peaks
                            else "fallback 6650 GB/s, of fallback"),
            "kernel_share_of_timed_classes": {c: v[0] / max(total_k, 1e-12) for c, v in cand.items()},
            "fp64_assembly": fp64, "fp64_peak_source": "148 SMs x 64 DFMA/clock x 2 flops x max SM clock, of nominal",
            "classes_gbs": {c: (v[2] / (v[0] / 1000) / 1e9 if v[0] > 0 else None) for c, v in cand.items()},
            # the same per class as a fraction of the measured HBM copy bandwidth
            "classes_frac": {c: (v[2] / (v[0] / 1000) / 1e9 / hbm_peak if v[0] > 0 else None)
                             for c, v in cand.items()},
            # device time of the timed classes over the profiled solve's whole device time (the rest:
            # coarse AMG levels, AMG set-up, waiting teams)
            "timed_classes_share_of_device_time": total_k / max(float(prof_info.device_ms), 1e-12),
            # the profiled solve's device time by phase (event ranges on the library's stream):
            # tangent and residual assemblies, AMG numeric set-ups with the node-slice fills, the
            # Krylov iterations (the resident solves with their first residuals)
            "device_split": _device_split(prof, float(prof_info.device_ms))}

    cpu, vs_oracle = None, None
    if rank == 0 and world == 1 and not args.skip_cpu:
        cpu, u_ref = _cpu_baseline_pool(count, CPU_SAMPLE)
        # the batched GPU solutions of the sampled meshes against the FP64 oracle's
        rel = lambda a, b: float(np.linalg.norm(a - b) / np.linalg.norm(b))
        e64 = [rel(u64[k], u_ref[k]) for k in sorted(u_ref)]
        emx = [rel(u_mx[k], u_ref[k]) for k in sorted(u_ref)]
        nes = [probs[k].Nele for k in sorted(u_ref)]
        vs_oracle = {"meshes": len(e64), "elements": f"{min(nes)}-{max(nes)}",
                     "fp64_batched_max": max(e64), "mixed_batched_max": max(emx),
                     "mixed_batched_median": statistics.median(emx),
                     "tolerance": {"fp64": 1e-10, "mixed": 1e-8}}

    if rank == 0:
        lat = sorted(per_mx)
        its = [i.iterations for i in infos_mx]
        kits = [i.krylov_its_total for i in infos_mx]
        line = {
            "metric": METRIC, "value": value, "unit": "solves/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": t_mx / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32/f64 mixed", "data": "synthetic",
            "config": {"workload": _workload(count), "systems_per_step": count, "elements": int(Ne),
                       "nodes": Nn_tot, "nnz": int(nnz),
                       "l2": "inputs 0.5 GB > L2; 512 MB buffer written between timed steps",
                       "parallelism": f"replicas x{world}" + (", each rank its own seeded batch of this size "
                                                              "distribution" if world > 1 else ""),
                       "precision": "mixed",
                       "krylov": "PCG, aggregation AMG V(1,1), adaptive forcing, one resident kernel a solve",
                       "newton_iterations_mean": float(np.mean(its)), "newton_iterations_max": int(max(its)),
                       "pcg_iterations_mean": float(np.mean(kits)), "converged": int(sum(i.converged for i in infos_mx))},
            "batch_latency_ms": {"p50": statistics.median(lat), "p99": lat[min(len(lat) - 1, int(0.99 * len(lat)))]},
            "serving": serving,
            "roofline": roof,
            "cpu_baseline": cpu,
            "clocks": clocks,
            "gpu_launches": int(launches_mx),
            "e2e": {"value": e2e_value, "unit": "solves/s", "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h},
            "cauchy_fallbacks": int(sum(i.cauchy_fallbacks for i in infos_mx) + sum(i.cauchy_fallbacks for i in infos64)),
            "rel_err_vs_fp64": {"max": max(errs), "median": statistics.median(errs)},
            "rel_err_vs_oracle": vs_oracle,
            "plain_fp64": {"value": value_plain, "unit": "solves/s", "form": "one mesh at a time, all FP64",
                           "sample": f"{len(sample)} meshes, one per size stratum of the batch",
                           "ms_per_pass": t_plain},
            "batched_fp64": {"value": value_b64, "unit": "solves/s", "ms_per_step": t_b64 / len(per_b64),
                             "converged": int(sum(i.converged for i in infos64))},
            "mixed_batched_over_plain_fp64": value / value_plain,
            "p2": p2,
            "autotune": None if tune is None else {
                "chosen": tune["chosen"], "default_ms": tune["default_ms"], "tuned_ms": tune["chosen"]["ms"],
                "gain": tune["gain"], "candidates": len(tune["candidates"]),
                "rule": "tangent+residual assembly of the whole batch at u=v=0, mean of 3 launches per schedule; "
                        "patches of clamp(nn/div, 16, cap) nodes x P1 (CTA threads, registers) of (256, 128), "
                        "(128, 128), (128, 96), (256, 80), (128, 80)"},
        }
        print(json.dumps(line), flush=True)
    mua.close()
    if world > 1:
        dist.destroy_process_group()
    return 0


def _serve_leg(args, ua, L, synth, np, device):
    """Served form: Poisson arrivals over resident templates; p50/p99 and solves/s,
    with a sample of results checked against plain FP64 solves."""
    from uasource_b200.serve import Request, SsaServer, perturbed_C, poisson_arrivals
    tpl = synth.serve_templates(args.serve_templates)
    ctrl = ua.CtrlVar(precision=L.UA_PREC_MIXED, krylov_rtol=1e-6).set_force_tolerance(1e-20)
    ctrl64 = ua.CtrlVar().set_force_tolerance(1e-20)
    # warm starts: each template's own solution
    base = ua.CreateMUABatch([(P.coordinates, P.connectivity) for P in tpl], device=device)
    warm = ua.uv_batch(ctrl, base, [ua.Fields.from_problem(P) for P in tpl], [ua.BCs.from_problem(P) for P in tpl])
    base.close()
    srv = SsaServer(tpl, ctrl, device=device)
    rng = np.random.default_rng(2024)

    def requests(n, t0):
        arr = poisson_arrivals(n, args.serve_rate, rng)
        out = []
        for i in range(n):
            k = int(rng.integers(len(tpl)))
            out.append(Request(rid=i, template=k, C=perturbed_C(tpl[k], rng), ub0=warm[k][0], vb0=warm[k][1],
                               arrival=t0 + arr[i]))
        return out

    srv.run(requests(min(8, args.serve_requests), 0.0), realtime=False)  # warm-up (graphs, hierarchies)
    reqs = requests(args.serve_requests, 0.0)
    st = srv.run(reqs, realtime=True)
    srv.close()
    # accuracy: a sample of requests against the plain FP64 form
    errs = []
    for r in reqs[:: max(1, len(reqs) // 6)]:
        P = tpl[r.template]
        m1 = ua.CreateMUA(P.coordinates, P.connectivity, device=device)
        F = ua.Fields.from_problem(P)
        F.C = r.C
        F.ub = r.ub0.copy(); F.vb = r.vb0.copy()
        Fo, _, _, _, _ = ua.uv(ctrl64, m1, ua.BCs.from_problem(P), F)
        m1.close()
        u64 = np.concatenate([Fo.ub, Fo.vb]); u = np.concatenate([r.ub, r.vb])
        errs.append(float(np.linalg.norm(u - u64) / np.linalg.norm(u64)))
    sizes = [P.Nele for P in tpl]
    return {"workload": f"{len(tpl)} resident templates of {min(sizes)}-{max(sizes)} P1 elements, Poisson arrivals "
                        f"{args.serve_rate:g} req/s, {len(reqs)} requests, lognormal C (sigma 0.3), warm starts",
            "solves_per_s": st.solves_per_s, "p50_ms": st.p50_ms, "p99_ms": st.p99_ms,
            "mean_queue_ms": st.mean_queue_ms, "slots": st.slots, "max_active": st.max_active,
            "makespan_s": st.makespan_s, "converged": int(sum(bool(r.info.converged) for r in reqs)),
            "rel_err_vs_fp64_max": max(errs) if errs else None, "checked": len(errs)}


def _oracle_p2(nx, ny):
    """Oracle uv solve of the nx x ny-vertex P2 ice stream/shelf mesh (seed 0; child process):
    (seconds, converged, solution [ub; vb])."""
    sys.path.insert(0, ROOT)
    import numpy as np
    from oracle import ua_ref as R
    from uasource_b200 import synth
    R.use_compiled_element_loop(True, 1)
    P = synth.ice_stream_shelf(nx, ny, nod=6, seed=0)
    p = R.Params()
    p.set_force_tolerance(1e-20)
    F = R.Fields(h=P.h, S=P.S, B=P.B, rho=P.rho, AGlen=P.AGlen, n=P.n, C=P.C, m=P.m, ub=P.ub, vb=P.vb)
    bcs = R.BCs(ubFixedNode=P.ubFixedNode, ubFixedValue=P.ubFixedValue, vbFixedNode=P.vbFixedNode,
                vbFixedValue=P.vbFixedValue)
    t = time.perf_counter()
    res = R.uv(p, R.create_mua(P.coordinates, P.connectivity), bcs, F)
    return time.perf_counter() - t, bool(res.converged), np.concatenate([res.ub, res.vb])


P2_UV = (101, 51)     # 10,000 P2 elements: the largest P2 uv mesh of the oracle leg
P2_UVH = (201, 101)   # 40,000 P2 elements: the implicit-step leg


def _p2_legs(args, ua, L, synth, np):
    """P2 forms of the path beside the batched headline: the FP64 implicit uvh step (dt = 0.1 a,
    from the converged diagnostic state) on a 40k-element P2 mesh, and the uv solve on a
    10k-element P2 mesh in mixed and plain FP64, each against the FP64 oracle's solution."""
    with _pool(1) as pool:
        job = pool.apply_async(_oracle_p2, P2_UV)
        out = {}
        # uv, mixed vs FP64, against the oracle
        P = synth.ice_stream_shelf(*P2_UV, nod=6, seed=0)
        mua = ua.CreateMUA(P.coordinates, P.connectivity)
        bcs = ua.BCs.from_problem(P)
        sol = {}
        for name, prec, rtol in (("fp64", L.UA_PREC_FP64, 1e-12), ("mixed", L.UA_PREC_MIXED, 1e-6)):
            ctrl = ua.CtrlVar(precision=prec, krylov_rtol=rtol).set_force_tolerance(1e-20)
            per, res = _timed_calls(lambda: ua.uv(ctrl, mua, bcs, ua.Fields.from_problem(P)), 2, 1)
            Fo, _, _, _, info = res
            sol[name] = (np.concatenate([Fo.ub, Fo.vb]), info, 1000 * len(per) / sum(per))
        mua.close()
        # uvh step
        Pt = synth.ice_stream_shelf(*P2_UVH, nod=6, seed=0, transient=True)
        bt = ua.BCs.from_problem(Pt)
        m2 = ua.CreateMUA(Pt.coordinates, Pt.connectivity)
        Fd, _, _, _, _ = ua.uv(ua.CtrlVar(precision=L.UA_PREC_MIXED, krylov_rtol=1e-6).set_force_tolerance(1e-20),
                               m2, bt, ua.Fields.from_problem(Pt))
        m2.close()
        m3 = ua.CreateMUA(Pt.coordinates, Pt.connectivity, ndof=3)
        F0 = ua.Fields.from_problem(Pt)
        F0.ub, F0.vb = Fd.ub, Fd.vb
        hb = ua.HBCs(ubFixedNode=bt.ubFixedNode, ubFixedValue=bt.ubFixedValue, vbFixedNode=bt.vbFixedNode,
                     vbFixedValue=bt.vbFixedValue)
        ctrl = ua.CtrlVar().set_force_tolerance(1e-20)
        per, res = _timed_calls(lambda: ua.uvh(ctrl, m3, F0, F0.copy(), hb, 0.1), 2, 1)
        info = res[2]
        m3.close()
        out["uvh_step"] = {"mesh": f"P2 {P2_UVH[0]}x{P2_UVH[1]} vertices, {Pt.Nele} elements, {Pt.Nnodes} nodes",
                           "form": "plain FP64, GMRES with the block preconditioner", "dt_a": 0.1,
                           "steps_per_s": 1000 * len(per) / sum(per), "ms_per_step": sum(per) / len(per),
                           "newton_iterations": info.iterations, "krylov_iterations": info.krylov_its_total,
                           "converged": bool(info.converged)}
        t_or, conv, u_ref = job.get()
    rel = lambda a: float(np.linalg.norm(a - u_ref) / np.linalg.norm(u_ref))
    out["uv_vs_oracle"] = {"mesh": f"P2 {P2_UV[0]}x{P2_UV[1]} vertices, {P.Nele} elements, {P.Nnodes} nodes",
                           "oracle_converged": conv, "oracle_s": t_or,
                           "fp64": {"solves_per_s": sol["fp64"][2], "rel_err": rel(sol["fp64"][0]),
                                    "newton_iterations": sol["fp64"][1].iterations},
                           "mixed": {"solves_per_s": sol["mixed"][2], "rel_err": rel(sol["mixed"][0]),
                                     "newton_iterations": sol["mixed"][1].iterations},
                           "tolerance": {"fp64": 1e-10, "mixed": 1e-8}}
    return out


def _big_p2_problem(transient):
    """The 400 km x 200 km P2 mesh of ~1M elements (1001x501 vertices before mid-nodes)."""
    from uasource_b200 import synth
    return synth.ice_stream_shelf(1001, 501, Lx=400e3, Ly=200e3, nod=6, seed=0, transient=transient)


def _timed_calls(fn, steps, warmup):
    import torch
    for _ in range(warmup):
        fn()
    torch.cuda.synchronize()
    e0 = torch.cuda.Event(enable_timing=True); e1 = torch.cuda.Event(enable_timing=True)
    per, out = [], None
    for _ in range(steps):
        torch.cuda.synchronize()
        e0.record()
        out = fn()
        e1.record()
        torch.cuda.synchronize()
        per.append(e0.elapsed_time(e1))
    return per, out


def _device_split(prof, device_ms):
    asm = prof["asmK_ms"] + prof["asmR_ms"]
    parts = {"assembly": asm, "amg_setup": prof.get("setup_ms", 0.0), "krylov": prof.get("krylov_ms", 0.0)}
    parts["other"] = max(device_ms - sum(parts.values()), 0.0)
    return {k: {"ms": v, "share": v / max(device_ms, 1e-12)} for k, v in parts.items()}


def run_uv1m(args):
    """Precision form on the 1M-element P2 mesh: one uv solve, mixed vs plain FP64."""
    import numpy as np
    import uasource_b200 as ua
    from uasource_b200 import lib as L
    P = _big_p2_problem(False)
    mua = ua.CreateMUA(P.coordinates, P.connectivity)
    bcs = ua.BCs.from_problem(P)
    res = {}
    for name, prec, rtol in (("fp64", L.UA_PREC_FP64, 1e-12), ("mixed", L.UA_PREC_MIXED, 1e-6)):
        ctrl = ua.CtrlVar(precision=prec, krylov_rtol=rtol).set_force_tolerance(1e-20)
        per, out = _timed_calls(lambda: ua.uv(ctrl, mua, bcs, ua.Fields.from_problem(P)), args.steps,
                                max(1, min(args.warmup, 1)))
        Fo, _, _, _, info = out
        # one more solve with per-class launch timing (not part of the timed steps)
        prof = ua.uv(ua.CtrlVar(precision=prec, krylov_rtol=rtol, profile=1).set_force_tolerance(1e-20), mua, bcs,
                     ua.Fields.from_problem(P))[4]
        res[name] = (per, np.concatenate([Fo.ub, Fo.vb]), info, {"kernels": prof.kernels, "device_ms": prof.device_ms})
    u64 = res["fp64"][1]
    err = float(np.linalg.norm(res["mixed"][1] - u64) / np.linalg.norm(u64))
    v_mx = 1000 * len(res["mixed"][0]) / sum(res["mixed"][0])
    v_64 = 1000 * len(res["fp64"][0]) / sum(res["fp64"][0])
    line = {"metric": "uv Newton solves/s, 1M-element P2 mesh (mixed vs plain FP64)", "value": v_mx,
            "unit": "solves/s", "n_gpus": 1, "steps": args.steps, "warmup": 1,
            "ms_per_step": sum(res["mixed"][0]) / len(res["mixed"][0]), "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32/f64 mixed", "data": "synthetic",
            "config": {"workload": f"uv solve from u=v=0, ice stream/shelf 400x200 km, P2, {P.Nele} elements, "
                                   f"{P.Nnodes} nodes, seed 0, rForce<1e-20"},
            "plain_fp64": {"value": v_64, "unit": "solves/s",
                           "newton_iterations": res["fp64"][2].iterations,
                           "pcg_iterations": res["fp64"][2].krylov_its_total, "profiled": res["fp64"][3]},
            "mixed": {"newton_iterations": res["mixed"][2].iterations,
                      "pcg_iterations": res["mixed"][2].krylov_its_total, "profiled": res["mixed"][3]},
            "rel_err_mixed_vs_fp64": err, "mixed_over_plain": v_mx / v_64}
    print(json.dumps(line), flush=True)
    mua.close()
    return 0


def run_uvh1m(args):
    """Plain FP64 implicit uvh step (dt = 0.1 a) on the 1M-element P2 mesh."""
    import numpy as np
    import uasource_b200 as ua
    from uasource_b200 import lib as L
    P = _big_p2_problem(True)
    bcs = ua.BCs.from_problem(P)
    m2 = ua.CreateMUA(P.coordinates, P.connectivity)
    F = ua.Fields.from_problem(P)
    Fo, _, _, _, info_uv = ua.uv(ua.CtrlVar(precision=L.UA_PREC_MIXED, krylov_rtol=1e-6).set_force_tolerance(1e-20),
                                 m2, bcs, F)
    m2.close()
    m3 = ua.CreateMUA(P.coordinates, P.connectivity, ndof=3)
    F0 = ua.Fields.from_problem(P)
    F0.ub, F0.vb = Fo.ub, Fo.vb
    F1 = F0.copy()
    ctrl = ua.CtrlVar().set_force_tolerance(1e-20)
    hb = ua.HBCs(ubFixedNode=bcs.ubFixedNode, ubFixedValue=bcs.ubFixedValue, vbFixedNode=bcs.vbFixedNode,
                 vbFixedValue=bcs.vbFixedValue)
    per, out = _timed_calls(lambda: ua.uvh(ctrl, m3, F0, F1, hb, 0.1), args.steps, 1)
    F1o, _, info = out
    prof = ua.uvh(ua.CtrlVar(profile=1).set_force_tolerance(1e-20), m3, F0, F1, hb, 0.1)[2]
    line = {"metric": "uvh implicit steps/s, 1M-element P2 mesh (plain FP64)", "value": 1000 * len(per) / sum(per),
            "unit": "steps/s", "n_gpus": 1, "steps": args.steps, "warmup": 1, "ms_per_step": sum(per) / len(per),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": f"implicit uvh step dt=0.1 a (SSTREAM_TransientImplicit, SUPG), ice stream/shelf "
                                   f"400x200 km, P2, {P.Nele} elements, {P.Nnodes} nodes, a=0.3+0.1N(0,1), "
                                   f"start: converged diagnostic state"},
            "newton_iterations": info.iterations, "krylov_iterations": info.krylov_its_total,
            "converged": bool(info.converged), "rForce": info.rForce,
            "kernels": prof.kernels, "device_ms": prof.device_ms,
            "dh_max_m": float(np.max(np.abs(F1o.h - P.h)))}
    print(json.dumps(line), flush=True)
    m3.close()
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--skip-cpu", action="store_true")
    ap.add_argument("--skip-serve", action="store_true")
    ap.add_argument("--skip-p2", action="store_true")
    ap.add_argument("--serve-requests", type=int, default=200)
    ap.add_argument("--serve-rate", type=float, default=200.0)
    ap.add_argument("--serve-templates", type=int, default=16)
    # profiling-only options (ncu captures on bounded cases); the bench line uses the defaults
    ap.add_argument("--legs", default="all", choices=["all", "mixed"])
    ap.add_argument("--no-autotune", action="store_true", help="keep the default assembly schedule")
    ap.add_argument("--batch", type=int, default=BATCH, help="meshes per step (default 256)")
    # the 1M-element P2 workloads (their own JSON line; the headline line is the batched one)
    ap.add_argument("--workload", default="batch", choices=["batch", "uv1m", "uvh1m", "p2"])
    args = ap.parse_args()
    if args.impl == "reference":
        return run_reference(args)
    if args.workload == "uv1m":
        return run_uv1m(args)
    if args.workload == "uvh1m":
        return run_uvh1m(args)
    if args.workload == "p2":  # the P2 legs alone (their own line; bounded cases for profiling)
        import numpy as np
        import uasource_b200 as ua
        from uasource_b200 import lib as L
        from uasource_b200 import synth
        print(json.dumps({"workload": "p2", "p2": _p2_legs(args, ua, L, synth, np)}), flush=True)
        return 0
    return run_ours(args)


if __name__ == "__main__":
    sys.exit(main())
