"""Benchmark of the B200 k-means (Lloyd) hot path through the AOCL-DA C ABI.

Workload (the configuration the headline metric is quoted on): fp32 k-means,
X = 1,000,000 x 64 drawn from a 256-component Gaussian mixture (means
U[-10,10]^64, per-component sigma U[0.5,2], mixing weights Dirichlet(1)),
n_clusters = 256, k-means++ initial centres from seed 1, max_iter = 50,
tol = 1e-4.  Seeded synthetic data stands in for the data set.

A step is one da_kmeans_compute_s call from the fixed k-means++ centres
(supplied init, n_init = 1), i.e. rinfo[3] Lloyd iterations over the whole
matrix; the metric is Lloyd iterations per second.  `value` keeps X resident
in HBM (set once); `e2e` re-uploads X from pinned host memory and reads the
labels and centres back inside every step.

With --gpus N > 1 (one rank per GPU under torch.distributed.run) the data
set is split across the ranks: every rank holds a copy of the 1,000,000 x
64 set as its shard (weak scaling: the job clusters N x 1,000,000 rows), the
ranks exchange their integer centroid sums in one NCCL all-reduce per Lloyd
iteration, and `value` is N x the fit's Lloyd iterations per second.
--sharded runs that path on one GPU too.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference]
"""
import argparse
import ctypes as C
import importlib.util
import json
import os
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(ROOT, "aocl-data-analytics_b200")
ORACLE = os.path.join(ROOT, "oracle")

N, D, K = 1_000_000, 64, 256
MAX_ITER, TOL, SEED = 50, 1e-4, 1
METRIC = "k-means Lloyd iterations/s (fp32, 1M x 64, k=256)"
UNIT = "iters/s"


def set_rows(rows):
    global N
    N = rows


def _load(name, path):
    spec = importlib.util.spec_from_file_location(name, path)
    mod = importlib.util.module_from_spec(spec)
    sys.modules[name] = mod
    spec.loader.exec_module(mod)
    return mod


def make_data(n=None, d=D, k=K, seed=SEED):
    n = N if n is None else n
    rng = np.random.default_rng(seed)
    means = rng.uniform(-10.0, 10.0, (k, d))
    sig = rng.uniform(0.5, 2.0, k)
    w = rng.dirichlet(np.ones(k))
    lab = rng.choice(k, n, p=w)
    X = means[lab] + rng.standard_normal((n, d)) * sig[lab, None]
    return np.ascontiguousarray(X, dtype=np.float32)


def load_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return p["hbm_gbs"], p["bf16_tflops"], "measured"
    except Exception:
        return 6650.0, 1590.0, "fallback"


REASONS = {0x1: "gpu_idle", 0x2: "applications_clocks_setting", 0x4: "sw_power_cap",
           0x8: "hw_slowdown", 0x10: "sync_boost", 0x20: "sw_thermal_slowdown",
           0x40: "hw_thermal_slowdown", 0x80: "hw_power_brake_slowdown",
           0x100: "display_clock_setting"}


class Clocks:
    """nvidia-smi sampling during the timed region."""

    def __init__(self, gpu):
        self.gpu = gpu
        self.proc = None
        self.path = tempfile.mktemp(suffix=".csv")

    def start(self):
        try:
            self.f = open(self.path, "w")
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu),
                 "--query-gpu=clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active",
                 "--format=csv,noheader,nounits", "-lms", "100"],
                stdout=self.f, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if not self.proc:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        self.f.close()
        sm, mx, reasons = [], 0.0, set()
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 4:
                continue
            try:
                s, m = float(parts[0]), float(parts[1])
                r = int(parts[3], 16) if parts[3].startswith("0x") else int(parts[3])
            except ValueError:
                continue
            sm.append(s)
            mx = max(mx, m)
            for bit, name in REASONS.items():
                if r & bit and bit != 0x1:
                    reasons.add(name)
        if not sm:
            return None
        return {"sm_mhz": float(np.median(sm)), "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm)}


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def _oracle():
    return _load("oracle_mod", os.path.join(ORACLE, "oracle.py"))


def cpu_baseline(X, C0, iters=3):
    """The reference's CPU Lloyd iteration (kmeans_lloyd.hpp:106-405: blocks
    of 512 rows over OpenMP threads, one BLAS sgemm per block, strict-'<'
    argmin, thread-local sums merged under a lock) restated in the oracle
    (oracle_blas.c) with scipy's OpenBLAS, on ALL rows of the workload from
    the same initial centres, every host thread.  Returns iterations/s."""
    orc = _oracle()
    blas = orc.openblas()
    Cc = np.ascontiguousarray(C0.copy())
    lab = np.full(X.shape[0], -1, dtype=np.int32)
    orc.lloyd_blas(X, Cc, lab, 1, blas)  # warm-up (first touch, thread pools)
    t0 = time.perf_counter()
    orc.lloyd_blas(X, Cc, lab, iters, blas)
    t = time.perf_counter() - t0
    cores = orc.num_threads()
    return {"value": iters / t, "unit": UNIT, "cores": cores, "kind": "port",
            "sample": f"{iters} Lloyd iterations over all {X.shape[0]} rows (k={C0.shape[0]}, "
                      f"d={X.shape[1]}) from the workload's k-means++ centres: the reference's "
                      f"blocked form (512-row blocks, one OpenBLAS sgemm each, {cores} OpenMP "
                      f"threads; {blas.config()})"}


def run_reference(args):
    """The reference arm: the reference's CPU k-means (the oracle's
    restatement, oracle_kpp.cpp + oracle_blas.c, with OpenBLAS) on the same
    workload -- k-means++ from seed 1 (timed once, reported as init_s), then
    Lloyd iterations from those centres, `ITERS_PER_REF_STEP` per step."""
    rank, world, _ = dist_env()
    if rank != 0:
        return 0
    orc = _oracle()
    blas = orc.openblas()
    X = make_data()
    t0 = time.perf_counter()
    chosen = orc.kmeanspp(X, K, SEED, gemm=blas)  # distances by BLAS, as the reference
    init_s = time.perf_counter() - t0
    C0 = np.ascontiguousarray(X[chosen])
    Cc = C0.copy()
    lab = np.full(N, -1, dtype=np.int32)
    per_step = 2
    for _ in range(max(1, args.warmup)):
        orc.lloyd_blas(X, Cc, lab, per_step, blas)
    t0 = time.perf_counter()
    for _ in range(args.steps):
        orc.lloyd_blas(X, Cc, lab, per_step, blas)
    t = time.perf_counter() - t0
    v = args.steps * per_step / t
    cores = orc.num_threads()
    cb = {"value": v, "unit": UNIT, "cores": cores, "kind": "port",
          "sample": f"{args.steps} steps of {per_step} Lloyd iterations over all {N} rows "
                    f"(k={K}, d={D}) continuing from k-means++ (seed {SEED}); the reference's "
                    f"blocked form (512-row blocks, one OpenBLAS sgemm each, {cores} OpenMP "
                    f"threads; {blas.config()})"}
    cfg = config_dict(args) | {"init": f"k-means++ seed {SEED} (oracle restatement, "
                                       f"{init_s:.1f} s on the host, not timed)",
                               "init_s": init_s, "iterations_per_step": per_step,
                               "step": f"{per_step} Lloyd iterations (blocked BLAS form) "
                                       "continuing the fit"}
    out = {"impl": "reference", "metric": METRIC, "value": v, "unit": UNIT, "n_gpus": args.gpus,
           "steps": args.steps, "warmup": args.warmup, "ms_per_step": t / args.steps * 1e3,
           "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
           "data": "synthetic", "config": cfg, "cpu_baseline": cb,
           "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(out))
    return 0


def config_dict(args):
    return {"workload": f"kmeans_lloyd_fp32_{N}x64_k256", "n_samples": N, "n_features": D,
            "n_clusters": K, "init": "k-means++ seed 1 (computed once, supplied to every step)",
            "max_iter": MAX_ITER, "tol": TOL,
            "step": "one da_kmeans_compute_s = rinfo[3] Lloyd iterations",
            "l2": "inputs (256 MB) larger than the 126 MB L2",
            "parallelism": f"replicas x{args.gpus}"}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=100)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="b200")
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline leg")
    ap.add_argument("--no-e2e", action="store_true", help="skip the end-to-end leg")
    ap.add_argument("--no-plain", action="store_true", help="skip the plain fp32 comparison")
    ap.add_argument("--no-knn", action="store_true", help="skip the kNN (4.04M x 128) leg")
    ap.add_argument("--no-c1", action="store_true", help="skip the fp64 kNN (10,000 x 32) leg")
    ap.add_argument("--no-accuracy", action="store_true",
                    help="skip the error checks against the fp64 oracle")
    ap.add_argument("--no-batched", action="store_true",
                    help="skip the batched k-means (512 data sets) leg")
    ap.add_argument("--no-radius", action="store_true",
                    help="skip the radius-neighbours leg")
    ap.add_argument("--no-ivf", action="store_true",
                    help="skip the IVF-flat approximate-neighbours leg")
    ap.add_argument("--no-serve", action="store_true",
                    help="skip the serving leg (8M x 96 index, 64 k-means models)")
    ap.add_argument("--serve-only", action="store_true",
                    help="run only the serving leg and print its JSON")
    ap.add_argument("--knn-only", action="store_true",
                    help="run only the kNN leg (profiling captures) and print its JSON")
    ap.add_argument("--kpp-only", action="store_true",
                    help="run only the k-means++ initialisation of the k-means data (profiling "
                         "captures) and print its times")
    ap.add_argument("--batched-only", action="store_true",
                    help="run only one batched k-means call over the 512 data sets (profiling "
                         "captures) and print its times")
    ap.add_argument("--knn-rows", type=int, default=4_000_000)
    ap.add_argument("--knn-queries", type=int, default=10_000)
    ap.add_argument("--knn-plain", type=int, default=1,
                    help="with --knn-only: also run the plain path (1) or not (0)")
    ap.add_argument("--sharded", action="store_true",
                    help="run the split-data path (every rank's shard, one NCCL all-reduce per "
                         "Lloyd iteration) also on one GPU; it is the path for --gpus > 1")
    ap.add_argument("--rows", type=int, default=N,
                    help="rows of X (default 1,000,000; smaller only for profiling captures)")
    args = ap.parse_args()
    set_rows(args.rows)
    if args.impl == "reference":
        return run_reference(args)

    import torch
    rank, world, local = dist_env()
    torch.cuda.set_device(local)
    if world > 1 or args.sharded:
        import torch.distributed as dist
        from datetime import timedelta
        kw = {}
        if world == 1:
            import socket
            with socket.socket() as sk:
                sk.bind(("127.0.0.1", 0))
                kw = {"init_method": f"tcp://127.0.0.1:{sk.getsockname()[1]}", "rank": 0,
                      "world_size": 1}
        dist.init_process_group("nccl", timeout=timedelta(seconds=300),
                                device_id=torch.device("cuda", local), **kw)
    ab = _load("aoclda_b200", os.path.join(PKG, "aoclda_b200.py"))
    if world > 1 or args.sharded:
        try:
            return run_sharded(ab, args, rank, world, local)
        finally:
            torch.distributed.destroy_process_group()
    if args.serve_only:
        if rank == 0:
            print(json.dumps(run_serving(ab)))
        return 0
    if args.knn_only:
        if rank == 0:
            print(json.dumps(run_knn(ab, nx=args.knn_rows, nq=args.knn_queries,
                                     plain=bool(args.knn_plain),
                                     accuracy=not args.no_accuracy)))
        return 0
    if args.kpp_only:
        if rank == 0:
            km = ab.KMeans(K, "s", order=ab.ROW_MAJOR, n_init=1, seed=SEED)
            km.set_data(make_data())
            ms = []
            for _ in range(max(1, args.steps)):
                t0 = time.perf_counter()
                km.init_centres(K)
                ms.append((time.perf_counter() - t0) * 1e3)
            km.close()
            print(json.dumps({"workload": "kmeans_pp_fp32_1000000x64_k256_seed1",
                              "init_ms": ms}))
        return 0
    if args.batched_only:
        if rank == 0:
            Xs, C0s = batched_workload()
            ab.kmeans_batched(Xs, C0s, max_iter=30, tol=1e-4)
            up, fit, down = ab.kmeans_batched_timing()
            print(json.dumps({"workload": "kmeans_batched_fp32_512_instances",
                              "device_ms": {"upload": up, "fit": fit, "download": down}}))
        return 0

    X = make_data()
    # the library's calls and the timing events share one (non-default) stream
    stream = torch.cuda.Stream()

    def handle(mode):
        km = ab.KMeans(K, "s", order=ab.ROW_MAJOR, max_iter=MAX_ITER, n_init=1, seed=SEED)
        km.L.da_b200_set_stream(km.h, C.c_void_p(stream.cuda_stream))
        km.set("convergence tolerance", TOL)
        km.set("precision mode", mode)
        km.set_data(X)
        return km

    mode = os.environ.get("BENCH_MODE", "bf16x3")
    km = handle(mode)
    t0 = time.perf_counter()
    C0 = km.init_centres(K)
    init_first_ms = (time.perf_counter() - t0) * 1e3  # with the upload of X
    t0 = time.perf_counter()
    C0b = km.init_centres(K)
    init_ms = (time.perf_counter() - t0) * 1e3        # X resident
    assert np.array_equal(C0, C0b)

    def prepare(h):
        h.set("initialization method", "supplied")
        h.call("da_kmeans_set_init_centres_s", ab.ptr(C0), D)

    def step(h):
        h.call("da_kmeans_compute_s", ok=(0, 21))
        return int(h.rinfo()[3])

    def timed(h, steps, warmup, sample_clocks=False):
        for _ in range(warmup):
            step(h)
        if world > 1:
            torch.distributed.barrier()
        torch.cuda.synchronize()
        clk = Clocks(local) if sample_clocks else None
        if clk:
            clk.start()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        iters = 0
        for _ in range(steps):
            iters += step(h)
        e1.record(stream)
        torch.cuda.synchronize()
        clocks = clk.stop() if clk else None
        ms = e0.elapsed_time(e1)
        if world > 1:
            t = torch.tensor([ms], device="cuda")
            torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
            ms = float(t.item())
            it = torch.tensor([iters], device="cuda", dtype=torch.float64)
            torch.distributed.all_reduce(it)
            iters_total = float(it.item())
        else:
            iters_total = iters
        return ms, iters, iters_total, clocks

    def kernel_times(h):
        # separate pass: event timing serialises the launches
        h.L.da_b200_set_kernel_timing(h.h, 1)
        h.L.da_b200_reset_kernel_time(h.h)
        step(h)
        h.L.da_b200_set_kernel_timing(h.h, 0)
        return {n: h.kernel_time(n) for n in
                ("kmeans_assign", "kmeans_rescore", "kmeans_sort", "kmeans_update")}

    prepare(km)
    ms, iters, iters_total, clocks = timed(km, args.steps, args.warmup, sample_clocks=True)
    value = iters_total / (ms / 1e3)
    n_iter = iters // args.steps
    relabelled = km.stat("relabelled_rows")
    full_scan = km.stat("full_scan_rows")
    graph_loop = km.stat("graph_loop")
    tensor_core = km.stat("tensor_core") == 1.0
    kt = kernel_times(km)

    plain = None
    if not args.no_plain:
        kp = handle("plain")
        prepare(kp)
        psteps = max(2, args.steps // 10)
        pms, piters, piters_total, _ = timed(kp, psteps, 1)
        pkt = kernel_times(kp)
        pa = pkt["kmeans_assign"]
        plain = {"value": piters_total / (pms / 1e3), "unit": UNIT, "steps": psteps,
                 "ms_per_step": pms / psteps,
                 "kernel_ms": {k: v[0] / max(v[1], 1) for k, v in pkt.items() if v[1]},
                 "assign_tflops": 2.0 * N * K * D / (pa[0] / max(pa[1], 1) / 1e3) / 1e12}
        kp.close()

    a_ms, a_n = kt["kmeans_assign"]
    a_avg = a_ms / max(a_n, 1)
    hbm, bf16, peak_src = load_peaks()
    flops = 2.0 * N * K * D
    ldbf = 64 * ((D + 63) // 64)
    terms = 2 if os.environ.get("BENCH_MODE", "bf16x3") == "bf16x3" else 1
    # bf16 copies of X read by the MMA (hi and lo for bf16x3) + labels,
    # previous labels and |x|
    traffic_alg = N * ldbf * 2 * terms + N * 4 * 3
    achieved_tflops = flops / (a_avg / 1e3) / 1e12
    k_pad = (K + 15) // 16 * 16
    executed = ((N + 127) // 128) * ((3 if terms == 2 else 1) * (ldbf // 16) + 1) * \
        2.0 * 128 * k_pad * 16
    achieved_gbs = traffic_alg / (a_avg / 1e3) / 1e9
    t_tensor = flops / (bf16 * 1e12)
    t_hbm = traffic_alg / (hbm * 1e9)
    if t_hbm >= t_tensor:
        roof = {"bound": "hbm", "achieved": achieved_gbs, "peak": hbm, "unit": "GB/s",
                "frac": achieved_gbs / hbm}
    else:
        roof = {"bound": "tensor", "achieved": achieved_tflops, "peak": bf16, "unit": "TFLOP/s",
                "frac": achieved_tflops / bf16}
    traffic, traffic_src = None, None
    prof = os.path.join(ROOT, "profiles", "kmeans_tc_kernels_600kx64_k256_ncu.md")
    if tensor_core and N == 1_000_000 and os.path.exists(prof):
        import re
        m = re.search(r"dram_bytes_per_launch_scaled_to_1000000_rows: (\d+)", open(prof).read())
        if m:
            traffic = int(m.group(1))
            traffic_src = ("ncu dram__bytes_read.sum + dram__bytes_write.sum of one launch at "
                           "600,000 rows, scaled by rows (profiles/kmeans_tc_kernels_600kx64_k256_ncu.md)")
    roof.update({"traffic": traffic, "traffic_source": traffic_src, "peak_source": peak_src,
                 "kernel": "kmeans_assign_tc_kernel (tcgen05 bf16, TMEM fp32)" if tensor_core
                 else "kmeans_assign_kernel (SIMT fp32)",
                 "algorithmic_flops_per_launch": flops,
                 "algorithmic_bytes_per_launch": traffic_alg,
                 "avg_launch_ms": a_avg, "tensor_tflops": achieved_tflops,
                 "tensor_frac": achieved_tflops / bf16, "hbm_gbs": achieved_gbs,
                 "hbm_frac": achieved_gbs / hbm,
                 # the MMAs the kernel executes: per 128-row tile, per 16-wide K
                 # step one product (bf16) or three (bf16x3), plus one K = 16
                 # MMA adding |c|^2, each 2 x 128 x k_pad x 16 flop
                 "executed_tensor_tflops": executed / (a_avg / 1e3) / 1e12,
                 "executed_tensor_frac": executed / (a_avg / 1e3) / 1e12 / bf16,
                 "kernel_ms": {k: v[0] / max(v[1], 1) for k, v in kt.items() if v[1]}})

    accuracy = None
    if rank == 0 and world == 1 and not args.no_accuracy:
        accuracy = c2_accuracy(ab, X, C0, km.labels(N), km.centres(K, D), float(km.rinfo()[4]))
    # e2e: host (pinned) -> device every step, labels + centres back
    e2e = None
    if not args.no_e2e:
        e2e = run_e2e(ab, km, X, C0, stream, args, world)
    cb = None
    if rank == 0 and world == 1 and not args.no_cpu:
        cb = cpu_baseline(X, C0)
    knn = None
    if rank == 0 and world == 1 and not args.no_knn:
        knn = run_knn(ab, accuracy=not args.no_accuracy)
    c1 = None
    if rank == 0 and world == 1 and not args.no_c1:
        c1 = run_c1(ab)
    batched = None
    if rank == 0 and world == 1 and not args.no_batched:
        batched = run_batched(ab)
    radius = None
    if rank == 0 and world == 1 and not args.no_radius:
        radius = run_radius(ab)
    ivf = None
    if rank == 0 and world == 1 and not args.no_ivf:
        ivf = run_ivf(ab)
    serving = None
    if rank == 0 and world == 1 and not args.no_serve:
        serving = run_serving(ab)
    extra = {"iterations_per_step": n_iter, "init_ms": init_ms,
             "init_ms_first_call": init_first_ms,
             "init_note": "k-means++ (seed 1) with X resident; the first call also uploads X",
             "accuracy": accuracy,
             "legs_summary": legs_summary(knn, c1, batched, serving, radius, ivf, plain, value),
             "relabelled_rows_last_iteration": relabelled,
             "lloyd_loop_as_cuda_graph": bool(graph_loop == 1.0),
             "full_scan_rows_last_iteration": full_scan,
             "precision_path": (f"{mode} tcgen05 candidate pass + exact fp32 re-score of "
                                "uncertified rows") if tensor_core else "plain fp32 (SIMT)"}
    out = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": config_dict(args) | extra,
        "roofline": roof,
        "cpu_baseline": cb,
        "e2e": e2e,
        "gpu_launches": (6 * n_iter + 8) * args.steps,
        "clocks": clocks,
        "plain_fp32": plain,
        "speedup_vs_plain_fp32": (value / plain["value"]) if plain else None,
        "knn": knn,
        "knn_fp64_c1": c1,
        "kmeans_batched": batched,
        "serving": serving,
        "ivf_flat": ivf,
        "radius": radius,
    }
    if rank == 0:
        print(json.dumps(out))
        sys.stdout.flush()
    return 0


def c2_accuracy(ab, X, C0, labels, centres, inertia, tie_rel=1e-6):
    """Errors of the k-means results against the fp64 oracle, over all rows:
    * the centre update: one Lloyd step from C0 on the default path (its
      centres are the means of the fp32 assignment to C0) against the fp64
      means of the oracle's fp32 assignment to C0 -- max abs / max rel error
      (elements above 1e-3 of the largest) and the Frobenius relative error;
    * the fit's labels against the oracle's fp32 assignment to the fit's
      centres (mismatches, expected 0), and the rows whose best and second
      best fp64 squared distances differ by at most tie_rel relative (where a
      label depends on rounding: counted, not excluded);
    * the fit's inertia against the fp64 inertia of its labels and centres."""
    orc = _oracle()
    k, d = C0.shape
    h = ab.KMeans(k, "s", order=ab.ROW_MAJOR, max_iter=1, n_init=1)
    h.set("convergence tolerance", TOL)
    h.fit(X, C0=C0)
    C1 = h.centres(k, d).astype(np.float64)
    h.close()
    lab0, _ = orc.kmeans_assign(X, C0)
    Cm, _ = orc.kmeans_update(X, lab0, k)
    err = np.abs(C1 - Cm)
    big = np.abs(Cm) > 1e-3 * np.abs(Cm).max()
    lab_o, gap = orc.kmeans_assign(X, centres)
    Xd = X.astype(np.float64)
    cd = centres.astype(np.float64)
    best = ((Xd[:4096, None, :] - cd[None, :, :]) ** 2).sum(-1).min(1)  # scale of the gaps
    scale = float(np.median(best))
    i64 = orc.kmeans_inertia(X, labels, cd)
    return {"centre_update_max_abs_err": float(err.max()),
            "centre_update_max_rel_err": float((err[big] / np.abs(Cm[big])).max()),
            "centre_update_frobenius_rel_err": float(np.linalg.norm(C1 - Cm) / np.linalg.norm(Cm)),
            "label_mismatches_vs_oracle": int((labels != lab_o).sum()),
            "near_tie_rows": int((gap <= tie_rel * scale).sum()),
            "tie_tolerance": f"fp64 gap between best and second-best squared distance <= "
                             f"{tie_rel:g} x the median best squared distance ({scale:.4g})",
            "inertia_rel_err_vs_fp64": float(abs(inertia - i64) / i64),
            "oracle": "fp32 assignment in the reference's fma order; fp64 means, inertia and gaps"}


def knn_accuracy(X, Q, ind, dist, k, metric, nsample=20, tie_rel=1e-6):
    """kNN results against the oracle on the first nsample queries: indices
    and distances identical to the oracle's fp32 search; the returned fp32
    distances against fp64 distances of the same rows (max abs / rel error);
    queries whose k-th and (k+1)-th fp64 distances differ by at most
    tie_rel relative."""
    orc = _oracle()
    Qs = np.ascontiguousarray(Q[:nsample])
    oi, od = orc.knn(X, Qs, k, metric=metric)
    same = bool(np.array_equal(oi, ind[:nsample]) and np.array_equal(od, dist[:nsample]))
    Qd = Qs.astype(np.float64)
    qn = (Qd * Qd).sum(1)
    ref = np.zeros((nsample, k))
    cand = []
    for b in range(0, X.shape[0], 262_144):
        xb = X[b:b + 262_144].astype(np.float64)
        xn = (xb * xb).sum(1)
        dot = xb @ Qd.T
        if metric == "cosine":
            dd = 1.0 - dot / np.sqrt(np.outer(xn, qn))
        else:
            dd = np.maximum(xn[:, None] + qn[None, :] - 2.0 * dot, 0.0)
        part = np.partition(dd, k, axis=0)[: k + 1]
        cand.append(part)
    allc = np.sort(np.concatenate(cand, axis=0), axis=0)[: k + 1].T
    for q in range(nsample):
        xr = X[ind[q]].astype(np.float64)
        if metric == "cosine":
            xn = (xr * xr).sum(1)
            ref[q] = 1.0 - (xr @ Qd[q]) / np.sqrt(xn * qn[q])
        else:
            ref[q] = np.sqrt(((xr - Qd[q]) ** 2).sum(1))
    kth = allc
    if metric != "cosine":
        kth = np.sqrt(kth)
    e = np.abs(dist[:nsample].astype(np.float64) - ref)
    ties = int((kth[:, k] - kth[:, k - 1] <= tie_rel * np.maximum(np.abs(kth[:, k]), 1e-30)).sum())
    return {"identical_to_oracle": same, "sample_queries": nsample,
            "max_abs_err_vs_fp64": float(e.max()),
            "max_rel_err_vs_fp64": float((e / np.maximum(np.abs(ref), 1e-30)).max()),
            "queries_with_kth_tie": ties,
            "tie_tolerance": f"k-th and (k+1)-th fp64 distances within {tie_rel:g} relative"}


def run_c1(ab, reps=5):
    """Plain brute-force kNN, fp64: 10,000 x 32 training rows from a
    16-component isotropic Gaussian mixture (means U[-5, 5]^32, sigma 1,
    labels = component id), 2,000 queries from the mixture, seed 0, k = 10,
    euclidean, uniform weights.  A timed call is da_nn_kneighbors_d plus
    da_nn_classifier_predict_d over all queries with host arrays (best of
    5); the neighbours, distances and labels must equal the oracle's.  CPU:
    the oracle's search (all host threads) and the same vote."""
    rng = np.random.default_rng(0)
    n, nq, d, comps, k = 10_000, 2_000, 32, 16, 10
    means = rng.uniform(-5.0, 5.0, (comps, d))
    y = rng.integers(0, comps, n)
    X = means[y] + rng.standard_normal((n, d))
    ql = rng.integers(0, comps, nq)
    Q = means[ql] + rng.standard_normal((nq, d))
    nn = ab.KNN("d", order=ab.ROW_MAJOR, weights="uniform", number_of_neighbors=k).fit(X, y=y)
    nn.kneighbors(Q[:64], k)
    nn.predict(Q[:64])
    ts = []
    for _ in range(reps):
        t = time.perf_counter()
        ind, dist = nn.kneighbors(Q, k)
        pred = nn.predict(Q)
        ts.append(time.perf_counter() - t)
    nn.close()
    orc = _oracle()
    t = time.perf_counter()
    oi, od = orc.knn(X, Q, k)
    classes = np.unique(y)
    cnt = np.zeros((nq, classes.size))
    for r in range(k):
        np.add.at(cnt, (np.arange(nq), np.searchsorted(classes, y[oi[:, r]])), 1.0)
    opred = classes[np.argmax(cnt, axis=1)]
    cpu_s = time.perf_counter() - t
    return {"workload": f"knn_fp64_euclidean_{n}x{d}_q{nq}_k{k}_gmm{comps}_predict",
            "unit": "queries/s", "qps": nq / min(ts),
            "identical_to_oracle": bool(np.array_equal(ind, oi) and np.array_equal(dist, od)
                                        and np.array_equal(pred, opred)),
            "flops_per_call": 2.0 * n * nq * d,
            "cpu_baseline": {"value": nq / cpu_s, "unit": "queries/s",
                             "cores": orc.num_threads(), "kind": "port",
                             "sample": "all 2,000 queries: the oracle's fp64 search (one query "
                                       "per OpenMP thread at a time) and the uniform vote"},
            "timing": "wall clock of da_nn_kneighbors_d + da_nn_classifier_predict_d with host "
                      "arrays (best of 5)"}


def legs_summary(knn, c1, batched, serving, radius, ivf, plain, value):
    """One compact line per workload, kept beside the headline numbers."""
    out = {"kmeans_c2": {"iters_per_s": value,
                         "plain_fp32_iters_per_s": plain["value"] if plain else None}}
    if knn:
        for m in ("euclidean", "cosine"):
            r = knn if m == "euclidean" else knn.get("cosine")
            if r:
                acc = r.get("accuracy") or {}
                out[f"knn_c3_{m}"] = {"qps": r["qps"], "plain_qps": r["plain_qps"],
                                      "identical_to_plain": r["identical_to_plain"],
                                      "identical_to_oracle_sample": acc.get("identical_to_oracle"),
                                      "max_rel_err_vs_fp64": acc.get("max_rel_err_vs_fp64"),
                                      "queries_with_kth_tie": acc.get("queries_with_kth_tie")}
    if c1:
        out["knn_fp64_c1"] = {"qps": c1["qps"], "identical_to_oracle": c1["identical_to_oracle"],
                              "cpu_qps": c1["cpu_baseline"]["value"]}
    if batched:
        out["kmeans_batched_c4"] = {"iters_per_s": batched["value"],
                                    "speedup_vs_per_instance": batched["speedup_vs_per_instance_calls"],
                                    "identical": batched["identical_to_single"]}
    if serving:
        srv = {}
        for key, v in serving.items():
            if isinstance(v, dict) and "requests_1_256_queries" in v:
                srv[key] = {"p50_ms": v["requests_1_256_queries"]["p50_ms"],
                            "p99_ms": v["requests_1_256_queries"]["p99_ms"],
                            "queries_per_s": v["queries_per_s"]}
        out["serving_c5_1_256_query_requests"] = srv
    if radius:
        out["radius"] = {"qps": radius["qps"], "identical_to_oracle_sample":
                         radius["identical_to_oracle_sample"]}
    if ivf:
        out["ivf_flat"] = {"qps": ivf["qps"], "recall": ivf["recall_at_k_vs_exact"]}
    return out


def run_sharded(ab, args, rank, world, local):
    """k-means over a data set split across the ranks (weak scaling): every
    rank holds a copy of the 1,000,000 x 64 set as its shard, so the job
    clusters world x 1,000,000 rows; per Lloyd iteration every rank assigns
    its rows and writes its integer centroid sums (sharded.py), ONE NCCL
    all-reduce of k*d + k + 1 int64 follows, and every rank computes the
    same centres.  value = world x Lloyd iterations / s (the single-GPU unit:
    iterations over 1,000,000 rows); e2e re-uploads the shard from pinned
    host memory and reads labels and centres back in every step."""
    import torch
    sd = _load("aoclda_sharded", os.path.join(PKG, "sharded.py"))
    comm = sd.TorchComm()
    X = make_data()
    mode = os.environ.get("BENCH_MODE", "bf16x3")
    # the k-means++ centres of the single-GPU workload, from rank 0
    C0 = np.zeros((K, D), dtype=np.float32)
    if rank == 0:
        km0 = ab.KMeans(K, "s", order=ab.ROW_MAJOR, max_iter=MAX_ITER, n_init=1, seed=SEED)
        km0.set_data(X)
        C0 = km0.init_centres(K)
        km0.close()
    c0 = torch.from_numpy(np.ascontiguousarray(C0)).cuda()
    torch.distributed.broadcast(c0, 0)
    C0 = c0.cpu().numpy()
    shard = sd.DeviceKMeansShard(ab, X, K, precision_mode=mode)
    stream = shard.stream

    def step():
        return sd.kmeans_fit([shard], C0, comm, max_iter=MAX_ITER, tol=TOL)["n_iter"]

    def timed(fn, steps, warmup, sample_clocks=False):
        for _ in range(warmup):
            fn()
        torch.distributed.barrier()
        torch.cuda.synchronize()
        clk = Clocks(local) if sample_clocks else None
        if clk:
            clk.start()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        iters = 0
        for _ in range(steps):
            iters += fn()
        e1.record(stream)
        torch.cuda.synchronize()
        clocks = clk.stop() if clk else None
        t = torch.tensor([e0.elapsed_time(e1)], device="cuda")
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
        return float(t.item()), iters, clocks

    ms, iters, clocks = timed(step, args.steps, args.warmup, sample_clocks=True)
    n_iter = iters // args.steps
    value = world * iters / (ms / 1e3)
    # kernel times of one step (event timing serialises the launches)
    L = shard.km.L
    L.da_b200_set_kernel_timing(shard.km.h, 1)
    L.da_b200_reset_kernel_time(shard.km.h)
    step()
    L.da_b200_set_kernel_timing(shard.km.h, 0)
    kt = {n: shard.km.kernel_time(n) for n in ("kmeans_assign", "kmeans_rescore", "kmeans_update")}
    a_ms, a_n = kt["kmeans_assign"]
    a_avg = a_ms / max(a_n, 1)
    hbm, bf16, peak_src = load_peaks()
    flops = 2.0 * N * K * D
    tensor_core = shard.km.stat("tensor_core") == 1.0
    achieved = flops / (a_avg / 1e3) / 1e12
    roof = {"bound": "tensor", "achieved": achieved, "peak": bf16, "unit": "TFLOP/s",
            "frac": achieved / bf16, "traffic": None, "peak_source": peak_src,
            "kernel": "kmeans_assign_tc_kernel (tcgen05 bf16, TMEM fp32)" if tensor_core
            else "kmeans_assign_kernel (SIMT fp32)", "avg_launch_ms": a_avg,
            "kernel_ms": {k: v[0] / max(v[1], 1) for k, v in kt.items() if v[1]}}

    e2e = None
    if not args.no_e2e:
        Xp = torch.empty((N, D), dtype=torch.float32, pin_memory=True).numpy()
        Xp[:] = X

        def e2e_step():
            shard.km.set_data(Xp)
            it = sd.kmeans_fit([shard], C0, comm, max_iter=MAX_ITER, tol=TOL)["n_iter"]
            shard.result()
            return it

        ems, eiters, _ = timed(e2e_step, args.steps, max(1, min(args.warmup, 2)))
        e2e = {"value": world * eiters / (ems / 1e3), "unit": UNIT,
               "h2d_bytes_per_step": N * D * 4 + K * D * 4 + D * 4,
               "d2h_bytes_per_step": N * 4 + K * D * 4 + D * 4}
    shard.close()
    cfg = config_dict(args) | {
        "workload": f"kmeans_lloyd_fp32_{N}x64_k256_split_over_{world}_ranks",
        "n_samples_total": N * world,
        "parallelism": f"data split over {world} ranks (one shard each, every shard a copy of "
                       f"the {N} x 64 set); one NCCL all-reduce of k*d+k+1 int64 per Lloyd "
                       "iteration",
        "iterations_per_step": n_iter,
        "step": "one sharded Lloyd fit (sharded.kmeans_fit) = n_iter iterations on every rank"}
    out = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
           "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True,
           "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
           "config": cfg, "roofline": roof, "cpu_baseline": None, "e2e": e2e,
           "gpu_launches": (7 * n_iter + 10) * args.steps, "clocks": clocks}
    if rank == 0:
        print(json.dumps(out))
        sys.stdout.flush()
    return 0


def run_knn(ab, nx=4_000_000, nq=10_000, d=128, k=100, comps=1024, seed=3, reps=3, plain=True,
            metrics=("euclidean", "cosine"), accuracy=True):
    """Brute-force kNN, fp32 euclidean and cosine: 4,000,000 x 128 training
    rows from a 1,024-component Gaussian mixture (the k-means recipe) plus 1%
    exact duplicate rows (ties), 10,000 queries from the same mixture, k =
    100.  Each timed call is one da_nn_kneighbors_s over all queries with host
    arrays (queries up, indices and distances down).  The tensor-core path
    (bf16x3 candidate pass + exact re-score) and the plain fp32 path must
    return identical indices and distances.  The top-level keys are the
    euclidean results; the cosine ones are under "cosine"."""
    rng = np.random.default_rng(seed)
    means = rng.uniform(-10.0, 10.0, (comps, d)).astype(np.float32)
    sig = rng.uniform(0.5, 2.0, comps).astype(np.float32)
    w = rng.dirichlet(np.ones(comps))
    lab = rng.choice(comps, nx, p=w)
    X = means[lab] + rng.standard_normal((nx, d), dtype=np.float32) * sig[lab, None]
    X = np.concatenate([X, X[rng.integers(0, nx, nx // 100)]])
    ql = rng.choice(comps, nq, p=w)
    Q = means[ql] + rng.standard_normal((nq, d), dtype=np.float32) * sig[ql, None]
    out = {}
    for metric in metrics:
        res = {}
        for mode in ("bf16x3", "plain") if plain else ("bf16x3",):
            nn = ab.KNN("s", order=ab.ROW_MAJOR, metric=metric, precision_mode=mode).fit(X)
            nn.kneighbors(Q[:512], k)
            nn.L.da_b200_set_kernel_timing(nn.h, 1)
            ts = []
            for _ in range(reps if mode == "bf16x3" else 1):
                t = time.perf_counter()
                ind, dist = nn.kneighbors(Q, k)
                ts.append(time.perf_counter() - t)
            kern = {}
            for name in ("knn_tc", "knn_chunks", "knn_merge"):
                ms_, n_ = nn.kernel_time(name)
                if n_:
                    kern[name] = ms_ / n_
            res[mode] = {"s": min(ts), "ind": ind, "dist": dist, "tc": nn.stat("tensor_core"),
                         "kernel_ms": kern, "list_mean": nn.stat("knn_tc_mean_list"),
                         "fallback": nn.stat("knn_tc_fallback_queries")}
            nn.close()
        tc, pl = res["bf16x3"], res.get("plain")
        flops = 2.0 * (nx + nx // 100) * nq * d
        out[metric] = {
            "workload": f"knn_fp32_{metric}_{nx + nx // 100}x{d}_q{nq}_k{k}",
            "unit": "queries/s", "qps": nq / tc["s"],
            "plain_qps": nq / pl["s"] if pl else None,
            "speedup_vs_plain_fp32": pl["s"] / tc["s"] if pl else None,
            "identical_to_plain": bool(np.array_equal(tc["ind"], pl["ind"]) and
                                       np.array_equal(tc["dist"], pl["dist"])) if pl else None,
            "tensor_core": tc["tc"] == 1.0, "kernel_ms": tc["kernel_ms"],
            "plain_kernel_ms": pl["kernel_ms"] if pl else None,
            "tensor_tflops_algorithmic":
                flops / (tc["kernel_ms"].get("knn_tc", float("nan")) / 1e3) / 1e12,
            "candidate_list_mean": tc["list_mean"], "plain_fallback_queries": tc["fallback"],
            "accuracy": knn_accuracy(X, Q, tc["ind"], tc["dist"], k, metric) if accuracy else None,
            "timing": "wall clock of one da_nn_kneighbors_s call with host arrays (best of 3)"}
    first = out[metrics[0]]
    res = dict(first, **{m: out[m] for m in metrics[1:]})
    if accuracy:
        res["fp8_candidate_measurement"] = fp8_candidate_measurement(X, Q, k)
    return res


def fp8_candidate_measurement(X, Q, k, nsample=64):
    """Certified candidate sets of a one-pass tensor-core candidate search,
    measured on the kNN workload's data (the first nsample queries, on the GPU
    with torch): operands rounded as the pass would round them -- bf16 hi + lo
    (the library's bf16x3 pass) or e4m3 hi + lo with a per-row power-of-two
    scale (fp8) -- and, per (query, row), the ranking value
    v' = |x|^2 - 2 x~.q~ with the rigorous operand-rounding bound
    e = 2 (|x - x~| |q| + |x~| |q - q~|).  A row can belong to the true top k
    only if v' - e <= T_q, with T_q the k-th smallest v' + e; those rows are
    the candidates the exact re-score must read.  (The tensor core's fp32
    accumulation adds to both bounds; it is left out, so the sets are lower
    bounds.)  Reported per query: mean and max candidates, and the re-score
    bytes they imply against one read of the bf16 operands."""
    import torch
    dev = torch.device("cuda")
    Xg = torch.from_numpy(X).to(dev)
    Qg = torch.from_numpy(np.ascontiguousarray(Q[:nsample])).to(dev)

    def split_bf16(A):
        h = A.to(torch.bfloat16).float()
        lo = (A - h).to(torch.bfloat16).float()
        return h + lo

    def split_e4m3(A):
        # per-row scale: a power of two that maps the row's max to <= 448
        amax = A.abs().amax(dim=1, keepdim=True).clamp_min(1e-30)
        sc = torch.exp2(torch.floor(torch.log2(448.0 / amax)))
        As = A * sc
        h = As.to(torch.float8_e4m3fn).float()
        lo = (As - h).to(torch.float8_e4m3fn).float()
        return (h + lo) / sc

    xn2 = (Xg.double() ** 2).sum(1)
    qn = Qg.double().norm(dim=1)
    out = {}
    for name, fn in (("bf16x3", split_bf16), ("fp8_e4m3_hi_lo", split_e4m3)):
        Xt, Qt = fn(Xg), fn(Qg)
        ex = (Xg - Xt).double().norm(dim=1)
        xtn = Xt.double().norm(dim=1)
        eq = (Qg - Qt).double().norm(dim=1)
        cand = []
        G = Xt.double() @ Qt.double().T  # rows x sample queries
        for q in range(Qg.shape[0]):
            v = xn2 - 2.0 * G[:, q]
            e = 2.0 * (ex * qn[q] + xtn * eq[q])
            T = torch.kthvalue((v + e).cpu(), k).values.item()
            cand.append(int(((v - e) <= T).sum().item()))
        del G
        c = np.array(cand, dtype=np.float64)
        out[name] = {"mean_candidates": float(c.mean()), "max_candidates": int(c.max()),
                     "rescore_bytes_per_query": float(c.mean() * X.shape[1] * 4)}
        del Xt, Qt
    bf16_pass = X.shape[0] * X.shape[1] * 4  # bf16 hi + lo of every training row, once
    for v in out.values():
        v["rescore_bytes_vs_one_bf16x3_read_per_query"] = v["rescore_bytes_per_query"] / bf16_pass
    out["sample_queries"] = int(Qg.shape[0])
    out["note"] = ("operand-rounding part of the certificate only (lower bounds on the sets); "
                   "re-score bytes = candidates x d x 4 per query")
    del Xg, Qg
    torch.cuda.empty_cache()
    return out


def run_radius(ab, nx=1_000_000, nq=10_000, d=32, comps=256, target=100, seed=6, reps=3,
               cpu_queries=20):
    """Radius neighbours, fp32 euclidean: 1,000,000 x 32 rows of a 256-component
    Gaussian mixture, 10,000 queries from the mixture, the radius at which the
    median query has 100 neighbours.  Each timed call is one
    da_nn_radius_neighbors_s over all queries with host arrays (queries up;
    counts, indices and distances down; results in index order).  Roofline: on
    the tensor-core path the mask pass's bf16x3 products (3 x 2 flop per pair
    and feature, features in steps of 16) over its CUDA-event time; on the
    plain path the distance blocks, written once and read once (8 bytes per
    pair), over the three kernels' time.
    CPU: the oracle on a sample of queries."""
    rng = np.random.default_rng(seed)
    means = rng.uniform(-3.0, 3.0, (comps, d)).astype(np.float32)
    lab = rng.integers(0, comps, nx)
    X = means[lab] + rng.standard_normal((nx, d), dtype=np.float32)
    ql = rng.integers(0, comps, nq)
    Q = means[ql] + rng.standard_normal((nq, d), dtype=np.float32)
    # the radius: median over 64 queries of the distance of their 100th neighbour
    xs = (X.astype(np.float64) ** 2).sum(1)
    kth = []
    for q in Q[:64].astype(np.float64):
        d2 = xs + (q * q).sum() - 2.0 * (X @ q.astype(np.float32)).astype(np.float64)
        kth.append(np.sqrt(max(np.partition(d2, target)[target], 0.0)))
    r = float(np.median(kth))
    nn = ab.KNN("s", order=ab.ROW_MAJOR).fit(X)
    nn.radius_neighbors(Q[:64], r, True, False)
    nn.L.da_b200_set_kernel_timing(nn.h, 1)
    ts = []
    for _ in range(reps):
        t = time.perf_counter()
        cnt, off, ind, dist = nn.radius_neighbors(Q, r, True, False)
        ts.append(time.perf_counter() - t)
    kern = {}
    for name in ("radius_distances", "radius_count", "radius_emit"):
        ms_, n_ = nn.kernel_time(name)
        kern[name] = (ms_, n_)
    tc = nn.stat("tensor_core") == 1.0
    nn.close()
    hbm, tflops, src = load_peaks()
    if tc:
        ms_ = kern["radius_distances"][0] / reps
        done = 3 * 2.0 * nx * nq * ((d + 15) // 16 * 16) / (ms_ / 1e3) / 1e12
        roofline = {"bound": "tensor", "achieved": done, "peak": tflops, "unit": "TFLOP/s",
                    "frac": done / tflops, "peak_source": src, "traffic": None,
                    "note": "bf16x3 products of the mask pass (K steps of 16)"}
    else:
        ms_ = sum(v[0] for v in kern.values()) / reps
        done = 8.0 * nq * nx / (ms_ / 1e3) / 1e9
        roofline = {"bound": "hbm", "achieved": done, "peak": hbm, "unit": "GB/s",
                    "frac": done / hbm, "peak_source": src, "traffic": None,
                    "note": "8 bytes per (query, row): distance written once, read once"}
    orc = _load("oracle_mod", os.path.join(ORACLE, "oracle.py"))
    t = time.perf_counter()
    ref = orc.radius(X, Q[:cpu_queries], r)
    cpu_s = time.perf_counter() - t
    same = all(np.array_equal(ind[off[q]:off[q] + cnt[q]], ref[q][0]) and
               np.array_equal(dist[off[q]:off[q] + cnt[q]], ref[q][1])
               for q in range(cpu_queries) if cnt[q])
    return {"workload": f"radius_fp32_euclidean_{nx}x{d}_q{nq}_median{target}neighbours",
            "unit": "queries/s", "qps": nq / min(ts), "radius": r,
            "neighbours_mean": float(cnt[nq]) / nq,
            "kernel_ms_per_call": {k: v[0] / reps for k, v in kern.items()},
            "launches_per_call": {k: v[1] // reps for k, v in kern.items()},
            "tensor_core": tc, "roofline": roofline,
            "identical_to_oracle_sample": bool(same),
            "cpu_baseline": {"value": cpu_queries / cpu_s, "unit": "queries/s", "cores": 1,
                             "kind": "port", "sample": f"{cpu_queries} queries, oracle"},
            "timing": "wall clock of one da_nn_radius_neighbors_s call with host arrays "
                      "(best of 3)"}


def run_ivf(ab, nx=1_000_000, nq=10_000, d=128, k=10, n_list=1024, n_probe=16, comps=1024,
            seed=5, reps=3, cpu_queries=100):
    """IVF-flat approximate neighbours, fp32 squared euclidean: 1,000,000 x 128
    rows of a 1,024-component Gaussian mixture, n_list = 1,024 lists (GPU
    k-means, 10 iterations), n_probe = 16, 10,000 queries from the mixture,
    k = 10.  Each timed search is one da_approx_nn_kneighbors_s over all
    queries with host arrays; recall@k against the exact GPU kNN of the same
    rows.  Roofline of the list scan: one read of every probed list (4 * 128 +
    8 bytes a row), which is all that has to come from HBM, over its CUDA-event
    time; the candidate rows as each query reads them, most of them from L2, are
    a figure of their own.  CPU: the oracle's search (numpy) on a sample of
    queries, one thread of Python per query."""
    rng = np.random.default_rng(seed)
    means = rng.uniform(-10.0, 10.0, (comps, d)).astype(np.float32)
    sig = rng.uniform(0.5, 2.0, comps).astype(np.float32)
    lab = rng.integers(0, comps, nx)
    X = means[lab] + rng.standard_normal((nx, d), dtype=np.float32) * sig[lab, None]
    ql = rng.integers(0, comps, nq)
    Q = means[ql] + rng.standard_normal((nq, d), dtype=np.float32) * sig[ql, None]
    h = ab.ApproxNN("s", order=ab.ROW_MAJOR, n_list=n_list, n_probe=n_probe, seed=seed,
                    kmeans_iter=10)
    h.set_training_data(X)
    t = time.perf_counter()
    h.train()
    train_s = time.perf_counter() - t
    t = time.perf_counter()
    h.add(X)
    add_s = time.perf_counter() - t
    h.kneighbors(Q[:256], k)
    h.L.da_b200_set_kernel_timing(h.h, 1)
    ts = []
    for _ in range(reps):
        t = time.perf_counter()
        ind, dist = h.kneighbors(Q, k)
        ts.append(time.perf_counter() - t)
    ms_, n_ = h.kernel_time("ivf_scan")
    scan_ms = ms_ / max(n_, 1)
    sizes = h.list_sizes(n_list).astype(np.int64)
    C = h.result(ab.APPROX_NN_CENTROIDS, n_list * d).reshape(n_list, d).astype(np.float64)
    Qd = Q.astype(np.float64)
    dc = (Qd * Qd).sum(1)[:, None] + (C * C).sum(1)[None] - 2.0 * Qd @ C.T
    probes = np.argsort(dc, axis=1, kind="stable")[:, :n_probe]
    cand = int(sizes[probes].sum())
    row = 4.0 * d + 8.0
    bytes_ = float(sizes[np.unique(probes)].sum()) * row
    hbm, _, src = load_peaks()
    h.close()
    exact = ab.KNN("s", order=ab.ROW_MAJOR, metric="sqeuclidean").fit(X)
    eind, _ = exact.kneighbors(Q, k)
    exact.close()
    recall = float(np.mean([len(set(a) & set(b)) / k for a, b in zip(ind, eind)]))
    orc = _load("oracle_mod", os.path.join(ORACLE, "oracle.py"))
    t = time.perf_counter()
    member = np.zeros(nx, dtype=np.int32)
    # the list of every row from the trained centroids (host, fp64), then
    # the oracle's per-query search on a sample
    for b in range(0, nx, 65536):
        xb = X[b:b + 65536].astype(np.float64)
        member[b:b + 65536] = np.argmin((xb * xb).sum(1)[:, None] + (C * C).sum(1)[None]
                                        - 2.0 * xb @ C.T, axis=1)
    assign_s = time.perf_counter() - t
    t = time.perf_counter()
    orc.ivf_kneighbors(C, X, Q[:cpu_queries], k, n_probe, "sqeuclidean", member)
    cpu_s = time.perf_counter() - t
    return {"workload": f"ivfflat_fp32_sqeuclidean_{nx}x{d}_nlist{n_list}_nprobe{n_probe}"
                        f"_q{nq}_k{k}",
            "unit": "queries/s", "qps": nq / min(ts), "train_s": train_s, "add_s": add_s,
            "recall_at_k_vs_exact": recall, "scan_kernel_ms": scan_ms,
            "candidates_per_query": cand / nq,
            "candidate_gb_per_s_with_l2": cand * row / (scan_ms / 1e3) / 1e9,
            "roofline": {"bound": "hbm", "achieved": bytes_ / (scan_ms / 1e3) / 1e9,
                         "peak": hbm, "unit": "GB/s",
                         "frac": bytes_ / (scan_ms / 1e3) / 1e9 / hbm,
                         "peak_source": src, "traffic": None,
                         "note": "one read of the probed lists"},
            "cpu_baseline": {"value": cpu_queries / cpu_s, "unit": "queries/s", "cores": 1,
                             "kind": "port",
                             "sample": f"{cpu_queries} queries, oracle numpy search "
                                       f"(list assignment of the rows, {assign_s:.1f} s, "
                                       "not included)"},
            "timing": "wall clock of one da_approx_nn_kneighbors_s call with host arrays "
                      "(best of 3)"}


def run_serving(ab, nx=8_000_000, d=96, comps=2048, n_models=64,
                rates=(250.0, 1000.0, 2000.0, 10000.0, 50000.0), seconds=2.0, seed=5,
                server_kw=None, plain=True):
    """Serving: a resident kNN index of 8,000,000 x 96 fp32 rows from a
    2,048-component Gaussian mixture (the k-means recipe) and 64 k-means
    models (d = 96, 256 centres, each fitted on 20,000 rows of its own
    mixture).  A seeded trace of Poisson arrivals at 2,000 requests/s for 2 s:
    per-request query count lognormal(ln 16, 1.5) clipped to [1, 4096],
    k uniform in {1, 10, 100}, one request in five a predict on a random
    model.  Served by the continuous-batching loop (two kNN workers, the
    first a fast lane for requests of at most 256 queries, at most 512 queries
    per library call, larger requests split into parts, small and
    long-waiting requests first), after 0.5 s of unmeasured traffic at the
    same rate; p50 / p99 latency (submit to completion)
    and queries/s at 250, 1,000, 2,000, 10,000 and 50,000 requests/s for the
    tensor-core path (the two highest rates as 2,000-request traces, past the
    device's capacity: their latency grows with the trace and their
    queries/s is the saturated throughput), and at 250 requests/s for the
    plain fp32 path (which cannot keep up, so its queue grows)."""
    sv = _load("aoclda_serving", os.path.join(PKG, "serving.py"))
    rng = np.random.default_rng(seed)
    means = rng.uniform(-10.0, 10.0, (comps, d)).astype(np.float32)
    sig = rng.uniform(0.5, 2.0, comps).astype(np.float32)
    w = rng.dirichlet(np.ones(comps))
    lab = rng.choice(comps, nx, p=w)
    X = means[lab] + rng.standard_normal((nx, d), dtype=np.float32) * sig[lab, None]
    models = {}
    for m in range(n_models):
        mm = rng.uniform(-10.0, 10.0, (256, d)).astype(np.float32)
        lm = rng.integers(0, 256, 20_000)
        Xm = mm[lm] + rng.standard_normal((20_000, d), dtype=np.float32)
        models[m] = (Xm, Xm[rng.choice(20_000, 256, replace=False)].copy())
    def make_trace(rate, trng):
        # 2 s of arrivals, at most 2,000 requests (the highest rates are past
        # the device's capacity: their trace measures the saturated service)
        span = min(seconds, 2000.0 / rate)
        trace, t = [], 0.0
        while t < span:
            t += trng.exponential(1.0 / rate)
            size = int(np.clip(trng.lognormal(np.log(16), 1.5), 1, 4096))
            if trng.random() < 0.2:
                trace.append((t, "predict", size, int(trng.integers(0, n_models))))
            else:
                trace.append((t, "knn", size, int(trng.choice([1, 10, 100]))))
        return trace

    qrng = np.random.default_rng(seed + 1)

    def queries(size):
        li = qrng.choice(comps, size, p=w)
        return means[li] + qrng.standard_normal((size, d), dtype=np.float32) * sig[li, None]

    out = {"workload": f"serve_fp32_index_{nx}x{d}_{n_models}_models_poisson_{seconds:g}s"}
    kw = {"workers": 2, "max_batch_queries": 512} | dict(server_kw or {})
    modes = (("bf16x3", rates), ("plain", rates[:1])) if plain else (("bf16x3", rates),)
    for mode, mode_rates in modes:
        server = sv.Server(ab, X, models=models, precision_mode=mode, **kw)
        for rate in mode_rates:
            # half a second of the same traffic first (not measured): the
            # measured trace starts from a serving steady state
            sv.replay(server, make_trace(rate, np.random.default_rng(seed + 7 * int(rate)))[
                : max(1, int(rate * 0.5))], queries)
            server.batches.clear()
            trace = make_trace(rate, np.random.default_rng(seed + int(rate)))
            t0 = time.perf_counter()
            reqs = sv.replay(server, trace, queries)
            wall = time.perf_counter() - t0
            small = [r for r in reqs if r.queries.shape[0] <= 256]
            nq = sum(r.queries.shape[0] for r in reqs)
            kb = [b for b in server.batches if b[0] == "knn"]
            pb = [b for b in server.batches if b[0] == "predict"]
            out[f"{mode}_{int(rate)}rps"] = {
                "requests": len(reqs), "all": sv.latency_summary(reqs),
                "requests_1_256_queries": sv.latency_summary(small),
                "knn_1_256_queries": sv.latency_summary([r for r in small if r.kind == "knn"]),
                "predict_1_256_queries": sv.latency_summary(
                    [r for r in small if r.kind == "predict"]),
                "predict_calls": len(pb),
                "mean_predict_call_ms": float(np.mean([b[3] for b in pb]) * 1e3) if pb else 0.0,
                "queries_per_s": nq / wall, "knn_calls": len(kb),
                "mean_queries_per_knn_call": float(np.mean([b[2] for b in kb])) if kb else 0.0,
                "mean_knn_call_ms": float(np.mean([b[3] for b in kb]) * 1e3) if kb else 0.0,
                "p99_knn_call_ms": float(np.percentile([b[3] for b in kb], 99) * 1e3) if kb else 0.0,
                "max_knn_call_ms": float(max(b[3] for b in kb) * 1e3) if kb else 0.0,
                "plain_fallback_queries": server.fallback_queries}
        server.close()
    return out


def batched_workload(count=512, seed=4):
    """512 independent fp32 data sets: n lognormal(ln 20000, 1) clipped to
    [1000, 200000], d uniform in {16, 32, 64, 128}, k uniform in [8, 64],
    each a Gaussian mixture with k components (the k-means recipe); initial
    centres k distinct rows."""
    rng = np.random.default_rng(seed)
    Xs, C0s = [], []
    for _ in range(count):
        n = int(np.clip(rng.lognormal(np.log(20000), 1.0), 1000, 200000))
        d = int(rng.choice([16, 32, 64, 128]))
        k = int(rng.integers(8, 65))
        means = rng.uniform(-10.0, 10.0, (k, d)).astype(np.float32)
        sig = rng.uniform(0.5, 2.0, k).astype(np.float32)
        w = rng.dirichlet(np.ones(k))
        lab = rng.choice(k, n, p=w)
        X = means[lab] + rng.standard_normal((n, d), dtype=np.float32) * sig[lab, None]
        Xs.append(np.ascontiguousarray(X))
        C0s.append(X[rng.choice(n, k, replace=False)].copy())
    return Xs, C0s


def run_batched(ab, count=512, max_iter=30, tol=1e-4, seed=4):
    """Batched k-means: 512 independent fp32 data sets, n lognormal(ln 20000,
    1) clipped to [1000, 200000], d uniform in {16, 32, 64, 128}, k uniform in
    [8, 64], each a Gaussian mixture with k components (the k-means recipe),
    initial centres k distinct rows, 30 Lloyd iterations at most (tol 1e-4).
    One da_b200_kmeans_batched_s call (host arrays in and out) against one
    da_kmeans_compute_s call per data set (precision mode plain, the
    semantics the batched path reproduces); results must be identical."""
    Xs, C0s = batched_workload(count, seed)
    # warm-up: one iteration over every data set (the tile-shape tuner meets
    # every shape here, so the timed call below uses its cached picks)
    ab.kmeans_batched(Xs, C0s, max_iter=1, tol=tol)
    t = time.perf_counter()
    out = ab.kmeans_batched(Xs, C0s, max_iter=max_iter, tol=tol)
    tb = time.perf_counter() - t
    up_ms, fit_ms, down_ms = ab.kmeans_batched_timing()
    # one launch per instance: the same call with one data set at a time
    t = time.perf_counter()
    one_fit = one_up = 0.0
    same_one = True
    for X, C0, r in zip(Xs, C0s, out):
        r1 = ab.kmeans_batched([X], [C0], max_iter=max_iter, tol=tol)[0]
        u, f, _ = ab.kmeans_batched_timing()
        one_up += u
        one_fit += f
        same_one = same_one and r1["n_iter"] == r["n_iter"] and \
            np.array_equal(r1["labels"], r["labels"])
    t1 = time.perf_counter() - t
    same = True
    t = time.perf_counter()
    for X, C0, r in zip(Xs, C0s, out):
        km = ab.KMeans(C0.shape[0], "s", order=ab.ROW_MAJOR, max_iter=max_iter, n_init=1)
        km.set("convergence tolerance", tol)
        km.set("precision mode", "plain")
        km.fit(X, C0)
        same = same and int(km.rinfo()[3]) == r["n_iter"] and \
            np.array_equal(km.labels(X.shape[0]), r["labels"])
        km.close()
    ts = time.perf_counter() - t
    iters = sum(r["n_iter"] for r in out)
    rows = sum(x.shape[0] for x in Xs)
    return {"workload": f"kmeans_batched_fp32_{count}_instances_{rows}_rows_maxit{max_iter}",
            "unit": "Lloyd iterations/s (summed over instances)",
            "value": iters / tb, "iters_per_s_fit_only": iters / (fit_ms / 1e3),
            "batched_s": tb, "device_ms": {"upload": up_ms, "fit": fit_ms, "download": down_ms},
            "one_launch_per_instance": {"wall_s": t1, "fit_ms_sum": one_fit,
                                        "upload_ms_sum": one_up,
                                        "speedup_fit_only": one_fit / fit_ms,
                                        "speedup_with_upload": t1 / tb,
                                        "identical": bool(same_one)},
            "per_instance_calls_s": ts,
            "speedup_vs_per_instance_calls": ts / tb, "identical_to_single": bool(same),
            "total_iterations": iters,
            "timing": "wall clock of the public calls with host arrays (upload, fit and "
                      "download inside); fit-only figures from the library's device timing; "
                      "one launch per instance = the same call with one data set at a time; "
                      "per-instance calls = da_kmeans_compute_s per data set (precision mode "
                      "plain), whose time includes labels download and comparison per call"}


def run_e2e(ab, km, X, C0, stream, args, world):
    import torch
    Xp = torch.empty((N, D), dtype=torch.float32, pin_memory=True).numpy()
    Xp[:] = X
    km2 = ab.KMeans(K, "s", order=ab.ROW_MAJOR, max_iter=MAX_ITER, n_init=1, seed=SEED)
    km2.L.da_b200_set_stream(km2.h, C.c_void_p(stream.cuda_stream))
    km2.set("convergence tolerance", TOL)
    km2.set("initialization method", "supplied")
    km2.set("precision mode", os.environ.get("BENCH_MODE", "bf16x3"))
    lab_host = torch.empty(N, dtype=torch.int32, pin_memory=True).numpy()
    cen_host = np.zeros(K * D, dtype=np.float32)

    def e2e_step():
        km2.call("da_kmeans_set_data_s", N, D, ab.ptr(Xp), D, ok=(0, 13))
        km2.call("da_kmeans_set_init_centres_s", ab.ptr(C0), D)
        km2.call("da_kmeans_compute_s", ok=(0, 21))
        dim = ab.da_int(N)
        km2.call("da_handle_get_result_int", ab.KMEANS_LABELS, C.byref(dim), ab.ptr(lab_host))
        dim = ab.da_int(K * D)
        km2.call("da_handle_get_result_s", ab.KMEANS_CENTRES, C.byref(dim), ab.ptr(cen_host))
        return int(km2.rinfo()[3])

    for _ in range(max(1, args.warmup)):
        e2e_step()
    torch.cuda.synchronize()
    f0, f1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    t0 = time.perf_counter()
    f0.record(stream)
    e2e_iters = 0
    for _ in range(args.steps):
        e2e_iters += e2e_step()
    f1.record(stream)
    torch.cuda.synchronize()
    wall_ms = (time.perf_counter() - t0) * 1e3
    e2e_ms = f0.elapsed_time(f1)
    e2e_value = e2e_iters * world / (e2e_ms / 1e3)
    return {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": N * D * 4 + K * D * 4,
            "d2h_bytes_per_step": N * 4 + K * D * 4 + 6 * 4, "ms_per_step": e2e_ms / args.steps,
            "host_wall_ms_per_step": wall_ms / args.steps,
            "iterations_per_step": e2e_iters / args.steps}


if __name__ == "__main__":
    sys.exit(main())
