#!/usr/bin/env python
"""FK20 benchmark: KZG proofs/s for 512 rows x 4096 coefficients on B200.

One step = all proofs of one batch: 512 polynomials of 4096 uniform seeded Fr
coefficients against one shared setup (tau^i G1, tau seeded), l = 16, 512
proofs per row (262,144 proofs).  Inputs are synthetic (seeded), resident in
HBM for `value`; `e2e` goes through the reference-facing C-ABI entry point
fk20_poly2h_fft with the polynomials copied from pinned host memory and the
proofs copied back, every step.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

With N > 1 (launched by torch.distributed.run) every rank proves its own 512
rows on its own GPU (weak scaling; rows are independent, no data-path
collective); the step time is the max over ranks.  `--impl reference` times
the reference algorithm's CPU path (FK20Py multi, restated in C: the oracle)
on the host cores, rank 0 only.
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
sys.path.insert(0, os.path.join(ROOT, "fk20-cuda_b200"))
sys.path.insert(0, os.path.join(ROOT, "oracle"))

R_MOD = 0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001
METRIC = "KZG proofs/s, 512 rows x 4096 coefs, bit-exact"
L = 16
# algorithmic products: Fp product = 300 limb products (12-limb Montgomery CIOS)
CLOCK_FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
                "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
                "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=("ours", "reference"), default="ours")
    ap.add_argument("--rows", type=int, default=512)
    ap.add_argument("--n", type=int, default=4096)
    ap.add_argument("--window", type=int, default=15,
                    help="table window of the 4096-coefficient tables (117 GB at 15); the 1024- and "
                         "2048-coefficient tables of the ragged and served loads use min(window, 13)")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--cpu-rows", type=int, default=0, help="rows per CPU sample (default: one per core)")
    ap.add_argument("--mode", choices=("batch", "serve", "ragged", "micro"), default="batch",
                    help="batch: the headline 512 x 4096 batch; serve: Poisson request load through the "
                         "continuous-batching server; ragged: 1000 mixed-length instances as one graph-captured batch; "
                         "micro: kernel microbenchmarks (Fp/Fr products, batched G1 FFT/IFFT, 16-term MSM)")
    ap.add_argument("--serve-seconds", type=float, default=8.0, help="arrival window per load level (serve)")
    ap.add_argument("--serve-warmup", type=float, default=1.0,
                    help="seconds of arrivals at the start of each level left out of the statistics (serve)")
    ap.add_argument("--serve-loads", default="0.5,0.8,0.9,1.2", help="offered load as fractions of plain-batch capacity")
    ap.add_argument("--serve-max-rows", type=int, default=160)
    ap.add_argument("--serve-slots", type=int, default=2)
    ap.add_argument("--serve-fft-blocks", type=int, default=0,
                    help="blocks per SM of each pack's persistent launch (0: by its number of products)")
    ap.add_argument("--serve-engine", type=int, default=0,
                    help="server engine: 0 packs on slots, 1 cohorts (continuous batching at FFT-stage granularity)")
    ap.add_argument("--serve-cohort-rows", type=int, default=0, help="engine 1: rows per cohort (0 = 64)")
    ap.add_argument("--serve-cohorts", type=int, default=0, help="engine 1: cohorts in flight (0 = 16)")
    ap.add_argument("--serve-form-ms", type=int, default=0, help="engine 1: longest partial-group wait (0 = 25)")
    ap.add_argument("--serve-stages", type=int, default=0, help="engine 1: FFT stages per launch (0 = 3)")
    ap.add_argument("--serve-max-queue", type=int, default=640,
                    help="waiting requests beyond which the server refuses submits with FK20_EAGAIN (overload "
                         "control; the client drops refused requests and counts them)")
    ap.add_argument("--serve-burst-rows", type=int, default=0,
                    help="pack size while more than 2 x max rows requests wait (0: 7/5 of max rows)")
    ap.add_argument("--serve-latency-rows", type=int, default=0,
                    help="latency-mode packs while at most this many requests wait (0: max rows)")
    ap.add_argument("--no-records", action="store_true",
                    help="batch mode at N = 1: skip the served-load and ragged-batch records of the line")
    ap.add_argument("--record-serve-seconds", type=float, default=6.0,
                    help="arrival window per load level of the served record (batch mode)")
    ap.add_argument("--record-serve-loads", default="0.5,0.8,0.9,1.2",
                    help="load levels of the served record, as fractions of plain-batch capacity (batch mode)")
    ap.add_argument("--autotune", action="store_true", help="autotune the context before timing (batch, ragged)")
    ap.add_argument("--msm-threads", type=int, default=0, help="MSM block size (64, 128, 256; 0 = the context's)")
    ap.add_argument("--tune-max-table-bytes", type=int, default=0,
                    help="table memory budget of the autotuner (0 = what the free device memory allows)")
    return ap.parse_args()


def workload_config(args, extra=None):
    cfg = {
        "workload": f"FK20 multi-proof batch: {args.rows} rows x {args.n} coefficients, l={L}, "
                    f"{2 * args.n // L} proofs/row, one shared setup",
        "rows": args.rows, "n": args.n, "l": L, "proofs_per_step": args.rows * 2 * args.n // L,
        "window_bits": args.window,
        "l2": "flushed between timed steps (256 MiB write); the MSM tables (GBs) exceed L2",
        "parallelism": f"rows-partitioned x{args.gpus} (replicated setup tables)",
    }
    if extra:
        cfg.update(extra)
    return cfg


# ------------------------------------------------------------------ distributed
def dist_init(args, backend: str = "nccl"):
    """One process per GPU (torchrun): NCCL on the GPU path; `gloo` runs the
    same host logic on the CPU (tests)."""
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if ws > 1:
        import datetime
        import torch
        import torch.distributed as dist
        if backend == "nccl":
            torch.cuda.set_device(local)
            # short: a rank that never reaches a collective ends the others' wait with an error
            dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=180),
                                    device_id=torch.device("cuda", local))
        else:
            dist.init_process_group(backend, timeout=datetime.timedelta(seconds=60))
    return ws, rank, local


def barrier(ws):
    if ws > 1:
        import torch.distributed as dist
        dist.barrier()


def max_over_ranks(x: float, ws: int) -> float:
    """The step time of the job: the slowest rank's (device-timed) time."""
    if ws == 1:
        return x
    import torch
    import torch.distributed as dist
    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([x], dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def load_other_lengths(ctx, args, n_main: int):
    """Tables of the 1024- and 2048-coefficient lengths (the ragged and served
    loads), at min(window, 13): with window 15 for 4096 (117 GB) all three
    lengths at 15 would not fit the device."""
    import fk20b200 as E
    main_w = ctx.get(E.FK20_OPT_WINDOW)
    ctx.set(E.FK20_OPT_WINDOW, min(main_w, 13))
    for n2 in (1024, 2048, 4096):
        if n2 != n_main:
            ctx.load_setup(n2, gpu_setup(E, n2))
    ctx.set(E.FK20_OPT_WINDOW, main_w)


def rank_rows_seed(rank: int) -> int:
    """Seed of a rank's polynomials: every rank proves its own rows (weak scaling)."""
    return 1000 + rank


def job_value(ws: int, proofs_per_rank: int, steps: int, total_ms: float) -> float:
    """Whole-job proofs/s: all ranks' proofs over the slowest rank's time."""
    return ws * proofs_per_rank * steps / (total_ms * 1e-3)


# ------------------------------------------------------------------ clocks
class ClockSampler:
    def __init__(self, dev: int):
        self.dev = dev
        self.proc = None
        import tempfile
        self.path = os.path.join(tempfile.gettempdir(), f"fk20_clocks_{os.getpid()}_{dev}.csv")

    def __enter__(self):
        try:
            self.f = open(self.path, "w")
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={CLOCK_FIELDS}", "--format=csv,noheader",
                                          "-lms", "200", "-i", str(self.dev)], stdout=self.f,
                                         stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None
        return self

    def __exit__(self, *a):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
            self.f.close()

    def summary(self):
        if self.proc is None or not os.path.exists(self.path):
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        mhz, maxs, reasons = [], [], set()
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        for line in open(self.path):
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                mhz.append(float(f[1].split()[0]))
                maxs.append(float(f[2].split()[0]))
            except ValueError:
                continue
            for nm, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(nm)
        os.unlink(self.path)
        return {"sm_mhz": statistics.median(mhz) if mhz else None, "sm_max_mhz": max(maxs) if maxs else None,
                "reasons": sorted(reasons), "samples": len(mhz)}


# ------------------------------------------------------------------ inputs
# Seeded synthetic inputs, generated here (the oracle is only the CPU
# baseline's and the reference arm's): uniform Fr values from a SplitMix64
# stream (4 draws per candidate, top limb masked to 63 bits, rejected if >= r;
# the same stream the tests draw), tau from the same generator.
P_MOD = 0x1A0111EA397FE69A4B1BA7B6434BACD764774B84F38512BF6730D2A0F6B0F6241EABFFFEB153FFFFB9FEFFFFFFFFAAAB
G1_X = 0x17F1D3A73197D7942695638C4FA9AC0FC3688C4F9774B905A14E3A3F171BAC586C55E83FF97A1AEFFB3AF00ADB22C6BB
G1_Y = 0x08B3F481E3AAA0F1A09E30ED741D8AE4FCF5E095D5D00AF600DB18CB2C04B3EDD03CC744A2888AE40CAA232946C5E7E1


def int_to_limbs(x: int, n: int):
    import numpy as np
    return np.array([(x >> (64 * k)) & 0xFFFFFFFFFFFFFFFF for k in range(n)], np.uint64)


def limbs_to_int(a) -> int:
    return sum(int(v) << (64 * k) for k, v in enumerate(a))


def g1_generator():
    """The BLS12-381 G1 generator as a reference g1p_t (x, y, 1), standard form."""
    import numpy as np
    return np.concatenate([int_to_limbs(G1_X, 6), int_to_limbs(G1_Y, 6), int_to_limbs(1, 6)])


def seeded_fr(seed: int, count: int):
    import numpy as np
    gamma, m1, m2 = np.uint64(0x9E3779B97F4A7C15), np.uint64(0xBF58476D1CE4E5B9), np.uint64(0x94D049BB133111EB)
    r_limbs = int_to_limbs(R_MOD, 4)
    out, have, j0 = [], 0, 0
    while have < count:
        need = int((count - have) * 1.12) + 64
        idx = np.arange(4 * j0, 4 * (j0 + need), dtype=np.uint64)
        with np.errstate(over="ignore"):
            z = np.uint64(seed) + (idx + np.uint64(1)) * gamma
            z = (z ^ (z >> np.uint64(30))) * m1
            z = (z ^ (z >> np.uint64(27))) * m2
            v = (z ^ (z >> np.uint64(31))).reshape(need, 4)
        v[:, 3] &= np.uint64(0x7FFFFFFFFFFFFFFF)
        lt, eq = np.zeros(need, bool), np.ones(need, bool)
        for k in (3, 2, 1, 0):
            lt |= eq & (v[:, k] < r_limbs[k])
            eq &= v[:, k] == r_limbs[k]
        acc = v[lt]
        out.append(acc[: count - have])
        have += min(len(acc), count - have)
        j0 += need
    return np.ascontiguousarray(np.concatenate(out)[:count])


def seeded_polys(seed: int, rows: int, n: int):
    return seeded_fr(seed, rows * n).reshape(rows, n, 4)


def seeded_tau(seed: int = 1) -> int:
    return limbs_to_int(seeded_fr(seed, 1)[0])


def gpu_setup(E, n: int, seed: int = 1):
    """setup s_i = tau^i G1 (i <= n) computed on the GPU (g1p_op_n scalar mul)."""
    import numpy as np
    tau = seeded_tau(seed)
    pw, acc = [], 1
    for _ in range(n + 1):
        pw.append(acc)
        acc = acc * tau % R_MOD
    scal = np.stack([int_to_limbs(x, 4) for x in pw])
    gen = np.repeat(g1_generator().reshape(1, 18), n + 1, 0)
    dgen, dscal = E.to_device(gen), E.to_device(scal)
    out = E.empty((n + 1, 18))
    E.call("g1p_op_n", E.G1_OPS["mul"], E._ptr(out), E._ptr(dgen), E._ptr(dscal), n + 1, E._stream())
    return out


def gpu_eq(E, a, b) -> bool:
    """a == b as G1 points (projective equality, on the GPU)."""
    import torch
    cnt = a.numel() // 18
    eq = torch.zeros(cnt, dtype=torch.uint8, device="cuda")
    # operands bound to names: a temporary passed only through its address
    # could be freed, and its memory reused, before the kernel reads it
    ac, bc = a.contiguous(), b.contiguous()
    E.call("g1p_eq_n", E._ptr(eq), E._ptr(ac), E._ptr(bc), cnt, E._stream())
    return int(eq.sum()) == cnt


# ------------------------------------------------------------------ our arm
def measure_imad_peak(E, torch):
    sink = torch.zeros(4, dtype=torch.int32, device="cuda")
    blocks, threads, iters = 148 * 8, 256, 4096
    E.call("fk20_bench_imad", E._ptr(sink), blocks, threads, 64, E._stream())
    best = 0.0
    for _ in range(3):
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        E.call("fk20_bench_imad", E._ptr(sink), blocks, threads, iters, E._stream())
        e.record()
        e.synchronize()
        best = max(best, blocks * threads * iters * 32 / (s.elapsed_time(e) * 1e-3))
    return best  # IMAD lane-instructions / s


def traffic_from_profiles(kind: str):
    p = os.path.join(ROOT, "profiles", "traffic.json")
    if os.path.exists(p):
        try:
            return json.load(open(p)).get(kind)
        except (OSError, ValueError):
            return None
    return None


def run_ours(args, ws, rank, dev):
    import numpy as np
    import torch
    import fk20b200 as E

    torch.cuda.set_device(dev)
    n, rows = args.n, args.rows
    m = 2 * n // L
    proofs = rows * m

    t0 = time.time()
    setup = gpu_setup(E, n)
    ctx = E.Context(dev, args.window)
    ctx.load_setup(n, setup)
    torch.cuda.synchronize()
    setup_s = time.time() - t0
    tune = None
    if args.msm_threads:
        ctx.set(E.FK20_OPT_MSM_THREADS, args.msm_threads)
    if args.autotune:  # window within the memory budget, MSM block size, FFT grid, fused vs staged
        t1 = time.time()
        tune = ctx.autotune(n, rows=min(rows, 512), max_table_bytes=args.tune_max_table_bytes)
        tune["tune_s"] = round(time.time() - t1, 1)

    poly_h = seeded_polys(rank_rows_seed(rank), rows, n)
    poly = E.to_device(poly_h)
    h_fft = E.empty((rows, m, 18))
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream()

    for _ in range(args.warmup):
        ctx.poly2h_fft(h_fft, poly, rows, n)
    torch.cuda.synchronize()

    # ---- timed region: device-resident inputs
    ctx.profile(True)
    barrier(ws)
    torch.cuda.synchronize()
    step_ms = []
    with ClockSampler(dev) as clk:
        for _ in range(args.steps):
            flush.fill_(1)
            s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            s.record(stream)
            ctx.poly2h_fft(h_fft, poly, rows, n)
            e.record(stream)
            e.synchronize()
            step_ms.append(s.elapsed_time(e))
    torch.cuda.synchronize()
    barrier(ws)
    prof = ctx.profile_read()
    prof_exe = ctx.profile_read_executed()
    ctx.profile(False)
    total_ms = max_over_ranks(sum(step_ms), ws)
    clocks = clk.summary()
    value = job_value(ws, proofs, args.steps, total_ms)

    # ---- roofline of the dominant kernel kind
    imad_peak = measure_imad_peak(E, torch)
    peak_products = imad_peak / 2  # a 32x32->64 product needs its lo and hi halves
    kind = max(prof, key=lambda k: prof[k][0])
    kms, klaunch, kalg = prof[kind]
    kprod = prof_exe[kind]
    achieved = (kprod / klaunch) / ((kms / klaunch) * 1e-3) if klaunch else 0.0
    all_ms = sum(v[0] for v in prof.values())
    all_prod = sum(prof_exe.values())
    launches = sum(v[1] for v in prof.values())
    roofline = {
        "bound": "imad", "kernel": f"k_proj ({kind})" if kind.startswith("stage") or kind == "middle" else kind,
        "achieved": achieved / 1e9, "peak": peak_products / 1e9, "unit": "Gprod/s",
        "frac": achieved / peak_products, "traffic": traffic_from_profiles(kind),
        "peak_source": "measured live: fk20_bench_imad (8 independent IMAD chains/thread), IMAD/s / 2",
        "whole_step": {"achieved": all_prod / (all_ms * 1e-3) / 1e9, "frac": all_prod / (all_ms * 1e-3) / peak_products},
        "per_kind_ms_per_step": {k: v[0] / args.steps for k, v in prof.items()},
        # every kernel kind against the same peak: executed products / its own launch time
        "per_kind_frac": {k: (prof_exe[k] / (v[0] * 1e-3)) / peak_products for k, v in prof.items() if v[0] > 0},
        "products_per_launch": kprod / klaunch if klaunch else None,
        "work_model": "limb products as the kernels execute them: Fp product 300, square 234 (triangular), Fr "
                      "product 136; XYZZ mixed additions, Jacobian programs, the projection plans' additions",
        # the same launches at the fixed unit costs (Fp product or square 300; G1 addition 12, mixed
        # addition 11, doubling 8 Fp products), the projection as the two radix-2 transforms it
        # replaces: products of that work per second, not the pipe's load
        "algorithmic": {
            "products_per_launch": kalg / klaunch if klaunch else None,
            "achieved": (kalg / (kms * 1e-3)) / 1e9 if kms else 0.0,
        },
    }
    if kind == "fft_fused" and klaunch:
        # the same launch against HBM: its algorithmic bytes are the point tiles
        # (rows x m points of 3 x 48 bytes) read once and written once
        hbm_peak, hbm_src = hbm_peak_gbs()
        tile_bytes = 2 * rows * m * 144
        hbm_achieved = tile_bytes / ((kms / klaunch) * 1e-3) / 1e9
        roofline["hbm"] = {"achieved": hbm_achieved, "peak": hbm_peak, "unit": "GB/s", "frac": hbm_achieved / hbm_peak,
                           "algorithmic_bytes_per_launch": tile_bytes, "peak_source": hbm_src}

    # ---- e2e: reference entry point, host buffers, copies inside the timed region
    e2e = None
    table_bytes = ctx.device_bytes()
    if not args.no_e2e:
        xext = E.empty((L, m, 18))
        E.call("fk20_setup2xext_fft", E._ptr(xext), E._ptr(setup), E._stream())
        # the reference-signature entry point keeps its own tables in a
        # process-wide default context: free this context's first (two sets
        # at window 15 would not fit), and the default context's afterwards
        torch.cuda.synchronize()
        ctx.close()
        ctx = None
        host_poly = torch.from_numpy(poly_h.view(np.int64)).pin_memory()
        host_out = torch.empty((rows, m, 18), dtype=torch.int64).pin_memory()
        dpoly = torch.empty_like(host_poly, device="cuda")
        dout = torch.empty((rows, m, 18), dtype=torch.int64, device="cuda")
        default = torch.cuda.default_stream()

        def e2e_step():
            dpoly.copy_(host_poly, non_blocking=True)
            E.call("fk20_poly2h_fft", E._ptr(dout), E._ptr(dpoly), E._ptr(xext), rows)
            host_out.copy_(dout, non_blocking=True)

        with torch.cuda.stream(default):
            for _ in range(max(1, args.warmup)):
                e2e_step()
            torch.cuda.synchronize()
            barrier(ws)
            e_ms = []
            for _ in range(args.steps):
                flush.fill_(1)
                s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                s.record(default)
                e2e_step()
                e.record(default)
                e.synchronize()
                e_ms.append(s.elapsed_time(e))
            barrier(ws)
        e_total = max_over_ranks(sum(e_ms), ws)
        # the e2e output is the same points as the device-resident run (projective equality)
        eq = torch.zeros(rows * m, dtype=torch.uint8, device="cuda")
        dchk = host_out.cuda()
        E.call("g1p_eq_n", E._ptr(eq), E._ptr(dchk), E._ptr(h_fft), rows * m, E._stream())
        same = int(eq.sum()) == rows * m
        torch.cuda.synchronize()
        E.call("fk20_default_release", dev)
        e2e = {"value": ws * proofs * args.steps / (e_total * 1e-3), "unit": "proofs/s",
               "h2d_bytes_per_step": rows * n * 32, "d2h_bytes_per_step": rows * m * 144,
               "ms_per_step": e_total / args.steps, "path": "C-ABI fk20_poly2h_fft (fk20_poly2h_fft.cu:47)",
               "output_matches_device_run": same}

    # ---- CPU baseline: the oracle (FK20Py restated in C) on the host cores
    cpu = ref_gpu = None
    if rank == 0 and ws == 1 and not args.no_cpu_baseline:
        import oracle as O
        cores = os.cpu_count() or 1
        srows = args.cpu_rows or cores
        xd = E.empty((L, m, 18))
        E.call("fk20_setup2xext_fft", E._ptr(xd), E._ptr(setup), E._stream())
        xh = E.to_host(xd)
        t = time.time()
        O.fk20_rows(poly_h[:srows], xh, L, cores)
        dt = time.time() - t
        cpu = {"value": srows * m / dt, "unit": "proofs/s", "cores": cores, "kind": "port",
               "sample": f"{srows} of the {rows} rows ({srows * m} proofs), {dt:.1f} s, one row per thread; "
                         "C restatement of FK20Py multi (variable-base double-and-add MSM, G1 FFT by scalar "
                         "multiplication), not py_ecc"}
        # the reference's GPU baseline: its own CUDA pipeline on the same batch
        ref_gpu = reference_gpu_same_batch(args, E, poly, xd, h_fft)
        del xd

    # ---- the rest of the metric at N = 1: the ragged batch and the served load
    ragged = served = None
    if ws == 1 and not args.no_records:
        del poly, h_fft
        if ctx is None:
            ctx = E.Context(dev, args.window)
            ctx.load_setup(n, setup)
        load_other_lengths(ctx, args, n)
        torch.cuda.synchronize()
        with ClockSampler(dev) as rclk:
            ragged = ragged_on(ctx, rank, 5, 3)
        ragged["clocks"] = rclk.summary()
        with ClockSampler(dev) as sclk:
            served = serve_on(args, ctx, rank, [float(x) for x in args.record_serve_loads.split(",")],
                              args.record_serve_seconds, 1.0, total_ms / args.steps)
        served["clocks"] = sclk.summary()

    line = {
        "metric": METRIC, "value": value, "unit": "proofs/s", "n_gpus": ws, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u32", "data": "synthetic (seeded uniform Fr, seeded tau)",
        "config": workload_config(args, {"setup_s": round(setup_s, 2),
                                         "table_bytes": table_bytes, "autotune": tune}),
        "e2e": e2e, "gpu_launches": launches, "roofline": roofline, "cpu_baseline": cpu, "clocks": clocks,
        "reference_gpu": ref_gpu, "ragged": ragged, "served": served, "impl": "ours",
    }
    if ctx is not None:
        ctx.close()
    return line


def hbm_peak_gbs():
    """The measured HBM copy bandwidth of this GPU pool (MEASURED_PEAKS.json at
    the repository root), else the earlier measurement of 6.65 TB/s."""
    try:
        with open(os.path.join(os.path.dirname(os.path.abspath(__file__)), "MEASURED_PEAKS.json")) as f:
            return float(json.load(f)["hbm_gbs"]), "measured (MEASURED_PEAKS.json hbm_gbs)"
    except (OSError, ValueError, KeyError):
        return 6650.0, "fallback (6.65 TB/s, earlier measurement)"


# ------------------------------------------------------------------ served load
SERVE_MIX = ((1024, 0.2), (2048, 0.3), (4096, 0.5))


def run_serve(args, ws, rank, dev):
    """Open-loop Poisson arrivals of blob-proof requests (1024/2048/4096
    coefficients, weights 0.2/0.3/0.5) at fractions of the measured plain-batch
    capacity, through the continuous-batching server (fk20_server_*); p50/p99
    latency (submit -> proofs in host memory) and sustained proofs/s beside the
    plain 512 x 4096 batch."""
    import torch
    import fk20b200 as E

    torch.cuda.set_device(dev)
    t0 = time.time()
    ctx = E.Context(dev, args.window)
    ctx.load_setup(4096, gpu_setup(E, 4096))
    load_other_lengths(ctx, args, 4096)
    torch.cuda.synchronize()
    setup_s = time.time() - t0
    # plain-batch capacity and latency: the full 512 x 4096 batch, device resident
    rows, n = args.rows, args.n
    poly = E.to_device(seeded_polys(1000 + rank, rows, n))
    h = E.empty((rows, 2 * n // L, 18))
    for _ in range(2):
        ctx.poly2h_fft(h, poly, rows, n)
    torch.cuda.synchronize()
    s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record()
    for _ in range(3):
        ctx.poly2h_fft(h, poly, rows, n)
    e.record()
    e.synchronize()
    plain_ms = s.elapsed_time(e) / 3
    del poly, h
    rec = serve_on(args, ctx, rank, [float(x) for x in args.serve_loads.split(",")], args.serve_seconds,
                   args.serve_warmup, plain_ms)
    sat = max(rec["loads"], key=lambda x: x["load"])
    line = {
        "metric": "served KZG proofs/s, mixed 1024/2048/4096 requests, bit-exact; p50/p99 latency",
        "value": sat["served_proofs_per_s"], "unit": "proofs/s", "n_gpus": ws, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u32", "mode": "serve",
        "data": "synthetic (seeded uniform Fr, seeded tau), open-loop Poisson arrivals",
    }
    line.update(rec)
    line["config"]["setup_s"] = round(setup_s, 2)
    line["impl"] = "ours"
    ctx.close()
    return line


def serve_on(args, ctx, rank, loads_frac, seconds, warmup_s, plain_ms):
    """The served load through a server on `ctx` (setups for 1024, 2048 and
    4096 loaded): Poisson arrivals at each fraction of the plain batch's
    capacity (512 x 4096 proofs in plain_ms), `seconds` of arrivals per level
    after `warmup_s` left out of the statistics; sampled results compared with
    the same polynomial proved alone."""
    import queue
    import threading
    import numpy as np
    import fk20b200 as E

    rows, n = args.rows, args.n
    plain_pps = rows * (2 * n // L) / (plain_ms * 1e-3)
    # request pool: seeded polynomials per length, reused round-robin
    pool = {n: [np.ascontiguousarray(p) for p in seeded_polys(5000 + n, 24, n)] for n, _ in SERVE_MIX}
    sizes = np.array([n for n, _ in SERVE_MIX])
    weights = np.array([w for _, w in SERVE_MIX])
    mean_proofs = float((sizes // 8 * weights).sum())
    srv = E.Server(ctx, max_rows=args.serve_max_rows, slots=args.serve_slots, fft_blocks_per_sm=args.serve_fft_blocks,
                   latency_rows=args.serve_latency_rows, burst_rows=args.serve_burst_rows,
                   max_queue=args.serve_max_queue, engine=args.serve_engine, cohort_rows=args.serve_cohort_rows,
                   cohorts=args.serve_cohorts, form_ms=args.serve_form_ms, stages_per_launch=args.serve_stages)
    loads = []
    rng = np.random.default_rng(42)
    check = []  # (n, pool index, output) kept for the bit-exactness check
    for frac in loads_frac:
        rate = frac * plain_pps / mean_proofs  # requests per second
        count = max(1, int(rate * (seconds + warmup_s)))
        gaps = rng.exponential(1.0 / rate, count)
        lens = rng.choice(sizes, count, p=weights)
        free = {int(n): [] for n in sizes}
        pending = queue.Queue()
        done_rc = []
        level_checks = []

        def collector():
            while True:
                item = pending.get()
                if item is None:
                    return
                t, nj, j, out = item
                done_rc.append(srv.wait(t, 120000))
                if len(level_checks) < 8 and j % 5 == 0:
                    level_checks.append((nj, j % 24, out))
                else:
                    free[nj].append(out)

        th = threading.Thread(target=collector)
        th.start()
        srv.reset_stats()
        start = time.perf_counter()
        due = start
        warm = warmup_s > 0
        lag = 0.0  # how far the client fell behind the arrival schedule
        refused = 0
        for j in range(count):
            if warm and due - start >= warmup_s:
                srv.reset_stats()  # steady state: later completions only
                warm = False
            due += gaps[j]
            d = due - time.perf_counter()
            if d > 0:
                time.sleep(d)
            nj = int(lens[j])
            out = free[nj].pop() if free[nj] else np.zeros((nj // 8, 18), np.uint64)
            lag = max(lag, time.perf_counter() - due)
            try:
                t = srv.submit(pool[nj][j % 24], out)
            except E.Fk20Error as err:
                if err.code != E.FK20_EAGAIN:
                    raise
                refused += 1  # overload: the queue is full; the request is dropped
                free[nj].append(out)
                continue
            pending.put((t, nj, j, out))
        submit_s = time.perf_counter() - start
        pending.put(None)
        th.join()
        st = srv.stats()
        check += level_checks
        loads.append({"load": frac, "requests": count, "offered_proofs_per_s": rate * mean_proofs,
                      "served_proofs_per_s": st["proofs_per_s"],
                      "served_vs_plain": st["proofs_per_s"] / plain_pps,
                      "p50_ms": st["p50_ms"], "p99_ms": st["p99_ms"], "mean_ms": st["mean_ms"],
                      "max_ms": st["max_ms"], "p99_below_plain_batch_latency": st["p99_ms"] < plain_ms,
                      "mean_pack_rows": st["mean_pack_rows"], "packs": st["packs"],
                      # where the latency goes: waiting for a pack, staging it, running it
                      "mean_wait_ms": st["mean_wait_ms"], "mean_enqueue_ms": st["mean_enqueue_ms"],
                      "mean_run_ms": st["mean_run_ms"], "mean_msm_ms": st["mean_msm_ms"],
                      "mean_launch_ms": st["mean_launch_ms"], "launches": st["launches"],
                      "errors": sum(1 for r in done_rc if r != 0),
                      # admission: submits refused with FK20_EAGAIN (max_queue requests waiting)
                      "admitted": count - refused, "refused": refused,
                      # the load generator itself: requests/s it achieved against the schedule's
                      "arrivals_per_s": {"offered": rate, "achieved": count / submit_s},
                      "client_max_lag_ms": lag * 1e3})
    srv.close()
    # served results are the ones the same polynomial gives alone
    same = True
    for nj, j, out in check:
        hh = E.empty((1, nj // 8, 18))
        ctx.poly2h_fft(hh, E.to_device(pool[nj][j].reshape(1, nj, 4)), 1, nj)
        same &= bool(np.array_equal(E.to_host(hh)[0], out))
    return {
        "config": {"workload": "served load: Poisson arrivals of 1024/2048/4096-coefficient requests "
                               "(weights 0.2/0.3/0.5) at fractions of plain-batch capacity",
                   "window_bits": {"4096": args.window, "1024/2048": min(args.window, 13)},
                   "max_rows_per_pack": args.serve_max_rows,
                   "slots": args.serve_slots, "fft_blocks_per_sm": args.serve_fft_blocks or "adaptive",
                   "latency_rows": args.serve_latency_rows or args.serve_max_rows,
                   "burst_rows": args.serve_burst_rows or min(4096, args.serve_max_rows * 7 // 5),
                   "max_queue": args.serve_max_queue,
                   "engine": "cohorts" if args.serve_engine == 1 else "packs on slots",
                   "cohort": {"rows": args.serve_cohort_rows or 64, "in_flight": args.serve_cohorts or 16,
                              "form_ms": args.serve_form_ms or 25, "stages_per_launch": args.serve_stages or 3}
                   if args.serve_engine == 1 else None,
                   "arrival_window_s": seconds, "warmup_s_excluded": warmup_s,
                   "table_bytes": ctx.device_bytes()},
        "plain_batch": {"rows": rows, "n": n, "proofs_per_s": plain_pps, "latency_ms": plain_ms},
        "loads": loads,
        # load levels that serve >= 80 % of plain-batch proofs/s with p99 below the plain batch's latency
        "loads_at_80pct_with_p99_below_plain": [x["load"] for x in loads
                                                 if x["served_vs_plain"] >= 0.8 and x["p99_below_plain_batch_latency"]],
        "results_same_alone_and_served": same, "checked_requests": len(check),
    }


# ------------------------------------------------------------------ ragged batch (graph)
def run_ragged(args, ws, rank, dev):
    """1000 FK20 instances, lengths uniform over {1024, 2048, 4096}, one shared
    setup: one ragged batch (one MSM launch + one persistent G1 FFT launch over
    the three lengths) captured once in a CUDA graph and replayed; checked
    against the plain per-length path."""
    import torch
    import fk20b200 as E

    torch.cuda.set_device(dev)
    ctx = E.Context(dev, args.window)
    ctx.load_setup(4096, gpu_setup(E, 4096))
    load_other_lengths(ctx, args, 4096)
    tune = None
    if args.autotune:
        tune = ctx.autotune(4096, rows=128, max_table_bytes=0)
    rec = ragged_on(ctx, rank, args.steps, args.warmup, ws)
    line = {
        "metric": "KZG proofs/s, ragged batch of 1000 instances (1024/2048/4096), bit-exact",
        "value": rec.pop("value"), "unit": "proofs/s", "n_gpus": ws,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": rec.pop("ms_per_step"), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u32", "mode": "ragged",
        "data": "synthetic (seeded uniform Fr, seeded tau)",
    }
    line.update(rec)
    line["config"]["window_bits"] = {"4096": args.window, "1024/2048": min(args.window, 13)}
    line["autotune"] = tune
    line["impl"] = "ours"
    ctx.close()
    return line


def ragged_on(ctx, rank, steps, warmup, ws=1):
    """The ragged batch on `ctx` (setups for 1024, 2048 and 4096 loaded): 1000
    instances as one CUDA-graph plan, `steps` timed replays (L2 flushed between
    them), then the graph output against a direct call and the per-length
    plain path."""
    import numpy as np
    import torch
    import fk20b200 as E

    rng = np.random.default_rng(77 + rank)
    sizes = [int(x) for x in rng.choice([1024, 2048, 4096], 1000)]
    poly_off, out_off, po, oo = [], [], 0, 0
    for n in sizes:
        poly_off.append(po)
        out_off.append(oo)
        po += n
        oo += n // 8
    polys = E.to_device(seeded_fr(31 + rank, po))
    out = E.empty((oo, 18))
    plan = E.Plan(ctx, out, polys, sizes, poly_off, out_off)
    for _ in range(warmup):
        plan.launch()
    torch.cuda.synchronize()
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    barrier(ws)
    ms = []
    stream = torch.cuda.current_stream()
    for _ in range(steps):
        flush.fill_(1)
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record(stream)
        plan.launch()
        e.record(stream)
        e.synchronize()
        ms.append(s.elapsed_time(e))
    barrier(ws)
    total = max_over_ranks(sum(ms), ws)
    # direct (non-graph) call and the per-length plain path give the same proofs
    direct = E.empty((oo, 18))
    ctx.batch(direct, polys, sizes, poly_off, out_off)
    exp = E.empty((oo, 18))
    for n in (1024, 2048, 4096):
        idx = [j for j, s_ in enumerate(sizes) if s_ == n]
        rows = torch.stack([polys[poly_off[j]:poly_off[j] + n] for j in idx])
        h = E.empty((len(idx), n // 8, 18))
        ctx.poly2h_fft(h, rows, len(idx), n)
        for r, j in enumerate(idx):
            exp[out_off[j]:out_off[j] + n // 8] = h[r]
    torch.cuda.synchronize()
    rec = {
        "value": ws * oo * steps / (total * 1e-3), "ms_per_step": total / steps, "steps": steps, "warmup": warmup,
        "config": {"workload": "1000 FK20 instances, lengths uniform over {1024, 2048, 4096}, one CUDA-graph "
                               "replay per step", "proofs_per_step": oo,
                   "instances": {str(n): sizes.count(n) for n in (1024, 2048, 4096)},
                   "l2": "flushed between timed steps (256 MiB write)"},
        "graph_equals_direct": bool(torch.equal(out, direct)), "equals_per_length_path": bool(torch.equal(out, exp)),
    }
    plan.close()
    return rec


# ------------------------------------------------------------------ kernel microbenchmarks
# limb products per Fp product (12-limb CIOS; an Fp square counts as a product
# in the algorithmic work), Fp square as executed (triangular), Fr product
MP, MS, MR = 300, 234, 136


def _timed(fn, reps, stream):
    import torch
    fn()
    torch.cuda.synchronize()
    best = None
    for _ in range(reps):
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record(stream)
        fn()
        e.record(stream)
        e.synchronize()
        t = s.elapsed_time(e)
        best = t if best is None else min(best, t)
    return best


def run_micro(args, ws, rank, dev):
    """2^24 independent Fp and Fr Montgomery products and squarings on uniform
    seeded residues; 512-point G1 FFT and IFFT over 512 rows of seeded
    multiples of G1; the 512 x 16-term fixed-base MSM with uniform scalars;
    proofs in the data-availability format; KZG commitments.  Each output is
    checked on a sample through an independent path (Python integers, the
    engine's double-and-add point operations, FFT round trips); the parity
    tests check the same kernels against the oracle.  Each kernel is reported
    against the IMAD roofline (limb products/s over the measured IMAD peak / 2)."""
    import numpy as np
    import torch
    import fk20b200 as E

    torch.cuda.set_device(dev)
    stream = torch.cuda.current_stream()
    peak = measure_imad_peak(E, torch) / 2
    out = {}
    # ---- field products: limb-major Montgomery data, `iters` dependent products per element
    count, iters = 1 << 24, 64
    rng = np.random.default_rng(3)
    for field, mod, nl, mp, ms_ in (("fp", P_MOD, 12, MP, MS), ("fr", R_MOD, 8, MR, MR)):
        words = rng.integers(0, 2**32, (nl, count), dtype=np.uint64).astype(np.uint32)
        words[nl - 1] &= np.uint32((1 << (mod.bit_length() - 32 * (nl - 1) - 1)) - 1)  # < 2^(bits-1) < mod
        d0 = torch.from_numpy(words.view(np.int32)).cuda()
        for sq in (0, 1):
            d = d0.clone()
            ms = _timed(lambda: E.call("fk20_bench_field", 0 if field == "fp" else 1, sq, E._ptr(d), count, iters,
                                       E._stream()), 3, stream)
            # bit-exactness on a sample: one more run from the same input, against pow() over the integers
            d = d0.clone()
            E.call("fk20_bench_field", 0 if field == "fp" else 1, sq, E._ptr(d), count, iters, E._stream())
            got = d.cpu().numpy().view(np.uint32)
            Rm = pow(2, 32 * nl, mod)
            Ri = pow(Rm, mod - 2, mod)
            ok = True
            for e in range(0, count, count // 16):
                X = sum(int(words[k, e]) << (32 * k) for k in range(nl))
                x = X * Ri % mod
                y = pow(x, 2 ** iters, mod) if sq else pow(x, iters + 1, mod)
                G = sum(int(got[k, e]) << (32 * k) for k in range(nl))
                ok &= G == y * Rm % mod
            prod = count * iters * mp
            exe = count * iters * (ms_ if sq else mp)
            out[f"{field}_{'sqr' if sq else 'mul'}"] = {
                "elements": count, "products_per_element": iters, "ms": ms,
                "gmul_per_s": count * iters / (ms * 1e-3) / 1e9,
                "achieved_gprod_s": prod / (ms * 1e-3) / 1e9, "frac": prod / (ms * 1e-3) / peak,
                "executed_frac": exe / (ms * 1e-3) / peak, "bit_exact_sample": ok}
    # ---- G1 FFT / IFFT, 512 rows x 512 points
    rows, m = 512, 512
    gen = E.to_device(np.repeat(g1_generator().reshape(1, 18), rows * m, 0))
    scal = E.to_device(seeded_fr(21, rows * m))
    pts = E.empty((rows, m, 18))
    E.call("g1p_op_n", E.G1_OPS["mul"], E._ptr(pts), E._ptr(gen), E._ptr(scal), rows * m, E._stream())
    del gen, scal
    res = E.empty((rows, m, 18))
    back = E.empty((rows, m, 18))
    for name, inv in (("g1_fft", 0), ("g1_ift", 1)):
        ms = _timed(lambda: E.call("g1p_fft_n", E._ptr(res), E._ptr(pts), 9, rows, inv, E._stream()), 3, stream)
        # round trip through the other direction gives the input back
        E.call("g1p_fft_n", E._ptr(back), E._ptr(res), 9, rows, 1 - inv, E._stream())
        out[name] = {"rows": rows, "m": m, "ms": ms,
                     "round_trip_exact": gpu_eq(E, back, pts)}
    del pts, res, back
    # ---- 16-term fixed-base MSM: tc_fft[512][16][512] uniform Fr -> hext_fft[512][512]
    n = 4096
    setup = gpu_setup(E, n)
    xext = E.empty((L, m, 18))
    E.call("fk20_setup2xext_fft", E._ptr(xext), E._ptr(setup), E._stream())
    ctx = E.Context(dev, args.window)
    ctx.load_xext_fft(n, xext)
    tc = seeded_fr(22, rows * L * m).reshape(rows, L, m, 4)
    dtc = E.to_device(tc)
    hext = E.empty((rows, m, 18))
    ctx.profile(True)
    ms = _timed(lambda: ctx.msm(hext, dtc, rows, n), 3, stream)
    prof, prof_exe = ctx.profile_read(), ctx.profile_read_executed()
    ctx.profile(False)
    kms, kl, kprod = prof["msm"]
    # sample columns recomputed by double-and-add on the GPU (g1p_op_n), summed term by term
    ok = True
    for r in (0, rows - 1):
        for c in range(4):
            terms = E.empty((L, 18))
            bases, scalars = xext[:, c].contiguous(), dtc[r, :, c].contiguous()
            E.call("g1p_op_n", E.G1_OPS["mul"], E._ptr(terms), E._ptr(bases), E._ptr(scalars), L, E._stream())
            acc = terms[0:1].clone()
            for i in range(1, L):
                term = terms[i:i + 1]
                E.call("g1p_op_n", E.G1_OPS["add"], E._ptr(acc), E._ptr(acc), E._ptr(term), 1, E._stream())
            ok &= gpu_eq(E, acc, hext[r, c:c + 1])
    out["msm"] = {"rows": rows, "columns": m, "terms": L, "window_bits": args.window, "ms": ms,
                  "kernel_ms": kms / kl, "achieved_gprod_s": kprod / kl / (kms / kl * 1e-3) / 1e9,
                  "frac": kprod / kl / (kms / kl * 1e-3) / peak,
                  "executed_frac": prof_exe["msm"] / kl / (kms / kl * 1e-3) / peak, "bit_exact_sample": ok}
    # ---- proofs in the data-availability wire format, straight from the tiles
    poly = E.to_device(seeded_polys(1000, rows, n))
    proofs = torch.zeros((rows, m, 48), dtype=torch.uint8, device="cuda")
    h = E.empty((rows, m, 18))
    t_h = _timed(lambda: ctx.poly2h_fft(h, poly, rows, n), 2, stream)
    t_p = _timed(lambda: ctx.poly2proofs(proofs, poly, rows, n), 2, stream)
    via_h = torch.zeros_like(proofs)
    E.call("fk20_h_fft2proofs", E._ptr(via_h), E._ptr(h), rows, n, E._stream())
    out["da_proofs"] = {"rows": rows, "n": n, "ms_h_fft": t_h, "ms_da_proofs": t_p,
                        "proofs_per_s": rows * m / (t_p * 1e-3), "overhead": t_p / t_h - 1.0,
                        "same_as_converting_h_fft": bool(torch.equal(proofs, via_h))}
    ctx.close()
    del h, proofs
    # ---- KZG commitments: 512 polynomials x 4096 coefficients, window 10 tables over the setup
    cw = min(args.window, 10)
    cctx = E.Context(dev, args.window)
    cctx.load_commit(n, setup[:n], cw)
    com = E.empty((rows, 18))
    cctx.profile(True)
    t_c = _timed(lambda: cctx.commit(com, poly, rows, n), 3, stream)
    cms, cl, cprod = cctx.profile_read()["msm"]
    cctx.profile(False)
    tau = seeded_tau(1)
    p0 = [limbs_to_int(x) for x in E.to_host(poly[0])]
    f_tau = 0
    for c_ in reversed(p0):
        f_tau = (f_tau * tau + c_) % R_MOD
    exp_c = E.empty((1, 18))
    dgen, dft = E.to_device(g1_generator().reshape(1, 18)), E.to_device(int_to_limbs(f_tau, 4).reshape(1, 4))
    E.call("g1p_op_n", E.G1_OPS["mul"], E._ptr(exp_c), E._ptr(dgen), E._ptr(dft), 1, E._stream())
    out["commit"] = {"rows": rows, "n": n, "window_bits": cw, "ms": t_c, "commitments_per_s": rows / (t_c * 1e-3),
                     "achieved_gprod_s": cprod / cl / (cms / cl * 1e-3) / 1e9,
                     "frac": cprod / cl / (cms / cl * 1e-3) / peak,
                     "row0_equals_f_tau_G1": gpu_eq(E, com[0:1], exp_c)}
    cctx.close()
    line = {"metric": "kernel microbenchmarks: fraction of the IMAD roofline, bit-exact samples",
            "value": min(v["frac"] for v in out.values() if "frac" in v), "unit": "min frac of IMAD roofline",
            "n_gpus": ws, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u32",
            "mode": "micro", "data": "synthetic (seeded uniform residues, seeded multiples of G1)",
            "config": {"workload": "2^24 Fp/Fr mul and sqr; 512 x 512-point G1 FFT/IFFT; 512 x 16-term MSM; "
                                   "512 x 4096 proofs in the DA wire format; 512 x 4096-term commitments",
                       "imad_peak_gprod_s": peak / 1e9}, "kernels": out, "impl": "ours"}
    return line


# ------------------------------------------------------------------ reference arm
def run_reference(args, ws, rank):
    """The reference's CPU path for this workload -- FK20Py multi
    (FK20Py/fk20_multi_cuda.py:67-246), whose py_ecc dependency is absent here,
    restated in C (oracle/fk20_oracle.c) -- on all host cores, each step a
    bounded sample of the 512 x 4096 batch."""
    import numpy as np
    import oracle as O
    n = args.n
    m = 2 * n // L
    cores = os.cpu_count() or 1
    srows = args.cpu_rows or cores
    tau = O.seeded_fr(1, 1)[0]
    setup = O.setup(tau, n + 1, cores)
    xext = O.xext_fft(setup, n, L, cores)
    poly = seeded_polys(1000, srows, n)
    for _ in range(args.warmup):
        O.fk20_rows(poly[:min(srows, cores)], xext, L, cores)
    step = []
    for _ in range(args.steps):
        t = time.time()
        O.fk20_rows(poly, xext, L, cores)
        step.append(time.time() - t)
    tot = sum(step)
    value = srows * m * args.steps / tot
    ref_gpu = reference_gpu_leg(args, xext, cores)
    return {
        "metric": METRIC, "value": value, "unit": "proofs/s", "n_gpus": ws, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": tot * 1e3 / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u64", "data": "synthetic (seeded uniform Fr, seeded tau)",
        "config": workload_config(args, {"cpu_sample_rows_per_step": srows}),
        "impl": "reference",
        "cpu_baseline": {"value": value, "unit": "proofs/s", "cores": cores, "kind": "port",
                         "sample": f"{srows} rows x {n} coefficients per step ({srows * m} proofs) on {cores} "
                                   "threads; FK20Py multi restated in C (py_ecc absent)"},
        "e2e": {"value": value, "unit": "proofs/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "reference_gpu": ref_gpu,
    }


def _ref_gpu_lib():
    """The unmodified reference library (oracle/_ref/libfk20ref.so, built from
    its sources for sm_100a by oracle/ref/Makefile), or the reason it cannot run."""
    lib_path = os.path.join(ROOT, "oracle", "_ref", "libfk20ref.so")
    if not os.path.exists(lib_path):
        return None, "reference library not built (oracle/ref/Makefile)"
    try:
        import torch
        if not torch.cuda.is_available():
            return None, "no CUDA device"
    except ImportError:
        return None, "torch not importable"
    import ctypes
    return ctypes.CDLL(lib_path, mode=os.RTLD_LOCAL), None


def _ref_gpu_time(lib, dpoly, dxext, rows, steps):
    """fk20_poly2h_fft of the reference on device buffers, timed with CUDA
    events around the call as fk20benchmark.cu:103-116 does: one warm-up call,
    then `steps` timed calls.  Returns (per-call ms list, output, error code)."""
    import ctypes
    import torch
    m = 2 * 4096 // L
    out = torch.zeros((rows, m, 18), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()  # the reference runs on the legacy default stream: nothing else in flight
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    ms = ctypes.c_float(0)
    rc = lib.ref_fk20_time(P(out), P(dpoly), P(dxext), ctypes.c_uint(rows), ctypes.byref(ms))  # warm-up
    times = []
    for _ in range(steps):
        if rc:
            break
        rc = lib.ref_fk20_time(P(out), P(dpoly), P(dxext), ctypes.c_uint(rows), ctypes.byref(ms))
        times.append(ms.value)
    return times, out, rc


REF_GPU_PATH = ("reference fk20_poly2h_fft (fk20_poly2h_fft.cu:47-78), reference kernels compiled for sm_100a; "
                "double-and-add fk20_msm, g1p_ift/g1p_fft wrappers")


def reference_gpu_leg(args, xext, cores):
    """The reference's own CUDA pipeline on this GPU, beside its CPU path: the
    unmodified reference library runs fk20_poly2h_fft (rows <= 512, l = 16,
    n = 4096) on the same seeded batch as this benchmark's own arm.  Two rows
    of its output are checked against the oracle."""
    import numpy as np
    import torch
    if args.n != 4096 or args.rows > 512:
        return {"unavailable": "the reference pipeline is fixed at n = 4096 and at most 512 rows"}
    lib, why = _ref_gpu_lib()
    if lib is None:
        return {"unavailable": why}
    import oracle as O
    rows = args.rows
    poly = seeded_polys(1000, rows, args.n)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.int64)).cuda()
    steps = max(1, min(args.steps, 3))
    times, out, rc = _ref_gpu_time(lib, dev(poly), dev(xext), rows, steps)
    if rc:
        return {"unavailable": f"reference pipeline returned CUDA error {rc}"}
    h = out.cpu().numpy().view(np.uint64)
    check = [0, rows - 1]
    exp = O.fk20_rows(poly[check], xext, L, cores)
    same = all(np.array_equal(O.g1_normalize(h[r]), e) for r, e in zip(check, exp))
    tot = sum(times)
    return {"ms_per_step": tot / steps, "proofs_per_s": rows * (2 * args.n // L) * steps / (tot * 1e-3),
            "steps": steps, "rows": rows, "n": args.n, "rows_checked_against_oracle": check,
            "same_as_oracle": same, "path": REF_GPU_PATH}


def reference_gpu_same_batch(args, E, poly, xext, h_fft):
    """The reference's own CUDA pipeline run on the very batch this arm timed
    (same polynomials, same xext_fft, device-resident), outside every timed
    region, with each of its proofs compared with the engine's on the device
    (projective equality): the GPU-to-GPU comparison beside the CPU baseline."""
    import torch
    if args.n != 4096 or args.rows > 512:
        return {"unavailable": "the reference pipeline is fixed at n = 4096 and at most 512 rows"}
    lib, why = _ref_gpu_lib()
    if lib is None:
        return {"unavailable": why}
    rows = args.rows
    steps = max(1, min(args.steps, 3))
    times, out, rc = _ref_gpu_time(lib, poly.view(torch.int64), xext.view(torch.int64), rows, steps)
    if rc:
        return {"unavailable": f"reference pipeline returned CUDA error {rc}"}
    same = gpu_eq(E, out.view(torch.uint64), h_fft)
    tot = sum(times)
    m = 2 * args.n // L
    return {"ms_per_step": tot / steps, "proofs_per_s": rows * m * steps / (tot * 1e-3), "steps": steps,
            "rows": rows, "n": args.n, "all_proofs_equal_engine": same, "proofs_compared": rows * m,
            "path": REF_GPU_PATH}


def main():
    args = parse()
    # the reference-signature entry points (the e2e leg) use the same table window
    os.environ.setdefault("FK20_WINDOW", str(args.window))
    if args.impl == "reference":
        # CPU arm: rank 0 alone works and prints; other ranks exit without work
        rank = int(os.environ.get("RANK", "0"))
        if rank == 0:
            print(json.dumps(run_reference(args, int(os.environ.get("WORLD_SIZE", "1")), rank)), flush=True)
        return
    ws, rank, local = dist_init(args)
    if args.mode == "serve":
        line = run_serve(args, ws, rank, local)
    elif args.mode == "ragged":
        line = run_ragged(args, ws, rank, local)
    elif args.mode == "micro":
        line = run_micro(args, ws, rank, local)
    else:
        line = run_ours(args, ws, rank, local)
    if rank == 0:
        print(json.dumps(line), flush=True)
    if ws > 1:
        import torch.distributed as dist
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
