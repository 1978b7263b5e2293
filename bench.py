#!/usr/bin/env python
"""bench.py -- Mzone-updates/s at 256^3 including self-gravity.

Workload (default): the 256^3 stellar explosion -- n=3 Lane-Emden star
(M=1, R=0.4, gamma 5/3) of the reference's STELLAR_OCTANT_EXPLOSION_3D set-up,
1% log-normal density noise from the reference's seeded LCG, thermal energy
1.0 inside r < 0.02 R, multipole boundary to l=8, every step's Poisson solve
to the 1e-8 update norm -- centred in [-0.75, 0.75]^3 with outflow faces
(the octant layout's cell size).  In the octant layout the symmetry planes
cut through the star and the l=8 boundary expansion diverges there.  Inputs
are generated on the host (synthetic, seeded) and uploaded once; W warm-up
steps (the first one includes the cold-start Poisson solve) are followed by K
timed steps.

One step = one godunov_step_3d of the reference (hydro_solver_3d.c:637-811):
gravity solve, CFL dt, fused flux/update/source, boundaries.

Arms:
  (default)          this library's fastest configuration (FP32 hydro, mixed
                     precision Poisson, learned warm start when weights exist)
  --variant fp64     the FP64 path: the reference's sweeps, stop rule and
                     operation order in FP64 (bit-identical to the reference
                     where the reference has the same boundary; the l=8
                     multipole moments here are summed in a fixed tree order)
  --impl reference   the reference's own C code (oracle/_ref, built from the
                     reference sources) on the host CPU, one core (it is
                     serial), on a bounded sample of each step

Multi-GPU: the step does not shard (one grid per GPU in the reference), so
--gpus N runs N independent replicas, one per rank; value = zones all ranks
updated / max over ranks of the device time.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "Mzone-updates/s at 256^3 incl. gravity"
UNIT = "Mzone-updates/s"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--variant", default="best", choices=["best", "fp32_unet", "fp32", "fp64", "fp64_tree"])
    # --grid: the same option under a name that no torchrun option starts with
    ap.add_argument("--n", "--grid", dest="n", type=int, default=256, help="grid cells per side")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-fp64-compare", action="store_true")
    ap.add_argument("--unet-passes", type=int, default=1, help="learned-start predictions per solve")
    ap.add_argument("--unet-weights", default=None, help="weight file of the learned start (default: the committed one)")
    ap.add_argument("--sor-depth", type=int, default=None,
                    help="FP32 correction sweeps: 0 per-colour split sweeps, -2 two iterations per pass")
    ap.add_argument("--no-fp32-compare", action="store_true",
                    help="skip the FP32 arm without the learned warm start")
    ap.add_argument("--start-step", type=int, default=0,
                    help="a late window: advance the workload this many steps (FP32 + learned start, untimed) "
                         "and start every arm from that state")
    ap.add_argument("--record-fp64-iterations", default=None, metavar="PATH",
                    help="with --variant fp64: write the per-step SOR iteration counts to this JSON file "
                         "(the reference arm reads hydrocode_astro1_b200/data/fp64_iterations.json)")
    return ap.parse_args()


# ---------------------------------------------------------------- clocks
class Clocks:
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        self.p = None

    def start(self):
        try:
            self.p = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.Q}",
                                       "--format=csv,noheader,nounits", "-lms", "200"],
                                      stdout=self.f, stderr=subprocess.DEVNULL)
        except Exception:
            self.p = None

    def stop(self):
        if self.p is None:
            return None
        self.p.terminate()
        try:
            self.p.wait(timeout=5)
        except Exception:
            self.p.kill()
        self.f.flush()
        self.f.seek(0)
        rows = [r.split(",") for r in self.f.read().strip().splitlines() if r.strip()]
        os.unlink(self.f.name)
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in rows:
            try:
                sm.append(float(r[1]))
                mx = float(r[2])
                for nm, v in zip(names, r[5:9]):
                    if v.strip().lower() == "active":
                        reasons.add(nm)
            except (ValueError, IndexError):
                continue
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm)}


# ---------------------------------------------------------------- helpers
def dist_setup(args):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    dist = None
    if world > 1:
        import datetime

        import torch
        import torch.distributed as dist
        # NCCL on the GPU box; gloo where there is no GPU (the CPU tests of
        # this plumbing).  Every rank runs the same arms, so ranks wait on one
        # another only for seconds: a short timeout turns a lost rank into an
        # error instead of a hang.
        backend = "nccl" if torch.cuda.is_available() else "gloo"
        if backend == "nccl":
            torch.cuda.set_device(local)
        dist.init_process_group(backend, timeout=datetime.timedelta(seconds=120))
    return world, rank, local, dist


def reduce_max(dist, v):
    if dist is None:
        return v
    import torch
    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([v], dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def barrier(dist):
    if dist is not None:
        dist.barrier()


def make_workload(n):
    from hydrocode_astro1_b200 import problems
    return problems.stellar_explosion(n)


def solver_kwargs(p, variant, device):
    import hydrocode_astro1_b200 as hc
    kw = dict(lo=p["lo"], hi=p["hi"], gamma=p["gamma"], G=p["G"], bc=p["bc"], lmax=p["lmax"],
              cfl=p["cfl"], tol=1e-8, max_iter=2_000_000, omega=1.5, device=device)
    if SOR_DEPTH is not None and not variant.startswith("fp64"):
        kw["sor_depth"] = SOR_DEPTH
    if variant == "fp64":
        kw.update(precision=hc.FP64, lmax=p["lmax"], moment_order=hc.MOMENTS_TREE)
    elif variant == "fp64_tree":
        kw.update(precision=hc.FP64, moment_order=hc.MOMENTS_TREE)
    elif variant == "fp32_unet":
        kw.update(precision=hc.FP32, moment_order=hc.MOMENTS_TREE, warm_start=hc.HC_WARM_UNET)
    else:
        kw.update(precision=hc.FP32, moment_order=hc.MOMENTS_TREE)
    return kw


# Weights of the warm-start U-Net, trained on the GPU by
# `python -m hydrocode_astro1_b200.train_unet` from solves of this workload
# with another density-noise seed (7); the benchmark run uses seed 42.
UNET_WEIGHTS = os.path.join(ROOT, "hydrocode_astro1_b200", "data", "unet_stellar_explosion_256.bin")
SOR_DEPTH = None   # FP32 correction sweep mode (library default when None)
UNET_PASSES = 1
UNET_GUARD = 3     # learned-start outcome monitor: consecutive losses that switch it off


def make_solver(p, variant, device):
    import hydrocode_astro1_b200 as hc
    s = hc.HydroSolver3D(p["shape"], **solver_kwargs(p, variant, device))
    if variant == "fp32_unet":
        s.unet_load_file(UNET_WEIGHTS)
        s.unet_passes(UNET_PASSES)
        s.unet_guard(UNET_GUARD)
    return s


def advance(q0, p, nsteps, device):
    """The workload's state after `nsteps` steps of the FP32 path with the
    learned start (without it when no weight file exists), untimed: the
    starting state of a late window.  Returns (state, time reached)."""
    variant = "fp32_unet" if os.path.exists(UNET_WEIGHTS) else "fp32"
    s = make_solver(p, variant, device)
    s.set_state(q0)
    t = 0.0
    for k in range(nsteps):
        t += float(s.step(1)[0])
        if (k + 1) % 100 == 0:
            log(f"[bench] advancing: step {k + 1} of {nsteps}, t = {t:.5f}")
    q = s.state()
    s.close()
    return q, t


def run_variant(q0, p, variant, steps, warmup, device, dist, clocks=None):
    """Warm up, then time `steps` steps with CUDA events on the solver's stream."""
    s = make_solver(p, variant, device)
    s.set_state(q0)
    cons0 = s.conservation()      # FP64 totals formed on the device
    warm_iters = []
    for w in range(warmup):
        t = time.perf_counter()
        s.step(1)
        warm_iters.append(s.diagnostics()["last_iterations"])
        log(f"[bench] {variant} warm-up step {w}: {time.perf_counter() - t:.3f} s, "
            f"{warm_iters[-1]} SOR iterations")
    warm_launches = s.timing(reset=True)["launches"]
    diag0 = s.diagnostics()
    iters = []
    barrier(dist)
    s.sync()
    if clocks:
        clocks.start()
    nvtx = nvtx_mod()
    if nvtx:
        nvtx.range_push("timed")     # lets `ncu --nvtx --nvtx-include timed/` list the timed launches
    s.timer_start()
    dts = []
    d0 = s.diagnostics()["total_iterations"]
    for _ in range(steps):
        dts.append(float(s.step(1)[0]))
        iters.append(s.diagnostics()["last_iterations"])
    ms = s.timer_stop()
    if nvtx:
        nvtx.range_pop()
    ck = clocks.stop() if clocks else None
    log(f"[bench] {variant}: {steps} timed steps {ms:.1f} ms, SOR iterations {iters}")
    tm = s.timing()
    d = s.diagnostics()
    return dict(solver=s, ms=ms, iters=iters, warm_iters=warm_iters, timing=tm, diag=d,
                dts=dts, clocks=ck, total_iters=d["total_iterations"] - d0, warm_launches=warm_launches,
                diag0=diag0, cons0=cons0)


def nvtx_mod():
    try:
        import torch
        return torch.cuda.nvtx
    except Exception:
        return None


def log(msg):
    print(msg, file=sys.stderr, flush=True)


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            pk = json.load(f)
        return float(pk["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


# ---------------------------------------------------------------- reference arm
class stdout_to_stderr:
    """Send file descriptor 1 to stderr while the reference's C code runs (it
    prints banners to stdout); the bench's stdout carries one JSON line."""

    def __enter__(self):
        sys.stdout.flush()
        self.saved = os.dup(1)
        os.dup2(2, 1)
        return self

    def __exit__(self, *exc):
        sys.stdout.flush()
        os.dup2(self.saved, 1)
        os.close(self.saved)
        return False


def reference_sample(q0, p, sor_iters=10):
    """Time the reference's own C code (oracle/_ref) on one bounded sample of a
    step: one hydro step (godunov_step_3d with gravity off) and `sor_iters`
    iterations of gravity_solve_potential, each of which in the reference
    re-evaluates the multipole boundary (gravity_solver_3d.c:712).  Returns
    (t_hydro_s, t_iter_s)."""
    from oracle.oracle import RefSim
    with stdout_to_stderr():
        r = RefSim(*p["shape"], lo=p["lo"], hi=p["hi"], G=p["G"], gamma=p["gamma"], cfl=p["cfl"],
                   bc=p["bc"], omega=1.5, max_iter=sor_iters, tol=0.0, grav_bc=1)
        r.set_state(q0)
        r.enable_gravity(False)
        t = time.perf_counter()
        r.step(1)
        t_h = time.perf_counter() - t
        rho = q0[0]
        t = time.perf_counter()
        r.gravity_solve(rho, potential_only=True)
        t_it = (time.perf_counter() - t) / sor_iters
        r.close()
    return t_h, t_it


# DRAM bytes (read + write) per grid cell of one launch, from ncu captures of
# the 256^3 workload (profiles/sor_stream_kernel_fp32_stellar_explosion_256.txt,
# profiles/sor_split_vec_kernel_fp32_stellar_explosion_256.txt,
# profiles/sor_split_kernel_fp64_stellar_explosion_256.txt), keyed by kernel and word.
NCU_DRAM_BYTES_PER_CELL = {("sor_stream_kernel", 4): 12.45, ("sor_split_vec_kernel", 4): 6.47,
                           ("sor_split_kernel", 8): 14.38}


def sor_unit(word, nz, iterations, launches):
    """(kernel, iterations of one unit) of the relaxation that ran, by its
    launches per iteration: a launch of many iterations of a grid resident in
    shared memory (counted per iteration), an FP32 pass of two, or two colour
    sweeps (in vectors where the FP32 rows of a colour are whole ones)."""
    if 4 * launches < iterations:
        return "sor_resident_kernel", 1.0
    if word == 4 and 2 * launches < 3 * iterations:
        return "sor_stream_kernel", 2.0
    return "sor_split_vec_kernel" if word == 4 and (nz + 1) // 2 % 4 == 0 else "sor_split_kernel", 0.5


REF_ITERS_FILE = os.path.join(ROOT, "hydrocode_astro1_b200", "data", "fp64_iterations.json")


def reference_iterations(n):
    """SOR iterations per warm step of the reference algorithm on this
    workload: the FP64 path runs the reference's red-black sweeps, relaxation
    and stop rule in the reference's operation order, so it takes the
    reference's iterates for a given boundary; its l=8 multipole moments are
    summed in a fixed tree order (the reference has l <= 2 only).  The counts
    were recorded by `bench.py --variant fp64 --record-fp64-iterations PATH`
    into hydrocode_astro1_b200/data/fp64_iterations.json."""
    try:
        with open(REF_ITERS_FILE) as f:
            d = json.load(f)
        return (float(d[str(n)]["mean_warm_iterations"]),
                "recorded from the FP64 path: reference sweeps and stop rule, tree-order l=8 moments")
    except Exception:
        return None, "unknown"


def main_reference(args):
    # rank 0 alone times the reference's serial code; the other ranks of a
    # torchrun launch exit at once (no process group: nothing is exchanged)
    if int(os.environ.get("RANK", "0")) != 0:
        return 0
    from oracle.oracle import have_reference
    if not have_reference():
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref not built"}))
        return 0
    q0, p = make_workload(args.n)
    ncell = p["shape"][0] * p["shape"][1] * p["shape"][2]
    I, src = reference_iterations(args.n)
    if I is None:
        I = 1000.0
        src = "assumed 1000 (no recorded FP64 iteration count)"
    for _ in range(args.warmup):
        reference_sample(q0, p, sor_iters=2)
    th, tit = [], []
    for _ in range(args.steps):
        a, b = reference_sample(q0, p, sor_iters=5)
        th.append(a)
        tit.append(b)
    t_h, t_it = statistics.median(th), statistics.median(tit)
    t_step = t_h + I * t_it
    value = ncell / t_step / 1e6
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": t_step * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic",
        "config": {"workload": f"stellar_explosion_{args.n}^3 (n=3 star, lmax 8, tol 1e-8)",
                   "grid": list(p["shape"]), "parallelism": "serial reference (1 core)",
                   "l2": "inputs larger than L2"},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": 1, "kind": "reference",
                         "sample": f"per step: 1 hydro step ({t_h:.2f} s) + 5 SOR iterations "
                                   f"({t_it * 1e3:.0f} ms each) of the reference at {args.n}^3, "
                                   f"extrapolated to {I:.0f} iterations/step ({src})"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))
    return 0


# ---------------------------------------------------------------- our arm
def main_ours(args):
    import numpy as np

    global UNET_PASSES, UNET_WEIGHTS, SOR_DEPTH
    SOR_DEPTH = args.sor_depth
    UNET_PASSES = args.unet_passes
    if args.unet_weights:
        UNET_WEIGHTS = os.path.abspath(args.unet_weights)
        if not os.path.exists(UNET_WEIGHTS):
            raise SystemExit("bench.py: no weight file %s" % UNET_WEIGHTS)

    import hydrocode_astro1_b200 as hc
    world, rank, local, dist = dist_setup(args)
    variant = args.variant
    if variant == "best":
        variant = "fp32_unet" if (args.n == 256 and os.path.exists(UNET_WEIGHTS)) else "fp32"
    q0, p = make_workload(args.n)
    ncell = p["shape"][0] * p["shape"][1] * p["shape"][2]
    t_start = 0.0
    if args.start_step > 0:
        q0, t_start = advance(q0, p, args.start_step, local)
    clocks = Clocks(local)
    r = run_variant(q0, p, variant, args.steps, args.warmup, local, dist, clocks)
    ms = reduce_max(dist, r["ms"])
    value = ncell * args.steps * world / (ms / 1e3) / 1e6
    tm = r["timing"]
    s = r["solver"]
    fp64 = variant.startswith("fp64")

    # roofline of the dominant kernel, the relaxation's.  Algorithmic bytes of
    # a unit: a pass of two FP32 iterations or one resident iteration 12 B/cell
    # (e read + write, r read), a colour sweep half of that, in FP64 of 24 (phi
    # read + write, rho read), over the interior cells.  Its time: the SOR family's
    # CUDA-event time over the units that counted; it also holds the
    # convergence checks and what was queued past convergence and returns at
    # once, so it is an upper bound.
    interior = (p["shape"][0] - 2) * (p["shape"][1] - 2) * (p["shape"][2] - 2)
    word = 8 if fp64 else 4
    kname, unit_its = sor_unit(word, p["shape"][2], sum(r["iters"]), tm["sor_launches"])
    bytes_per_launch = interior * 3 * word * min(unit_its, 1.0)
    units = max(sum(r["iters"]) / unit_its, 1)
    sor_avg_ms = tm["sor_ms"] / units
    pk, pk_kind = peaks()
    achieved = bytes_per_launch / (sor_avg_ms / 1e3) / 1e9 if sor_avg_ms > 0 else 0.0
    shares = {k: tm[k] for k in ("hydro_ms", "bc_ms", "sor_ms", "residual_ms", "moments_ms", "unet_ms")}
    traffic = NCU_DRAM_BYTES_PER_CELL.get((kname, word))
    roofline = {"bound": "hbm", "kernel": kname, "achieved": achieved, "peak": pk, "unit": "GB/s",
                "frac": achieved / pk, "peak_kind": pk_kind,
                "traffic": traffic * ncell if traffic else None,
                "algorithmic_bytes_per_launch": bytes_per_launch,
                "iterations_per_unit": unit_its,
                "avg_launch_ms": sor_avg_ms, "units": units, "launches": tm["sor_launches"]}
    hydro_bytes = interior * (48 if not fp64 else 88)
    hydro_avg = tm["hydro_ms"] / max(tm["hydro_launches"], 1)
    hydro_roof = {"kernel": "hydro_interior", "achieved": hydro_bytes / (hydro_avg / 1e3) / 1e9 if hydro_avg else 0,
                  "unit": "GB/s", "avg_launch_ms": hydro_avg,
                  "algorithmic_bytes_per_launch": hydro_bytes}
    hydro_roof["frac"] = hydro_roof["achieved"] / pk

    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None,
        "dtype": "f64" if fp64 else ("f32 hydro / f64+f32 poisson / bf16 u-net" if variant == "fp32_unet"
                                     else "f32 hydro / f64+f32 poisson"),
        "data": "synthetic",
        "config": {"workload": f"stellar_explosion_{args.n}^3 (n=3 star, lmax 8, tol 1e-8)"
                               + (f", window from step {args.start_step}" if args.start_step else ""),
                   "grid": list(p["shape"]), "variant": variant,
                   "start_step": args.start_step, "t_start": t_start,
                   "parallelism": "replicas" if world > 1 else "single GPU",
                   "l2": "inputs larger than L2 (state >= 335 MB per buffer)"},
        "sor_iterations_per_step": r["iters"],
        "warmup_iterations": r["warm_iters"],
        "time_ms": shares,
        "roofline": roofline,
        "roofline_hydro": hydro_roof,
        "gpu_launches": tm["launches"],
        "warmup_gpu_launches": r["warm_launches"],
        "clocks": r["clocks"],
    }

    def poisson_ms(t, k):
        return (t["sor_ms"] + t["residual_ms"] + t["moments_ms"] + t["unet_ms"]) / k

    # the same FP32 path without the learned warm start
    cons_main = s.conservation()
    if variant == "fp32_unet" and not args.no_fp32_compare:
        qmain = s.state()
        s.close()
        rp = run_variant(q0, p, "fp32", args.steps, args.warmup, local, dist, None)
        msp = reduce_max(dist, rp["ms"])
        d1, dd0 = r["diag"], r["diag0"]
        line["fp32_plain"] = {"value": ncell * args.steps * world / (msp / 1e3) / 1e6,
                              "ms_per_step": msp / args.steps, "sor_iterations_per_step": rp["iters"]}
        line["learned_warm_start"] = {
            "weights": os.path.relpath(UNET_WEIGHTS, ROOT),
            "accepted": d1["unet_accepted"] - dd0["unet_accepted"],
            "fallbacks": d1["unet_fallbacks"] - dd0["unet_fallbacks"],
            "monitor": {"consecutive_losses_to_switch_off": UNET_GUARD,
                        "probes_in_window": d1["unet_probes"] - dd0["unet_probes"],
                        "probes_total": d1["unet_probes"], "wins": d1["unet_wins"],
                        "losses": d1["unet_losses"], "switch_offs": d1["unet_switch_offs"],
                        "off_at_end": d1["unet_off"]},
            "sor_iterations_learned": r["iters"], "sor_iterations_plain": rp["iters"],
            "iterations_saved_frac": 1.0 - sum(r["iters"]) / max(1, sum(rp["iters"])),
            "poisson_ms_per_solve_learned": poisson_ms(tm, args.steps),
            "poisson_ms_per_solve_plain": poisson_ms(rp["timing"], args.steps),
            "unet_ms_per_solve": tm["unet_ms"] / args.steps,
            "density_l1_vs_plain": float(np.abs(qmain[0] - rp["solver"].state()[0]).mean()
                                         / np.abs(rp["solver"].state()[0]).mean())}
        rp["solver"].close()
        s = None

    # the plain FP64 path on the same workload, for the FP32/FP64 speed-up
    if not fp64 and not args.no_fp64_compare:
        if s is None:
            q32 = qmain
        else:
            q32 = s.state()
            s.close()
        r64 = run_variant(q0, p, "fp64", args.steps, args.warmup, local, dist, None)
        ms64 = reduce_max(dist, r64["ms"])
        v64 = ncell * args.steps * world / (ms64 / 1e3) / 1e6
        q64 = r64["solver"].state()
        c64 = r64["solver"].conservation()
        line["fp64_plain"] = {"value": v64, "ms_per_step": ms64 / args.steps,
                              "sor_iterations_per_step": r64["iters"],
                              "speedup_of_value": value / v64}
        # accuracy of this run against the FP64 path after the same W+K steps;
        # drifts from the FP64 totals each solver forms on the device
        c0m, c064 = r["cons0"], r64["cons0"]
        line["accuracy_vs_fp64"] = {
            "steps": args.warmup + args.steps,
            "density_l1": float(np.abs(q32[0] - q64[0]).mean() / np.abs(q64[0]).mean()),
            "mass_drift": float(cons_main[0] / c0m[0] - 1.0),
            "mass_drift_fp64": float(c64[0] / c064[0] - 1.0),
            "energy_drift": float(cons_main[4] / c0m[4] - 1.0),
            "energy_drift_fp64": float(c64[4] / c064[4] - 1.0),
            "drift_source": "hc_conservation_sums (FP64, on the device)",
            "finite": bool(np.isfinite(q32).all()),
            "time_fp32": float(sum(r["dts"]) + 0.0), "time_fp64": float(sum(r64["dts"]))}
        del q32, q64
        r64["solver"].close()
        s = make_solver(p, variant, local)
        s.set_state(q0)
        for _ in range(args.warmup):
            s.step(1)

    if s is None:   # the main solver was closed for a comparison arm
        s = make_solver(p, variant, local)
        s.set_state(q0)
        for _ in range(args.warmup):
            s.step(1)

    # end to end through the C ABI with host buffers (AoS State3D, pinned)
    if not args.no_e2e:
        U = hc.pin(s.state_aos())
        ne = min(args.steps, 3)
        barrier(dist)
        t = time.perf_counter()
        for _ in range(ne):
            s.step_host(U)
        te = time.perf_counter() - t
        log(f"[bench] e2e: {ne} steps through hc_step_host in {te:.3f} s")
        te = reduce_max(dist, te)
        hc.unpin(U)
        line["e2e"] = {"value": ncell * ne * world / te / 1e6, "unit": UNIT,
                       "h2d_bytes_per_step": int(U.nbytes), "d2h_bytes_per_step": int(U.nbytes),
                       "steps": ne, "api": "hc_step_host (State3D host array in, out)"}
    s.close()

    # the reference C code on the host, bounded sample
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        from oracle.oracle import have_reference
        if have_reference():
            t0 = time.perf_counter()
            th, tit = reference_sample(q0, p, sor_iters=5)
            log(f"[bench] cpu baseline sample: hydro {th:.2f} s, SOR {tit * 1e3:.0f} ms/iteration "
                f"({time.perf_counter() - t0:.1f} s total)")
            # SOR iterations per step of the reference's algorithm: this run's
            # FP64 arm when it ran, else the count recorded for the default window
            I = statistics.mean(r["iters"]) if fp64 else None
            if I is None and "fp64_plain" in line:
                I = statistics.mean(line["fp64_plain"]["sor_iterations_per_step"])
            if I is None and args.start_step == 0:
                I, _src = reference_iterations(args.n)
            I = I or 1000.0
            t_step = th + I * tit
            line["cpu_baseline"] = {
                "value": ncell / t_step / 1e6, "unit": UNIT, "cores": 1, "kind": "reference",
                "sample": f"1 hydro step ({th:.2f} s) + 5 SOR iterations ({tit * 1e3:.0f} ms each) "
                          f"of the reference at {args.n}^3, extrapolated to {I:.0f} iterations/step"}
        else:
            line["cpu_baseline"] = None

    if fp64 and rank == 0 and args.record_fp64_iterations:
        path = os.path.abspath(args.record_fp64_iterations)
        d = {}
        if os.path.exists(path):
            with open(path) as f:
                d = json.load(f)
        d[str(args.n)] = {"mean_warm_iterations": statistics.mean(r["iters"]),
                          "per_step": r["iters"], "warmup": r["warm_iters"],
                          "moments": "tree order, lmax 8"}
        with open(path, "w") as f:
            json.dump(d, f, indent=1)

    if rank == 0:
        print(json.dumps(line))
    if dist is not None:
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    a = parse()
    sys.exit(main_reference(a) if a.impl == "reference" else main_ours(a))
