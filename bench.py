"""Benchmark: 3D FP32 FDTD leapfrog steps on B200 (GCUPS and HBM roofline).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl b200|reference]
                    [--scene 3d_512|capacity|2d_400]

One bench "step" is one leapfrog time step of the scene (pre-E source, H, E,
CPML psi, PEC, DFT monitors).  The default scene is the 512 x 512 x 256
CPML + Si-box + dipole + 4-plane DFT workload.  Every rank runs its own
replica (the step is single-GPU: no sharding, no collectives), so
``value`` = cells x steps x ranks / max-over-ranks device time ("weak").

``--impl reference`` times the CPU restatement of beamz's float32 step
(oracle/fdtd_cpu.c, OpenMP over every host thread) on the same scene, each
step a bounded z-slab sample of it, on rank 0 only.
"""

from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

from beamz_b200 import replicas  # noqa: E402

FALLBACK_HBM_GBS = 6650.0


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=1000)
    ap.add_argument("--warmup", type=int, default=20)
    ap.add_argument("--impl", default="b200", choices=["b200", "reference"])
    ap.add_argument("--scene", default="3d_512", choices=["3d_512", "capacity", "2d_400"])
    ap.add_argument("--tile", default="32x8")
    ap.add_argument("--z-chunk", type=int, default=16)
    ap.add_argument("--cpml-faces", choices=["all", "x", "y", "z", "none"], default="all",
                    help="3d_512 only: the faces that carry the absorber (the absorber's cost per axis)")
    ap.add_argument("--material", choices=["dielectric", "conductive"], default="dielectric",
                    help="3d_512 only: conductive Si boxes (sigma 4e4 S/m: per-site E and H decay)")
    ap.add_argument("--grid", choices=["uniform", "axis_uniform", "rectilinear"], default="uniform",
                    help="3d_512 only: seeded cell widths of 1-1.25 x 20 nm per axis (derivative metrics)")
    ap.add_argument("--step-kernel", choices=["classes", "codebook"], default=None,
                    help="pitched 3D step (default: the runtime's choice)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--kernel-steps", type=int, default=200)
    ap.add_argument("--shape", default=None, help="override the scene grid as ZxYxX (profiling runs)")
    ap.add_argument("--serving", action="store_true", help="the request stream: batched serving vs one-at-a-time")
    ap.add_argument("--requests", type=int, default=256)
    ap.add_argument("--rate", type=float, default=200.0, help="Poisson arrival rate (requests/s)")
    ap.add_argument("--adjoint", choices=["2d", "3d"], default=None, help="inverse design: forward + adjoint gradient")
    ap.add_argument("--accuracy", choices=["reduced", "full"], default="reduced",
                    help="accuracy key: a reduced copy of the scene against the FP32 and FP64 oracles (default), "
                         "or the full 512x512x256 scene over all 1000 steps against the C restatement (minutes)")
    args = ap.parse_args()
    if args.grid != "uniform" and args.scene != "3d_512":
        ap.error("--grid applies to the 3d_512 scene")
    return args


def peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(path) as fh:
            data = json.load(fh)
        return float(data["hbm_gbs"]), "measured"
    except (OSError, KeyError, ValueError):
        return FALLBACK_HBM_GBS, "fallback"


class ClockSampler:
    """nvidia-smi clock / throttle samples during the timed region."""

    QUERY = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.QUERY}", "--format=csv,noheader,nounits",
                 "-lms", "100"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
            time.sleep(0.3)
        except OSError:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *exc):
        if self.proc is not None:
            time.sleep(0.2)
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], [], set()
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        for line in self.lines:
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx.append(float(parts[2]))
            except ValueError:
                continue
            for name, flag in zip(names, parts[5:9]):
                if flag.lower() == "active":
                    reasons.add(name)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx), "reasons": sorted(reasons),
                "samples": len(sm)}


def cpu_sample(spec_fn, total_steps, budget_s, threads=0):
    """Time the C restatement on z-slabs of the scene; returns (gcups, steps, shape, threads)."""
    from oracle import cpu_port

    cpu_port.build()
    nthreads = threads or cpu_port.max_threads()
    probe = spec_fn(total_steps=3, shape=(16, 512, 512), monitors=False)
    run = cpu_port.HostRun(probe)
    t0 = time.perf_counter()
    run.run(2, threads=nthreads)
    per_cell_step = (time.perf_counter() - t0) / (2 * probe.cells)
    return per_cell_step, nthreads


def config_block(args, spec) -> dict:
    """The workload description both arms print (the driver compares them)."""
    suffix = ("_conductive" if getattr(args, "material", "") == "conductive" else "") + (
        "_" + args.grid if getattr(args, "grid", "uniform") != "uniform" else "")
    scene = {"3d_512": "3d_512x512x256_cpml12_sibox_dipole_dft4x5" + suffix,
             "capacity": "capacity_1536x1024x1024_cpml12",
             "2d_400": "2d_400x400_tm_cpml20_strip_dft3"}[args.scene]
    return {"workload": scene, "grid_zyx": [int(v) for v in spec.grid_shape], "cells": int(spec.cells),
            "parallelism": f"replicas x{max(1, int(os.environ.get('WORLD_SIZE', '1')))}",
            "l2": "inputs larger than L2 (two field banks of %.1f GB)" % (2 * 4 * 6 * spec.cells / 1e9)}


def reference_arm(args, scene_fn, cells_full):
    """CPU restatement of the reference step: bounded z-slab samples per step."""
    from oracle import cpu_port

    per_cell, nthreads = cpu_sample(scene_fn, 3, 10.0)
    steps = args.steps + args.warmup
    budget = 150.0
    nz = int(max(8, min(256, budget / max(steps, 1) / (per_cell * 512 * 512))))
    spec = scene_fn(total_steps=steps, shape=(nz, 512, 512), monitors=True)
    run = cpu_port.HostRun(spec)
    run.run(args.warmup, threads=nthreads)
    t0 = time.perf_counter()
    run.run(args.steps, threads=nthreads)
    dt = time.perf_counter() - t0
    gcups = spec.cells * args.steps / dt / 1e9
    sample = f"{args.steps} steps of a {nz}x512x512 z-slab of the 512x512x256 scene (CPML, Si boxes, dipole, 4 DFT planes)"
    line = {
        "impl": "reference", "metric": "GCUPS", "value": round(gcups, 4), "unit": "Gcell-updates/s",
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(dt / args.steps * 1e3, 3),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": config_block(args, scene_fn(total_steps=1, monitors=False, sources=False)),
        "cpu_baseline": {"value": round(gcups, 4), "unit": "Gcell-updates/s", "cores": nthreads, "kind": "port",
                         "sample": sample, "sample_cells": spec.cells},
        "e2e": {"value": round(gcups, 4), "unit": "Gcell-updates/s", "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def serving_arm(args, rank, world):
    """Config 4: a seeded Poisson stream through the serving engine, then the
    same requests one at a time through the plain path (rank-local shards)."""
    import torch

    from beamz_b200 import serve
    from beamz_b200 import workloads as W

    stream = W.serving_requests(args.requests, rate=args.rate, seed=2024)
    mine = replicas.shard(stream, rank, world)
    reqs = [serve.Request(i, s, s.total_steps, a) for i, (a, s) in enumerate(mine)]
    warm = [serve.Request(0, W.scene_2d(total_steps=16, shape=(64, 64)), 16, 0.0),
            serve.Request(1, W.scene_3d_512(total_steps=16, shape=(32, 32, 32), pml_cells=4, n_monitors=1, n_freqs=3),
                          16, 0.0)]
    serve.run_sequential(warm)
    serve.ServingEngine().run(warm)
    engine = serve.ServingEngine()
    with ClockSampler(int(os.environ.get("LOCAL_RANK", "0"))) as clocks:
        batched = engine.run(reqs)
        sequential = serve.run_sequential(reqs)
    b, q = serve.summarize(batched), serve.summarize(sequential)
    same = all(np.array_equal(x.dft_re, y.dft_re) and np.array_equal(x.dft_im, y.dft_im)
               for x, y in zip(batched, sequential))
    line = {"metric": "sims/s (batched serving)", "value": round(b.sims_per_s, 3), "unit": "simulations/s",
            "n_gpus": world, "higher_is_better": True, "scaling": "weak", "dtype": "f32",
            "data": "synthetic (seeded request stream)",
            "config": {"workload": "serving: Poisson arrivals, 2D 256^2-1024^2 and 3D 128^3/192^3/256x256x128, "
                                   "500-4000 steps, 1-4 DFT monitors", "requests": len(reqs), "rate_per_s": args.rate},
            "batched": {"sims_per_s": round(b.sims_per_s, 3), "p50_s": round(b.p50_s, 3), "p99_s": round(b.p99_s, 3),
                        "makespan_s": round(b.makespan_s, 2), "peak_resident": engine.peak_active,
                        "peak_gb": round(engine.peak_bytes / 1e9, 2)},
            "sequential": {"sims_per_s": round(q.sims_per_s, 3), "p50_s": round(q.p50_s, 3),
                           "p99_s": round(q.p99_s, 3), "makespan_s": round(q.makespan_s, 2),
                           **{k: round(v, 3) for k, v in q.extra.items()}},
            "speedup": round(b.sims_per_s / q.sims_per_s, 3), "results_identical": same,
            "clocks": clocks.summary()}
    if rank == 0:
        print(json.dumps(line), flush=True)


def adjoint_arm(args):
    """Config 5: forward with checkpoints every 100 steps plus the adjoint
    gradient of a port-overlap objective w.r.t. a design density."""
    import torch

    from beamz_b200 import adjoint as A
    from beamz_b200 import plan as P
    from beamz_b200 import workloads as W

    gen = torch.Generator(device="cpu").manual_seed(5)
    out = {}
    if args.adjoint == "2d":
        ny = nx = 600
        nsteps = 3000
        spec = W.scene_2d(total_steps=nsteps, seed=5, shape=(ny, nx), pml_cells=20, n_monitors=1)
        y0, x0 = 200, 200
        box = ((y0, x0), (y0 + 200, x0 + 200))
        problem = A.AdjointProblem(spec, nsteps, box, checkpoint_every=100)
        raw = torch.rand((1, 1, 200, 200), generator=gen)
        k = torch.exp(-0.5 * (torch.arange(-9, 10, dtype=torch.float32) / 3.0) ** 2)
        k = (k / k.sum())
        blur = torch.nn.functional.conv2d(torch.nn.functional.conv2d(raw, k.view(1, 1, 1, -1), padding=(0, 9)),
                                          k.view(1, 1, -1, 1), padding=(9, 0))[0, 0]
        rho = blur.cuda().requires_grad_(True)
        eps_bg = torch.full((ny, nx), W.OXIDE, device="cuda")
        mon = spec.monitors[0]
        npts = np.asarray(mon.indices[0]).shape[0]
        nf = len(mon.freqs)
        prof = torch.exp(-0.5 * ((torch.arange(npts, dtype=torch.float32) - npts / 2) / (npts / 10)) ** 2).cuda()
        ez = P.COMPONENT_INDEX["Ez"]

        def objective(r):
            eps = eps_bg.clone()
            eps[y0:y0 + 200, x0:x0 + 200] = W.OXIDE + r * (W.SI - W.OXIDE)
            re, im = A.simulate(problem, [A.eps_to_coefficients_2d(eps, spec.dt, P.EPS_0)])
            sl = slice((ez * nf + nf // 2) * npts, (ez * nf + nf // 2 + 1) * npts)
            return (prof * re[sl]).sum() ** 2 + (prof * im[sl]).sum() ** 2

        designs = [rho]
        cells = ny * nx
        workload = "2D TM 600x600, 200x200 design, 3000 steps, checkpoints every 100"
    else:
        shape = (128, 256, 256)
        nsteps = 1500
        spec = W.scene_3d_512(total_steps=nsteps, seed=6, shape=shape, n_monitors=1, n_freqs=3)
        base = torch.as_tensor(spec.eps_table[spec.voxel_ids], device="cuda")
        coefs0 = A.eps_to_coefficients_3d(base, spec.dt, P.EPS_0)
        sspec = A.site_spec(spec, {c: v.cpu().numpy() for c, v in zip(("Ex", "Ey", "Ez"), coefs0)})
        z0 = shape[0] // 2 - 5
        box = ((z0, 96, 96), (z0 + 12, 160, 160))
        problem = A.AdjointProblem(sspec, nsteps, box, checkpoint_every=100)
        mon = spec.monitors[0]
        npts = max(np.asarray(ix).shape[0] for ix in mon.indices)
        nf = len(mon.freqs)
        w = torch.randn(npts, generator=gen).cuda()
        ey = P.COMPONENT_INDEX["Ey"]

        def objective(r):
            eps = base.clone()
            eps[z0 + 1:z0 + 11, 97:159, 97:159] = W.OXIDE + r * (W.SI - W.OXIDE)
            re, im = A.simulate(problem, A.eps_to_coefficients_3d(eps, spec.dt, P.EPS_0))
            sl = slice((ey * nf + nf // 2) * npts, (ey * nf + nf // 2 + 1) * npts)
            return (w * re[sl]).sum() ** 2 + (w * im[sl]).sum() ** 2

        designs = [torch.rand((10, 62, 62), generator=gen).cuda().requires_grad_(True) for _ in range(8)]
        cells = int(np.prod(shape))
        workload = "3D 256x256x128, batch of 8 designs (10x62x62), 1500 steps, checkpoints every 100"
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    fwd = bwd = 0.0
    for r in designs:
        a = time.perf_counter()
        val = objective(r)
        torch.cuda.synchronize()
        b = time.perf_counter()
        val.backward()
        torch.cuda.synchronize()
        fwd += b - a
        bwd += time.perf_counter() - b
    total = time.perf_counter() - t0
    out = {"metric": "adjoint gradient time", "value": round(total / len(designs), 3), "unit": "s per design",
           "higher_is_better": False, "n_gpus": 1, "dtype": "f32", "data": "synthetic (seeded density)",
           "config": {"workload": workload, "designs": len(designs)},
           "forward_s": round(fwd / len(designs), 3), "backward_s": round(bwd / len(designs), 3),
           "forward_gcups": round(cells * nsteps / (fwd / len(designs)) / 1e9, 2),
           "peak_hbm_gb": round(torch.cuda.max_memory_allocated() / 1e9, 2),
           "grad_norm": float(designs[0].grad.norm())}
    print(json.dumps(out), flush=True)


def accuracy_report(dev) -> dict:
    """The engine against the FP32 oracle (the reference's arithmetic) and the
    FP64 oracle on a reduced copy of the scene (same generator), from seeded
    random fields so every cell is live: the largest per-component relative L2
    error of the fields and the DFT arena's."""
    from beamz_b200 import plan as P
    from beamz_b200 import runtime as R
    from beamz_b200 import workloads as W
    from oracle import fdtd_oracle as O
    from oracle.from_spec import oracle_program

    steps = 24
    spec = W.scene_3d_512(total_steps=steps, shape=(32, 64, 64), pml_cells=6)
    rng = np.random.default_rng(7)
    fields = {c: rng.standard_normal(P.component_shape(c, spec.grid_shape)).astype(np.float32)
              * np.float32(1.0 if c[0] == "E" else 1.0 / 376.73) for c in P.COMPONENTS}
    prog = R.compile_program(spec, device=dev)
    out = R.run_steps(R.initial_state(prog, fields=fields), prog, steps).numpy()
    report = {"case": f"32x64x64 copy of the scene, CPML 6, {steps} steps from seeded random fields"}
    for name, dtype in (("fp32", np.float32), ("fp64", np.float64)):
        oprog = oracle_program(spec, dtype)
        st = O.new_state(oprog, dtype)
        for c, v in fields.items():
            st.fields[c] = v.astype(dtype)
        st = O.run(st, oprog, steps)
        report[f"fields_rel_l2_{name}"] = float(max(O.relative_l2(out[c], st.fields[c]) for c in P.COMPONENTS))
        report[f"dft_rel_l2_{name}"] = float(max(O.relative_l2(out["dft_re"], st.dft_re),
                                                 O.relative_l2(out["dft_im"], st.dft_im)))
    return report


def accuracy_full(dev, step_kernel: str) -> dict:
    """The 512 x 512 x 256 workload over its full 1000 steps from zero fields
    (the dipole pulse and the 4 x 5 DFT planes) against the C restatement of
    the reference's float32 step on every host thread: the largest
    per-component relative L2 error of the fields and of the DFT arena.  The
    float64 error is the reduced case's (no float64 restatement runs this size
    in bounded time)."""
    from beamz_b200 import plan as P
    from beamz_b200 import runtime as R
    from beamz_b200 import workloads as W
    from oracle import cpu_port
    from oracle import fdtd_oracle as O

    steps = 1000
    spec = W.scene_3d_512(total_steps=steps)
    prog = R.compile_program(spec, device=dev, step_kernel=step_kernel)
    out = R.run_steps(R.initial_state(prog), prog, steps).numpy()
    del prog
    import torch

    torch.cuda.empty_cache()
    cpu_port.build()
    t0 = time.perf_counter()
    ref = cpu_port.HostRun(spec).run(steps, threads=0)
    cpu_s = time.perf_counter() - t0
    fields = {c: O.relative_l2(out[c], ref.fields[c]) for c in P.COMPONENTS}
    report = {"case": "512x512x256 scene (CPML 12, Si boxes, Ey dipole pulse, 4 DFT planes x 5 f), "
                      f"{steps} steps from zero fields, against the C restatement (float32)",
              "steps": steps, "fields_rel_l2_fp32": float(max(fields.values())),
              "fields_rel_l2_fp32_per_component": {c: float(v) for c, v in fields.items()},
              "fields_bit_identical_fp32": bool(all(np.array_equal(out[c], ref.fields[c]) for c in P.COMPONENTS)),
              "dft_rel_l2_fp32": float(max(O.relative_l2(out["dft_re"], ref.dft_re),
                                           O.relative_l2(out["dft_im"], ref.dft_im))),
              "dft_weights_equal": bool(np.array_equal(out["dft_w"], ref.dft_w)),
              "reference_cpu_s": round(cpu_s, 1), "step_kernel": step_kernel}
    report["reduced_fp64"] = accuracy_report(dev)
    return report


def main():
    args = parse()
    import torch

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    from beamz_b200 import workloads as W

    scene_fn = W.SCENES[args.scene]
    if args.adjoint:
        if rank == 0:
            adjoint_arm(args)
        return
    if args.serving and args.impl == "b200":
        if world > 1:
            import torch.distributed as dist

            dist.init_process_group("nccl", init_method="env://",
                                    timeout=__import__("datetime").timedelta(seconds=600))
            torch.cuda.set_device(local)
        serving_arm(args, rank, world)
        if world > 1:
            dist.barrier()
            dist.destroy_process_group()
        return
    if args.impl == "reference":
        if rank == 0:
            reference_arm(args, W.scene_3d_512, 512 * 512 * 256)
        return

    import torch.distributed as dist

    from beamz_b200 import runtime as R

    if world > 1:
        dist.init_process_group("nccl", init_method="env://", timeout=__import__("datetime").timedelta(seconds=120))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    tile = tuple(int(v) for v in args.tile.split("x"))
    primes = 1 if args.steps % 2 == 0 else 2
    total = args.warmup + (primes + 2) * args.steps
    shape_kw = {"shape": tuple(int(v) for v in args.shape.split("x"))} if args.shape else {}
    if args.scene == "3d_512" and args.cpml_faces != "all":
        shape_kw["cpml_edges"] = {"x": ("left", "right"), "y": ("bottom", "top"), "z": ("front", "back"),
                                  "none": ()}[args.cpml_faces]
    spec = scene_fn(total_steps=total, **shape_kw)
    if args.material == "conductive":
        spec = W.conductive(spec)
    if args.grid != "uniform":
        spec = W.graded(spec, args.grid)
    sk = {"step_kernel": args.step_kernel} if args.step_kernel else {}
    prog = R.compile_program(spec, device=dev, schedule="fused", tile=tile, z_chunk=args.z_chunk, **sk)
    state = R.initial_state(prog)
    stream = torch.cuda.current_stream(dev)

    def barrier():
        if world > 1:
            dist.barrier()

    def prime(st, pr, nsteps):
        """Untimed pass over the exact chunk sequence of a timed run, so every
        CUDA graph it replays is captured and instantiated before timing (the
        graph key holds the bank order, hence a second pass for odd counts)."""
        for _ in range(1 if nsteps % 2 == 0 else 2):
            R.run_steps(st, pr, nsteps)

    # ---- device-resident throughput -----------------------------------------
    R.run_steps(state, prog, args.warmup)
    prime(state, prog, args.steps)
    torch.cuda.synchronize(dev)
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with ClockSampler(local) as clocks:
        barrier()
        torch.cuda.synchronize(dev)
        start.record(stream)
        R.run_steps(state, prog, args.steps)
        end.record(stream)
        torch.cuda.synchronize(dev)
        barrier()
    ms = replicas.max_over_ranks(start.elapsed_time(end), device=dev)
    cells = spec.cells
    value = replicas.aggregate_rate(cells * args.steps, ms / 1e3, world) / 1e9
    # Our kernels per step: the fused step (H-timing sources inside it, and
    # 2D pre-E sources too), one launch per other source, the DFT sample; per
    # batch of up to dft_batch steps within a graph chunk one DFT flush; per
    # chunk the step-counter advance.
    separate = sum(1 for s in spec.sources
                   if s.timing == "e" or (s.timing == "pre_e" and spec.ndim == 3))
    per_step = 1 + separate + (1 if spec.monitors else 0)
    chunks = [min(R.GRAPH_CHUNK_STEPS, args.steps - c) for c in range(0, args.steps, R.GRAPH_CHUNK_STEPS)]
    flushes = sum(-(-n // prog.dft_batch) for n in chunks) if spec.monitors and prog.dft_batch > 1 else 0
    launches = per_step * args.steps + flushes + len(chunks)
    if spec.ndim == 2:  # up to eight steps per launch, the launches of the steps' parity; a last flush; the counters
        most = min(8, prog.dft_batch // 2) if spec.monitors else 8
        blocks = [-(-n // max(1, most)) for n in chunks]
        launches = sum(b + ((b ^ n) & 1) for b, n in zip(blocks, chunks)) + len(chunks) * (2 if spec.monitors else 1)

    # ---- dominant kernel alone: the fused step without sources or monitors ---
    if args.scene == "3d_512":
        kspec = scene_fn(total_steps=3 * args.kernel_steps + 3, monitors=False, sources=False, **shape_kw)
        if args.material == "conductive":
            kspec = W.conductive(kspec)
        if args.grid != "uniform":
            kspec = W.graded(kspec, args.grid)
        kprog = R.compile_program(kspec, device=dev, schedule="fused", tile=tile, z_chunk=args.z_chunk, **sk)
        kstate = R.initial_state(kprog)
    else:  # other scenes time their own step (a second copy of the 1.6 G-cell scene would not fit)
        kprog, kstate = prog, state
        kprog._times_for(kstate.step + 3 * args.kernel_steps + 3)
    R.run_steps(kstate, kprog, 3)
    prime(kstate, kprog, args.kernel_steps)
    torch.cuda.synchronize(dev)
    k0, k1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    k0.record(stream)
    R.run_steps(kstate, kprog, args.kernel_steps)
    k1.record(stream)
    torch.cuda.synchronize(dev)
    kernel_ms = k0.elapsed_time(k1) / args.kernel_steps
    peak_hbm = torch.cuda.max_memory_allocated(dev)
    del kstate, kprog
    alg_bytes = W.algorithmic_bytes(spec)
    achieved = alg_bytes / (kernel_ms / 1e3) / 1e9
    peak, peak_kind = peaks()
    traffic = None
    # The ncu capture of the dominant kernel on this workload, when one is committed.
    kname = {"classes": "class_step", "codebook": "tma_step"}.get(prog.step_kernel, "fused_step")
    prof = os.path.join(ROOT, "profiles", f"{kname}_{args.scene}.json")
    if os.path.exists(prof) and not args.shape and tile == (32, 8) and args.z_chunk == 16 and args.cpml_faces == "all" \
            and args.material == "dielectric" and args.grid == "uniform":
        with open(prof) as fh:
            traffic = json.load(fh).get("dram_bytes_per_launch")

    # ---- end to end through the public API with host buffers ---------------
    e2e = None
    if not args.no_e2e:
        from beamz_b200.plan import COMPONENTS

        views = [state.field(c) for c in COMPONENTS]
        host = [torch.empty(v.shape, dtype=v.dtype, pin_memory=True) for v in views]
        for h, v in zip(host, views):
            h.copy_(v)
        out_fields = [torch.empty_like(h, pin_memory=True) for h in host]
        out_dft = [torch.empty(t.shape, dtype=t.dtype, pin_memory=True) for t in (state.dft_re, state.dft_im, state.dft_w)]
        h2d = sum(h.numel() * 4 for h in host)
        d2h = h2d + sum(t.numel() * 4 for t in out_dft)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        barrier()
        torch.cuda.synchronize(dev)
        e0.record(stream)
        for c, h in zip(COMPONENTS, host):
            state.field(c).copy_(h, non_blocking=True)
        R.run_steps(state, prog, args.steps)
        for h, c in zip(out_fields, COMPONENTS):
            h.copy_(state.field(c), non_blocking=True)
        for h, t in zip(out_dft, (state.dft_re, state.dft_im, state.dft_w)):
            h.copy_(t, non_blocking=True)
        e1.record(stream)
        torch.cuda.synchronize(dev)
        barrier()
        e2e_ms = replicas.max_over_ranks(e0.elapsed_time(e1), device=dev)
        e2e_value = replicas.aggregate_rate(cells * args.steps, e2e_ms / 1e3, world) / 1e9
        e2e = {"value": round(e2e_value, 3), "unit": "Gcell-updates/s",
               "h2d_bytes_per_step": int(h2d // args.steps), "d2h_bytes_per_step": int(d2h // args.steps),
               "transfers": "initial fields H2D from pinned host memory, final fields + DFT arena D2H, "
                            "amortised over the run's steps"}

    # ---- CPU baseline (rank 0, one GPU) -------------------------------------
    cpu = None
    accuracy = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline and args.scene == "3d_512" and not args.shape:
        from oracle import cpu_port

        cpu_port.build()
        nthreads = cpu_port.max_threads()
        per_cell, _ = cpu_sample(W.scene_3d_512, 3, 10.0, nthreads)
        nz = int(max(8, min(256, 15.0 / 5 / (per_cell * 512 * 512))))
        cspec = W.scene_3d_512(total_steps=5, shape=(nz, 512, 512))
        run = cpu_port.HostRun(cspec)
        t0 = time.perf_counter()
        run.run(5, threads=nthreads)
        cdt = time.perf_counter() - t0
        cpu = {"value": round(cspec.cells * 5 / cdt / 1e9, 4), "unit": "Gcell-updates/s", "cores": nthreads,
               "kind": "port",
               "sample": f"5 steps of a {nz}x512x512 z-slab of the scene, C restatement (OpenMP, {nthreads} threads)"}
        accuracy = accuracy_full(dev, prog.step_kernel) if args.accuracy == "full" else accuracy_report(dev)

    if rank == 0:
        line = {
            "metric": "GCUPS", "value": round(value, 3), "unit": "Gcell-updates/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms / args.steps, 4),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic (seeded voxels, beamz-style workload)",
            "config": config_block(args, spec),
            "launch": {"schedule": "fused", "step_kernel": prog.step_kernel, "arithmetic": prog.arithmetic,
                       "tile": list(tile), "z_chunk": args.z_chunk},
            "roofline": {"bound": "hbm", "achieved": round(achieved, 1), "peak": peak, "unit": "GB/s",
                         "frac": round(achieved / peak, 4), "traffic": traffic,
                         "kernel": {"classes": "class_step_kernel + class_column_kernel (one step)",
                                    "codebook": "tma_step_kernel"}.get(
                             prog.step_kernel, "fused step"), "kernel_ms": round(kernel_ms, 4),
                         "algorithmic_bytes_per_launch": alg_bytes, "peak_source": f"{peak_kind} hbm_gbs"},
            "peak_hbm_gb": round(peak_hbm / 1e9, 2),
            "accuracy": accuracy,
            "gpu_launches": launches,
            "clocks": clocks.summary(),
            "e2e": e2e,
            "cpu_baseline": cpu,
        }
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
