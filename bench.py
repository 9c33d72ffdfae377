"""Benchmark: stroke increments per second of the closed-die gear blank on one B200, the learned warm start with the
single-precision factor against the plain FP64 form.

Headline workload (one "step" = one forging increment, Forging3DSolver.Step, with the host-side remeshing wherever
the reference remeshes): closed-die forging of an axisymmetric gear blank (hub r15, web 6 mm, rim r45, 3 mm flash
gap, land 3:1) between two height-field dies sampled at 0.5 mm; billet d40 x h50, quarter model, meshed by
isosurface stuffing at 1.0 mm (~202k tets); C = 140 MPa, eps0 = 0.01, n = 0.08, m = 0.15, friction m_f = 0.3, ram
50 mm/s, 200 increments to closure. Synthetic data.

Forms, timed on the same increments (warm-up W, then K timed, L2 flushed between timed increments):
  value        learned warm start (per-node MLP trained before the timed region on trajectories of geometry
               variants of this case, recorded by the solver) + FP32 multifrontal factor refined by FP64 PCG to 1e-7,
               Newton tolerance 2e-4;
  plain_fp64   the reference's defaults: previous-step start, Newton tolerance 1e-3, FP64 factor and direct solve.
Both are checked increment by increment against an FP64 run converged to 1e-6 (loads always, velocities and
strains while the meshes agree); the oracle's agreement with the GPU on this mesh is a test
(tests/test_gpu_baseline_meshes.py).

Also in the line: the 3D upsetting drop-in (31.9k tets) in both forms, the 2D axisymmetric upsetting (20 x 60
quads) with its band Cholesky, each beside the CPU oracle on the same increments, and the 64-case sweep of
independent upsetting cases stepped one after another, batched, and batched with tuned launch parameters.

Arms:
  default            the CUDA path (libifea_gpu.so), device-timed with CUDA events on the solver's stream;
  --impl reference   the reference algorithm on the host cores: its C restatement under oracle/ (the C# reference
                     cannot run here), all host threads, the same workload and increments (W untimed, then timed
                     until K or the time budget, the steps it ran reported).

Multi-GPU: a forging case does not shard (one mesh, one sparse factorisation); N GPUs run N independent replicas
of the case ("scaling": "weak"), one process per GPU, timing = max over ranks.
"""
import argparse
import dataclasses
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "stroke steps/s on 1 B200, warm-start+FP32 vs plain FP64, at <=0.5% load error"
UNIT = "stroke steps/s"
FAST_TOL = 2e-4          # Newton tolerance of the timed form: five times tighter than the reference default
PCG_FORCING = 0.05       # timed form: inexact Newton, PCG to 0.05 x the previous update norm (within [1e-7, 1e-3])
WS_VARIANTS = (101, 102, 103, 104)   # geometry variants whose trajectories train the warm start
WS_TETS = 60000          # their mesh size (the network's inputs are scaled by h, so it transfers across sizes)


def headline_workload():
    from impressionfea_b200.workloads import closed_die_gear_blank
    return closed_die_gear_blank()


def config_dict(cfg, mesh, extra=None):
    d = {"workload": "closed-die gear blank (d40 x h50 billet, ~202k tets stuffed at 1.0 mm, height-field dies at "
                     "0.5 mm, 200 increments to closure, host remeshing on)",
         "tets": int(mesh.ne), "nodes": int(mesh.nn), "dof": int(3 * mesh.nn), "h_mm": cfg.h, "ds_mm": cfg.ds,
         "friction": cfg.friction, "tolerance": cfg.tol, "global_batch": 1, "parallelism": "replicas"}
    if extra:
        d.update(extra)
    return d


class ClockSampler:
    """nvidia-smi clock / throttle sampling during the timed region."""

    def __init__(self, index=0):
        self.samples = []
        self.index = index
        self._proc = None

    def __enter__(self):
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
             "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
             "clocks_event_reasons.sw_power_cap")
        try:
            self._proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={q}", "--format=csv,noheader,nounits",
                                           "-lms", "50"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self._t = threading.Thread(target=self._read, daemon=True)
            self._t.start()
            t0 = time.time()  # sampling is live before the timed region starts
            while not self.samples and time.time() - t0 < 5.0:
                time.sleep(0.01)
            self._n0 = len(self.samples)
        except Exception:
            self._proc = None
        return self

    def _read(self):
        for line in self._proc.stdout:
            self.samples.append([s.strip() for s in line.split(",")])

    def __exit__(self, *a):
        if self._proc:
            self._proc.terminate()
            try:
                self._proc.wait(timeout=5)
            except Exception:
                self._proc.kill()

    def summary(self):
        # the samples taken while the timed region ran (the ones before it only proved that sampling was live)
        if len(self.samples) > getattr(self, "_n0", 0):
            self.samples = self.samples[self._n0:]
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(s[1]) for s in self.samples if len(s) > 7 and s[1].replace(".", "").isdigit()]
        mx = [float(s[2]) for s in self.samples if len(s) > 7 and s[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for s in self.samples if len(s) > 7 for i in range(4) if s[4 + i].lower() == "active"})
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None, "reasons": reasons}


def measured_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), float(d.get("bf16_tflops_sustained", d["bf16_tflops"])), "measured"
    except Exception:
        return 6650.0, 1400.0, "fallback"


def assembly_algorithmic_bytes(ne, nn, nnz):
    """Algorithmic bytes of one matrix assembly (conn, gradients, volume, strain, element fields out; velocities,
    frames; K_vol read, K write, row index; residual and fixed flags)."""
    ndof = 3 * nn
    return ne * (16 + 96 + 8 + 8 + 64) + nn * (24 + 72) + nnz * (8 + 8 + 4) + ndof * (8 + 1)


def fast_form(cfg):
    """The timed form's configuration: Newton tolerance five times tighter than the reference default; the warm
    start and the single-precision factorisation are switched on per context."""
    return dataclasses.replace(cfg, tol=FAST_TOL)


# ------------------------------------------------------------------ reference arm (host cores)

def oracle_window(cfg, mesh, dies, warmup, steps, budget_s, threads, remesh=True):
    """The oracle over the same increments as the GPU arm: `warmup` untimed, then timed until `steps` or the
    budget; returns (increments per second, increments timed, their Newton iterations, loads, seconds). With
    remesh, it remeshes where the GPU arm does, by the same host remesher."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    from build_oracle import build_oracle
    build_oracle()
    os.environ["OMP_NUM_THREADS"] = str(threads)
    from oracle import Oracle3D
    o = Oracle3D(cfg, mesh, dies)
    if remesh:
        o.enable_remesh(dies)
    t_start = time.perf_counter()
    for _ in range(warmup):
        o.step()
    n, its, loads = 0, [], []
    t0 = time.perf_counter()
    while n < steps and (n == 0 or time.perf_counter() - t_start < budget_s):
        o.step()
        its.append(int(o.scalar("iterations")))
        loads.append(o.scalar("load"))
        n += 1
    el = time.perf_counter() - t0
    o.close()
    return n / el, n, its, loads, el


def cpu_newton_sample(cfg, mesh, dies, threads, plain_infos):
    """A bounded sample of the oracle on the headline workload: one Newton iteration at the first increment's
    start (PrepareStep, matrix assembly, boundary conditions, one factorisation and solve), scaled to increments by
    the plain FP64 form's Newton iterations and factorisations per increment in the timed window."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    from build_oracle import build_oracle
    build_oracle()
    os.environ["OMP_NUM_THREADS"] = str(threads)
    from oracle import Oracle3D, OracleSpd
    o = Oracle3D(cfg, mesh, dies)
    t0 = time.perf_counter()
    o.prepare_step()
    o.assemble(1, 1, o.array("v"))
    o.apply_bc()
    t_asm = time.perf_counter() - t0
    f = OracleSpd()
    f.set_geometry(o.array("x"))
    cp, ri, val = o.array("col_ptr"), o.array("row_idx"), o.array("val")
    f.analyze(len(cp) - 1, cp, ri)
    t0 = time.perf_counter()
    f.factorize(val)
    t_fact = time.perf_counter() - t0
    t0 = time.perf_counter()
    f.solve(o.array("r"))
    t_solve = time.perf_counter() - t0
    its = sum(i["iterations"] for i in plain_infos) / max(len(plain_infos), 1)
    facts = (plain_infos[-1]["n_factor"] - plain_infos[0]["n_factor"] + 1) / max(len(plain_infos), 1) if plain_infos else 1
    per_inc = its * (t_asm + t_solve) + facts * t_fact
    o.close()
    f.close()
    return {"value": 1.0 / per_inc, "unit": UNIT, "cores": threads, "kind": "port",
            "sample": f"one Newton iteration of the oracle on the closed-die mesh (assembly + BC {t_asm:.2f} s, "
                      f"factorisation {t_fact:.2f} s, solve {t_solve:.2f} s), scaled by the plain FP64 form's "
                      f"{its:.1f} Newton iterations and {facts:.2f} factorisations per timed increment; the measured "
                      f"window is the reference arm's (--impl reference)"}


def run_reference(args, rank, world):
    if rank != 0:
        return
    threads = os.cpu_count()
    cfg, mesh, dies = headline_workload()
    value, n, its, _, el = oracle_window(cfg, mesh, dies, args.warmup, args.steps, args.ref_budget, threads)
    sample = (f"increments {args.warmup + 1}..{args.warmup + n} of the closed-die case after {args.warmup} untimed "
              f"({n} of the {args.steps} asked within the {args.ref_budget:.0f} s budget; {sum(its)} Newton "
              f"iterations); project C restatement of the reference path, OpenMP element phase, serial scatter, "
              f"supernodal multifrontal Cholesky (the reference's MKL PARDISO is unavailable here; its published "
              f"0.09-0.18 s per 17k-DOF factorisation is README.md:339-340)")
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus, "steps": n,
            "warmup": args.warmup, "ms_per_step": 1000.0 / value, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": config_dict(cfg, mesh, {"remesh": "on, by the library's host remesher (the same host code as the GPU arm's)"}),
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port", "sample": sample},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line))


# ------------------------------------------------------------------ GPU arm

def _solver(cfg, mesh, dies, stream, fp32, net=None, remesh=True):
    from impressionfea_b200.forging3d import Forging3DSolver

    s = Forging3DSolver(cfg, mesh, dies)
    if stream is not None:
        s.set_stream(stream.cuda_stream)
    if fp32:
        s.set_scalar("factor_fp32", 1)
        s.set_scalar("pcg_forcing", PCG_FORCING)
    if remesh:
        s.set_scalar("remesh", 1)
    if net is not None:
        net.attach(s, predict=True)
    return s


def _timed_steps(s, stream, flush, k, snap=("vg", "eps")):
    """k increments of solver s, each bracketed by CUDA events on the solver's stream, L2 flushed in between."""
    import torch

    durs, infos, snaps = [], [], []
    for _ in range(k):
        if s.IsFinished:
            break
        flush.zero_()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        infos.append(s.step())
        b.record(stream)
        b.synchronize()
        durs.append(a.elapsed_time(b))
        snaps.append(dict({nm: s.array(nm).copy() for nm in snap}, mesh=hash(s.array("tets").tobytes())) if snap else {})
    return durs, infos, snaps


def _errors(run_infos, run_snaps, ref_infos, ref_snaps):
    """Worst load error over the increments; velocity / strain relative L2 where both runs are on the same mesh."""
    k = min(len(run_infos), len(ref_infos))
    if k == 0:
        return None
    rl2 = lambda a, b: float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))
    same = [i for i in range(k) if run_snaps[i]["mesh"] == ref_snaps[i]["mesh"]]  # the same connectivity
    return {"load_rel_max": max(abs(run_infos[i]["load"] / ref_infos[i]["load"] - 1) for i in range(k)),
            "velocity_rel_l2_max": max((rl2(run_snaps[i]["vg"], ref_snaps[i]["vg"]) for i in same), default=None),
            "strain_rel_l2_max": max((rl2(run_snaps[i]["eps"], ref_snaps[i]["eps"]) for i in same), default=None),
            "increments": k, "increments_on_equal_meshes": len(same)}


def train_warm_start(stream, increments):
    """The learned warm start, trained before the timed region: the solver records (inputs, velocity change) of
    every accepted increment of geometry variants of the case (FP32 form, reference start), then the project's
    tensor-core kernels train the network by Adam."""
    from impressionfea_b200.warmstart import WarmStartNetwork
    from impressionfea_b200.workloads import closed_die_gear_blank

    net = WarmStartNetwork(11)
    t0 = time.perf_counter()
    tets = []
    for seed in WS_VARIANTS:
        cfg, mesh, dies = closed_die_gear_blank(target_tets=WS_TETS, seed=seed)
        tets.append(int(mesh.ne))
        s = _solver(cfg, mesh, dies, stream, True)
        net.attach(s, record=True)
        for _ in range(increments):
            s.step()
        s.close()
    t_record = time.perf_counter() - t0
    net.fit_normalisation()
    loss = net.train(steps=1500, batch=8192, lr=1e-3, seed=3)
    return net, {"variants": len(WS_VARIANTS), "tets": tets, "increments_each": increments, "samples": net.samples,
                 "record_s": round(t_record, 2), "train_steps": 1500, "batch": 8192,
                 "train_gpu_ms": round(net.last_train_ms, 1), "final_loss_normalised": loss}


def _count_launches(make, stream, warmup, k):
    """Kernels of this library launched during k increments (after the same warm-up), counted by the CUDA
    profiler interface on a re-run of the timed increments."""
    import torch

    try:
        s = make()
        for _ in range(warmup):
            s.step()
        torch.cuda.synchronize()
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            for _ in range(k):
                s.step()
            torch.cuda.synchronize()
        s.close()
        return sum(1 for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA and "at::" not in e.name
                   and ("k_" in e.name or "mf::" in e.name or "wsm::" in e.name))
    except Exception:
        return None


def whole_job_value(total_ms, k, world, device="cuda"):
    """Increments per second of the whole job: every rank ran k increments and the job took as long as its
    slowest rank (max over ranks of each rank's device time). Returns (value, that time in ms)."""
    if world > 1:
        import torch
        import torch.distributed as dist
        t = torch.tensor([total_ms], device=device, dtype=torch.float64)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        total_ms = float(t.item())
        dist.barrier()
    return world * k / (total_ms / 1000.0), total_ms


def upsetting_leg(stream, flush, warmup, steps, cpu_steps, threads):
    """The 3D upsetting drop-in (31.9k tets): FP32 form with the extrapolated start against plain FP64 on the same
    increments, and the oracle on the first of them."""
    from impressionfea_b200.workloads import upsetting_drop_in

    cfg, mesh, dies = upsetting_drop_in()
    s64 = _solver(cfg, mesh, dies, stream, False, remesh=False)
    for _ in range(warmup):
        s64.step()
    d64, i64, _ = _timed_steps(s64, stream, flush, steps, snap=None)
    s64.close()
    s32 = _solver(dataclasses.replace(fast_form(cfg), extrapolate_start=True), mesh, dies, stream, True, remesh=False)
    for _ in range(warmup):
        s32.step()
    d32, i32, _ = _timed_steps(s32, stream, flush, steps, snap=None)
    s32.close()
    ms64, ms32 = float(np.mean(d64)), float(np.mean(d32))
    out = {"workload": "3D upsetting drop-in (quarter cylinder d30 x h45, ~31.9k tets, flat dies, 40% in 80 steps)",
           "tets": int(mesh.ne), "increments": f"{warmup + 1}..{warmup + len(d32)}",
           "fp32_extrapolated_ms_per_step": ms32, "plain_fp64_ms_per_step": ms64, "speedup": ms64 / ms32,
           "newton_iterations": {"fp32": int(sum(i["iterations"] for i in i32)), "plain_fp64": int(sum(i["iterations"] for i in i64))},
           "load_rel_max_vs_plain": max(abs(a["load"] / b["load"] - 1) for a, b in zip(i32, i64))}
    if cpu_steps > 0:
        v, n, _, loads, el = oracle_window(cfg, mesh, dies, warmup, cpu_steps, 120.0, threads)
        out["oracle"] = {"value": v, "unit": UNIT, "increments": f"{warmup + 1}..{warmup + n}", "cores": threads,
                         "seconds": el, "load_rel_max_vs_plain_fp64": max(abs(a / b["load"] - 1) for a, b in zip(loads, i64))}
    return out


def leg_2d(stream, threads):
    """2D axisymmetric upsetting (20 x 60 quads, flat dies, 50 % in 100 increments; the mesh folds past increment
    80 without the remeshing the reference would do there): increments 1..80 timed, the band Cholesky kernel timed
    on its own, and the oracle over the same increments."""
    import ctypes as C

    import torch

    from impressionfea_b200 import _lib
    from impressionfea_b200.forging2d import ForgingSolver2D
    from impressionfea_b200.workloads import upsetting_2d

    cfg = upsetting_2d()
    g = ForgingSolver2D(cfg)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    its = 0
    n_inc = 80
    for _ in range(n_inc):
        its += g.step()["iterations"]
    t_gpu = time.perf_counter() - t0
    ne, ndof, hb = int(g.scalar("ne")), int(g.scalar("ndof")), int(g.scalar("half_band"))
    g.close()
    # the band factorisation + solve alone, on a system of the case's size (device buffers, CUDA events)
    rng = np.random.default_rng(5)
    w = hb + 1
    a = np.zeros(ndof * w)
    for i in range(ndof):
        lo = max(0, i - hb)
        a[i * w + (lo - i + hb):i * w + hb] = rng.random(i - lo) - 0.5
        a[i * w + hb] = 2.0 * hb + 1.0
    L = _lib.lib()
    da = torch.tensor(a, dtype=torch.float64, device="cuda")
    dr = torch.ones(ndof, dtype=torch.float64, device="cuda")
    row, piv = C.c_int32(), C.c_double()
    st = torch.cuda.current_stream()
    times = []
    for it in range(12):
        da.copy_(torch.tensor(a, dtype=torch.float64, device="cuda"))
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        L.ifea_band_factor_solve_noalloc(ndof, hb, C.c_void_p(da.data_ptr()), C.c_void_p(dr.data_ptr()), C.byref(row),
                                         C.byref(piv), C.c_void_p(st.cuda_stream))
        e1.record(st)
        e1.synchronize()
        if it >= 2:
            times.append(e0.elapsed_time(e1))
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    from oracle import Oracle2D
    os.environ["OMP_NUM_THREADS"] = str(threads)
    o = Oracle2D(cfg)
    t0 = time.perf_counter()
    for _ in range(n_inc):
        o.step()
    t_cpu = time.perf_counter() - t0
    o.close()
    return {"workload": "2D axisymmetric upsetting r10 x h30, 20 x 60 quads, 50% in 100 steps (increments 1..80)",
            "increments_per_s": n_inc / t_gpu, "ms_per_increment": 1000.0 * t_gpu / n_inc, "newton_iterations": its,
            "element_evaluations_per_s": ne * its / t_gpu, "band_factor_solve_ms": float(np.median(times)),
            "band": {"dof": ndof, "half_bandwidth": hb},
            "oracle": {"increments_per_s": n_inc / t_cpu, "cores": threads, "kind": "port"}}


def batch_leg(increments=3):
    """64 independent upsetting cases of uneven size (32 2D axisymmetric, 2k-20k quads; 32 3D quarter models,
    5k-80k tets): every case warmed up by one increment, then `increments` more stepped one case after another and
    then all cases together from a pool of host threads (ForgingBatch), with and without the tuned launch
    parameters. Wall clock around synchronised regions (the cases run on many streams)."""
    import torch

    from impressionfea_b200.batch import ForgingBatch, autotune
    from impressionfea_b200.forging2d import ForgingSolver2D
    from impressionfea_b200.forging3d import Forging3DSolver
    from impressionfea_b200.workloads import batched_sweep

    cases = batched_sweep()

    def make(tune=False):
        s3, s2 = [], []
        for c in cases:
            if c[0] == "3d":
                s = Forging3DSolver(c[1], c[2], c[3])
                s.set_scalar("factor_fp32", 1)
                s3.append(s)
            else:
                s2.append(ForgingSolver2D(c[1]))
        for s in s3 + s2:
            s.step()
        if tune:
            for s in s3:
                autotune(s)
        torch.cuda.synchronize()
        return s3, s2

    out = {"workload": "64 independent upsetting cases (32 2D axisymmetric 2k-20k quads, 32 3D quarter cylinders "
                       "5k-80k tets, seeded aspect/friction/material draws)", "increments_per_case": increments}
    s3, s2 = make()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    loads_seq = []
    for s in s3 + s2:
        for _ in range(increments):
            loads_seq.append(s.step()["load"])
    torch.cuda.synchronize()
    t_seq = time.perf_counter() - t0
    for s in s3 + s2:
        s.close()
    n = len(cases) * increments
    out["sequential"] = {"case_increments_per_s": n / t_seq, "seconds": t_seq}
    for name, tune in (("batched", False), ("batched_tuned", True)):
        s3, s2 = make(tune)
        b = ForgingBatch(s3, s2)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        infos, status = b.step(increments)
        torch.cuda.synchronize()
        t = time.perf_counter() - t0
        loads = [i["load"] for case in infos for i in case]
        out[name] = {"case_increments_per_s": n / t, "seconds": t, "speedup_vs_sequential": t_seq / t,
                     "failed_cases": int((status != 0).sum()),
                     "load_rel_max_vs_sequential": float(max(abs(a / c - 1) for a, c in zip(loads, loads_seq) if c))}
        b.close()
        for s in s3 + s2:
            s.close()
    return out


def run_gpu(args, rank, world):
    import torch

    dev = int(os.environ.get("LOCAL_RANK", 0))
    torch.cuda.set_device(dev)
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=600))
    cfg, mesh, dies = headline_workload()
    stream = torch.cuda.current_stream()
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device="cuda")
    W, K = args.warmup, args.steps

    # the learned warm start, trained before anything is timed (its cost is reported, not timed)
    net, ws = train_warm_start(stream, W + K + 2)

    # plain FP64 form: the reference's start, tolerance and FP64 direct solve
    s64 = _solver(cfg, mesh, dies, stream, False)
    for _ in range(W):
        s64.step()
    torch.cuda.synchronize()
    d64, i64, sn64 = _timed_steps(s64, stream, flush, K)
    s64.close()

    # timed form
    s = _solver(fast_form(cfg), mesh, dies, stream, True, net)
    for _ in range(W):
        s.step()
    torch.cuda.synchronize()
    if world > 1:
        torch.distributed.barrier()
    torch.cuda.synchronize()
    with ClockSampler(dev) as clk:
        # the timed increments are the profiler's range (ncu --profile-from-start off captures only them)
        torch.cuda.cudart().cudaProfilerStart()
        durs, infos, snaps = _timed_steps(s, stream, flush, K)
        torch.cuda.synchronize()
        torch.cuda.cudart().cudaProfilerStop()
    torch.cuda.synchronize()
    k = len(durs)
    value, total_ms = whole_job_value(float(sum(durs)), k, world)
    ms64 = float(sum(d64)) / len(d64)
    form = {q: s.scalar(q) for q in ("remesh_count", "ws_used", "ws_fallbacks", "n_fact", "factor_gflop", "nn", "ne")}

    # rooflines on the timed form's mesh at the end of the window: the FP32 factorisation (tensor cores), the
    # triangular-solve sweep and the matrix assembly (HBM)
    hbm_peak, tflops_peak, peak_kind = measured_peaks()
    s.set_scalar("profile_solves", 1)  # events around every factorisation and solve (a host wait each)
    f0, fms0, n_solves0, sms0 = s.scalar("n_fact"), s.scalar("factor_gpu_ms"), s.scalar("solves"), s.scalar("solve_gpu_ms")
    for _ in range(2):
        if not s.IsFinished:
            s.step()
    nf = s.scalar("n_fact") - f0
    factor_ms = (s.scalar("factor_gpu_ms") - fms0) / max(nf, 1)
    n_solves = s.scalar("solves") - n_solves0
    solve_ms = (s.scalar("solve_gpu_ms") - sms0) / max(n_solves, 1)
    s.set_scalar("profile_solves", 0)
    gflop = s.scalar("factor_gflop")
    lnnz, ndof, nnz = s.scalar("factor_nnz"), 3 * int(s.scalar("nn")), int(s.scalar("nnz"))
    sbytes = 2 * lnnz * 4 + ndof * (8 + 8 + 4 * 4)
    s.prepare_step()
    for _ in range(3):
        s.assemble(1, 1)
    asm = []
    for _ in range(10):
        flush.zero_()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        s.assemble(1, 1)
        b.record(stream)
        b.synchronize()
        asm.append(a.elapsed_time(b))
    asm_ms = float(np.median(asm))
    abytes = assembly_algorithmic_bytes(int(s.scalar("ne")), int(s.scalar("nn")), nnz)
    s.close()

    # FP64 converged to 1e-6 over the same increments (untimed): the reference of both forms' errors
    st = _solver(dataclasses.replace(cfg, tol=1e-6), mesh, dies, stream, False)
    for _ in range(W):
        st.step()
    _, itight, sntight = _timed_steps(st, stream, flush, K)
    st.close()

    # end to end through the public API with host buffers: mesh / die upload and setup, then the same increments
    # (the warm-up increments run between, untimed), each step's snapshot arrays read back to the host
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    s2 = _solver(fast_form(cfg), mesh, dies, None, True, net)
    t_setup = time.perf_counter() - t0
    for _ in range(W):
        s2.step()
    d2h, t_inc = 0, 0.0
    for _ in range(K):
        t1 = time.perf_counter()
        s2.step()
        for nm in ("x", "vg", "contact", "eps", "dmg", "el_sig", "el_rate", "el_mean"):
            d2h += s2.array(nm).nbytes
        t_inc += time.perf_counter() - t1
    e2e_s = t_setup + t_inc
    s2.close()
    h2d = mesh.x.nbytes + mesh.tets.nbytes + mesh.on_x0.nbytes + mesh.on_y0.nbytes + sum(d.h.nbytes for d in dies)

    gpu_launches = None
    if rank == 0 and not args.no_launch_count:
        gpu_launches = _count_launches(lambda: _solver(fast_form(cfg), mesh, dies, stream, True, net), stream, W, K)
    legs = {}
    threads = os.cpu_count()
    if rank == 0 and not args.no_side_legs:
        for name, fn in (("upsetting_drop_in", lambda: upsetting_leg(stream, flush, W, K, 0 if args.no_cpu_baseline else 3, threads)),
                         ("axisymmetric_2d", lambda: leg_2d(stream, threads)),
                         ("batched_sweep", batch_leg)):
            try:
                legs[name] = fn()
            except Exception as e:  # reported, not fatal: the headline stands on its own
                legs[name] = {"error": str(e)}
    if rank == 0:
        clocks = clk.summary()
        f_ach = gflop / (factor_ms / 1000.0) / 1000.0 if factor_ms > 0 else None
        s_ach = sbytes / (solve_ms / 1000.0) / 1e9 if solve_ms > 0 else None
        a_ach = abytes / (asm_ms / 1000.0) / 1e9
        line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": k, "warmup": W,
                "ms_per_step": total_ms / k, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
                "dtype": "f64 (factorisation f32 on tf32 tensor cores, refined in f64; warm-start network bf16)",
                "data": "synthetic",
                "config": config_dict(cfg, mesh, {
                    "form": "learned warm start (per-node MLP, BF16 on tcgen05) + FP32 multifrontal factor with FP64 "
                            "PCG refinement, inexact Newton (PCG to 0.05 x the previous update norm), Newton tolerance "
                            "2e-4 (plain FP64 form: reference start, 1e-3, FP64 direct)",
                    "increments": f"{W + 1}..{W + k}", "l2": "flushed (256 MiB write) between timed increments",
                    "newton_iterations": int(sum(i["iterations"] for i in infos)),
                    "factorisations": int(infos[-1]["n_factor"] - infos[0]["n_factor"]) + 1 if infos else 0,
                    "remesh_requests_in_window": int(infos[-1]["remesh_requests"] - infos[0]["remesh_requests"]) if infos else 0,
                    "end_state": form}),
                "plain_fp64": {"value": 1000.0 / ms64, "unit": UNIT, "ms_per_step": ms64, "steps": len(d64),
                               "newton_iterations": int(sum(i["iterations"] for i in i64)),
                               "speedup_of_value": value / world / (1000.0 / ms64)},
                "error_vs_tight_fp64": {"reference": "FP64 form, Newton tolerance 1e-6, same increments",
                                        "timed_form": _errors(infos, snaps, itight, sntight),
                                        "plain_fp64": _errors(i64, sn64, itight, sntight)},
                "warm_start": ws,
                "roofline": {"kernel": "FP32 multifrontal factorisation (one CUDA graph: panels, tf32 tensor-core and "
                                       "SIMT trailing updates, extend-add)", "bound": "tensor",
                             "achieved": f_ach, "peak": tflops_peak, "unit": "TFLOP/s",
                             "frac": f_ach / tflops_peak if f_ach else None, "peak_kind": peak_kind + " (bf16 dense, sustained)",
                             "traffic": None, "gflop_per_launch": gflop, "ms_per_launch": factor_ms,
                             "launches": int(nf)},
                "roofline_solve": {"kernel": "multifrontal triangular-solve sweep (forward + backward, one persistent kernel)",
                                   "bound": "hbm", "achieved": s_ach, "peak": hbm_peak, "unit": "GB/s",
                                   "frac": s_ach / hbm_peak if s_ach else None, "algorithmic_bytes": sbytes,
                                   "ms_per_launch": solve_ms, "launches": int(n_solves)},
                "roofline_assembly": {"kernel": "assembly (k_element<MATRIX> + k_columns<MATRIX,BC>)", "bound": "hbm",
                                      "achieved": a_ach, "peak": hbm_peak, "unit": "GB/s", "frac": a_ach / hbm_peak,
                                      "algorithmic_bytes": abytes, "ms_per_launch": asm_ms},
                "e2e": {"value": K / e2e_s, "unit": UNIT, "h2d_bytes_per_step": h2d / K, "d2h_bytes_per_step": d2h / K,
                        "increments": f"{W + 1}..{W + K}", "setup_s": round(t_setup, 3),
                        "note": "setup (mesh and die upload, topology, analysis thread) + the timed increments; the "
                                "warm-up increments run between, untimed"},
                "gpu_launches": gpu_launches, "clocks": clocks, **legs}
        if not args.no_cpu_baseline:
            line["cpu_baseline"] = cpu_newton_sample(cfg, mesh, dies, threads, i64)
        print(json.dumps(line))
    if world > 1:
        torch.distributed.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="cuda", choices=["cuda", "reference"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--cpu-budget", type=float, default=30.0)
    ap.add_argument("--ref-budget", type=float, default=600.0, help="reference arm: seconds for warm-up + timed increments")
    ap.add_argument("--no-side-legs", action="store_true", help="skip the upsetting and 2D measurements")
    ap.add_argument("--no-launch-count", action="store_true")
    args = ap.parse_args()
    rank = int(os.environ.get("RANK", 0))
    world = int(os.environ.get("WORLD_SIZE", 1))
    if args.impl == "reference":
        run_reference(args, rank, world)
    else:
        run_gpu(args, rank, world)


if __name__ == "__main__":
    main()
