#!/usr/bin/env python3
"""Benchmark of the formal-solve hot path: point.ray.freq solves per second.

Workload (default): the 64^3 Cartesian grid cut to a sphere of radius half the box
(rays of uneven length), 48 HEALPix rays (24 ray pairs), a 5-level linear rotor
(4 lines) with nquads 31 (124 frequencies), temperature ~ r^-0.5 from 300 K, radial
outflow 5-15 km/s plus 0.5 km/s noise; the split-precision solver.  A step is one
second-order Feautrier formal solve over all points, ray pairs and frequencies
(Model::compute_radiation_field_feautrier_order_2).

Arms:
  default           : this library on the GPU.  `value` = solves/s with the model
                      resident in HBM (CUDA events on the solver's stream, L2 flushed
                      between steps); `e2e` = the same through the public API
                      core.Model.compute_radiation_field_feautrier_order_2 with a fresh
                      host->device upload and the J/ALO read-back every step.
  --impl reference  : the reference algorithm on the host cores (the CPU oracle port,
                      all threads), on a bounded sample of the same workload.
Under torchrun with N>1 the ray pairs of the one model are sharded over the ranks
(contiguous blocks, magritte_gb300.distributed.ray_shard) and every step ends with
one FP64 NCCL sum-allreduce of the packed partial J and ALO diagonal (strong
scaling: the whole job solves the same model; `value` = its solves / the slowest
rank's time).
"""
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

METRIC = "point.ray.freq solves/s"
# DRAM bytes per solve of the split staged solve kernel, ncu on the 33^3 sphere cutout:
# 4870.5 MB read + written / 50.8 M solves
TRAFFIC_BYTES_PER_SOLVE = 4870.516e6 / 50_821_152.0
UNIT = "solves/s"


def parse():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=5)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", default="ours", choices=["ours", "reference"])
    p.add_argument("--n", type=int, default=64, help="grid points per side")
    p.add_argument("--nside", type=int, default=2)
    p.add_argument("--nquads", type=int, default=31)
    p.add_argument("--precision", default="split", choices=["split", "fp64"])
    p.add_argument("--no-cpu-baseline", action="store_true")
    p.add_argument("--no-e2e", action="store_true")
    p.add_argument("--no-parity", action="store_true", help="skip the oracle parity sample")
    p.add_argument("--no-ali", action="store_true", help="skip the ALI wall-time leg")
    p.add_argument("--ali-points", type=int, default=50_000)
    p.add_argument("--ali-nside", type=int, default=2)
    p.add_argument("--ali-iterations", type=int, default=20)
    p.add_argument("--ali-full", action="store_true",
                   help="the ALI leg at the stated size: 500k points, nside 4 (192 rays)")
    p.add_argument("--no-batch", action="store_true", help="skip the many-model batch leg")
    p.add_argument("--batch-models", type=int, default=512)
    p.add_argument("--batch-steps", type=int, default=1)
    p.add_argument("--no-adjoint", action="store_true", help="skip the differentiable-imager leg")
    p.add_argument("--adjoint-points", type=int, default=100_000)
    p.add_argument("--adjoint-pixels", type=int, default=256)
    p.add_argument("--adjoint-fd-points", type=int, default=64)
    p.add_argument("--no-adjoint-j", action="store_true", help="skip the differentiable formal-solve leg")
    p.add_argument("--adjoint-j-n", type=int, default=58, help="grid points per side of the J-adjoint model")
    p.add_argument("--no-autotune", action="store_true",
                   help="keep the library's default launch shape (for profiling one production launch)")
    return p.parse_args()


def workload(args):
    from magritte_gb300 import synthetic
    raw = synthetic.grid_sphere(n=args.n, nside=args.nside, nquads=args.nquads)
    desc = (f"grid_sphere {args.n}^3 cutout r=box/2 ({raw.npoints} points), {raw.nrays} rays, "
            f"5-level rotor (4 lines) x nquads {args.nquads}")
    return raw, desc


def dist_init():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    if ws > 1:
        import torch.distributed as dist
        backend = "nccl"
        dist.init_process_group(backend=backend)
        import torch
        torch.cuda.set_device(int(os.environ.get("LOCAL_RANK", "0")))
    return rank, ws


def barrier(ws):
    if ws > 1:
        import torch.distributed as dist
        dist.barrier()


def max_over_ranks(x, ws):
    if ws == 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64, device="cuda")
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


class Clocks:
    """nvidia-smi sampling of SM clocks and throttle reasons during a timed region."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self):
        self.proc = None
        self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits",
                                          "-lms", "200"], stdout=self.f, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        self.f.flush()
        rows = [r.split(",") for r in open(self.f.name).read().strip().splitlines() if r.strip()]
        os.unlink(self.f.name)
        dev = os.environ.get("LOCAL_RANK", "0")
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in rows:
            r = [x.strip() for x in r]
            if len(r) < 9:
                continue
            try:
                sm.append(float(r[1]))
                mx.append(float(r[2]))
            except ValueError:
                continue
            for name, val in zip(names, r[5:9]):
                if val.lower() == "active":
                    reasons.add(name)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(sm)}


# The CPU legs (this arm's cpu_baseline and the --impl reference arm) time the same
# bounded sample of the workload: every SAMPLE_STRIDE-th origin with every ray pair and
# frequency, the reference's arithmetic (the oracle port with glibc's erff), all host
# threads.  The sizing pass (Solver::get_ray_lengths_max) runs over the sampled origins.
SAMPLE_STRIDE = 32


def _oracle():
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle
    oracle.build()
    return oracle


def cpu_sample(raw):
    """(oracle module, Oracle, sampled origins, solves per sample) of the CPU legs."""
    import numpy as np
    oracle = _oracle()
    arrays = oracle.reference_setup(raw)
    orc = oracle.Oracle(arrays)
    origins = np.arange(0, arrays["npoints"], SAMPLE_STRIDE, dtype=np.uint32)
    solves = len(origins) * arrays["hnrays"] * arrays["nfreqs"]
    return oracle, orc, origins, solves


def _sample_desc(origins, solves):
    return (f"every {SAMPLE_STRIDE}th origin ({len(origins)}) x all ray pairs x all frequencies "
            f"({solves} solves per step)")


def cpu_baseline(raw, nthreads):
    """The oracle port of the reference CPU algorithm on the bounded sample."""
    oracle, orc, origins, solves = cpu_sample(raw)
    oracle.set_erf_mode(0)
    t0 = time.perf_counter()
    orc.formal_solve_fo2_origins(origins, nthreads=nthreads)
    dt = time.perf_counter() - t0
    return {"value": solves / dt, "unit": UNIT, "cores": nthreads, "kind": "port",
            "sample": _sample_desc(origins, solves) + f", {dt:.2f} s"}


def parity_sample(raw, gpu_rows, stride=50):
    """Max relative error of the GPU's J and ALO diagonal (FP64 and split) against the
    oracle on every ``stride``-th origin, in both oracle arithmetics: erf mode 1 (the
    correctly rounded erff of the GPU's FP64 mode) and erf mode 0 (glibc's erff, the
    reference's own arithmetic).  ``gpu_rows[prec] = (J [P][F], lam [P][L])``."""
    import numpy as np
    oracle = _oracle()
    arrays = oracle.reference_setup(raw)
    orc = oracle.Oracle(arrays)
    origins = np.arange(0, arrays["npoints"], stride, dtype=np.uint32)
    ref = {}
    t0 = time.perf_counter()
    try:
        for mode in (0, 1):
            oracle.set_erf_mode(mode)
            ref[mode] = orc.formal_solve_fo2_origins(origins)
    finally:
        oracle.set_erf_mode(0)
    rel = lambda a, b: float(np.max(np.abs(a - b) / np.maximum(np.abs(b), 1e-300)))
    out = {"sample": f"every {stride}th origin ({len(origins)}) x all ray pairs x all frequencies",
           "oracle_s": time.perf_counter() - t0, "bar": 1e-5}
    for prec, (J, lam) in gpu_rows.items():
        for mode, name in ((1, "erf_cr"), (0, "erf_glibc")):
            out[f"{prec}_J_vs_oracle_{name}"] = rel(J[origins], ref[mode]["J"])
            out[f"{prec}_alo_vs_oracle_{name}"] = rel(lam[origins], ref[mode]["lambda_diag"])
    out["oracle_erf_glibc_vs_erf_cr_J"] = rel(ref[0]["J"], ref[1]["J"])
    out["note"] = ("erf_cr: the oracle with the correctly rounded erff of the GPU's FP64 mode; erf_glibc: the "
                   "reference's own arithmetic (glibc erff)")
    return out


def pipe_rates():
    """Measured issue rates of the FP64-pipe instruction kinds (mgr_measure_pipe_rate)."""
    from magritte_gb300 import _abi
    out = {}
    for kind in ("dfma", "dadd", "dmul", "dsetp", "f2f", "mufu_rcp64"):
        r = _abi.pipe_rate(kind, iterations=4096 if kind != "mufu_rcp64" else 16384)
        out[kind] = {"thread_ops_per_s": r["thread_ops_per_s"],
                     "per_clk_per_sm": r["thread_ops_per_clk_per_sm"], "ms": r["ms"]}
    return out


def ali_parity(args):
    """Level populations of the ALI loop against the oracle's on the non-LTE workload
    reduced to 1,000 interior points (nside-8 outer shell, nside-4 rays, the 10-level
    rotor x 21): 8 iterations with Default Ng every 4 and no early stop, in both
    precisions; the oracle in the GPU FP64 mode's arithmetic (correctly rounded erff)."""
    import numpy as np
    from magritte_gb300 import _abi, synthetic
    oracle = _oracle()
    raw = synthetic.nlte_sphere(npoints=1000, nside=4, nside_out=8)
    params = dict(use_adaptive_Ng_acceleration=0, Ng_acceleration_mem_limit=4, pop_prec=0.0)
    oracle.set_erf_mode(1)
    t0 = time.perf_counter()
    try:
        ref = oracle.AliOracle(raw, oracle.reference_setup(raw)).run(use_ng=True, max_it=8, **params)
    finally:
        oracle.set_erf_mode(0)
    oracle_s = time.perf_counter() - t0
    tot = raw.abundance[:, raw.linedata[0].num][:, None]
    out = {"workload": f"nlte_sphere 1000 interior points ({raw.npoints} with the boundary shells), "
                       f"{raw.nrays} rays, 8 iterations, Ng every 4", "oracle_s": oracle_s, "bar": {"fp64": 1e-6,
                                                                                                "split": 1e-5}}
    for prec in ("fp64", "split"):
        a = oracle.reference_setup(raw)
        dev = _abi.DeviceModel(a)
        try:
            dev.set_species(raw.linedata, raw.abundance, a["populations"])
            dev.compute_level_populations(prec, use_ng=True, max_it=8, **params)
            pop = dev.populations(0)
        finally:
            dev.close()
        out[f"{prec}_max_rel_err_populations"] = float(np.max(np.abs(pop - ref["populations"][0]) /
                                                              np.maximum(np.abs(ref["populations"][0]), 1e-10 * tot)))
    return out


def run_ali(args):
    """ALI wall time: compute_level_populations(use_Ng=True, N) through core.Model on
    the non-LTE sphere workload (Delaunay points ~ r^-2, 10-level rotor, nquads 21),
    Default Ng every 4 iterations, exactly N normal iterations (pop_prec = 0 keeps
    the loop from stopping early), formal solves in the bench's precision,
    graph-captured iterations.  The timed call includes the model upload.  The device
    time of each phase comes from events inside the captured iteration
    (mgr_ali_phase_times); the populations are checked against the oracle on a reduced
    model (ali_parity)."""
    import time as _t

    from magritte_gb300 import loader, synthetic

    t_setup = _t.perf_counter()
    raw = synthetic.nlte_sphere(npoints=args.ali_points, nside=args.ali_nside)
    model = loader.to_core(raw, precision=args.precision)
    model.compute_spectral_discretisation()
    model.compute_inverse_line_widths()
    model.compute_LTE_level_populations()
    setup_s = _t.perf_counter() - t_setup
    prm = model.parameters
    prm.store_u = False
    prm.use_adaptive_Ng_acceleration = False
    prm.Ng_acceleration_mem_limit = 4
    prm.pop_prec = 0.0
    t0 = _t.perf_counter()
    it = model.compute_level_populations(True, args.ali_iterations)
    wall = _t.perf_counter() - t0
    ms = list(model.ali_phase_times())
    phases = None
    if len(ms) != 4:
        from magritte_gb300 import _abi
        phases = {"unavailable": _abi.load().mgr_last_error().decode()}
    if len(ms) == 4:
        phases = {"formal_solve_ms": ms[0], "jeff_ms": ms[1], "stateq_corrections_refresh_ms": ms[2],
                  "ng_ms": ms[3], "per_iteration_formal_solve_ms": ms[0] / max(it, 1)}
    P, F, R = prm.npoints(), prm.nfreqs(), prm.hnrays()
    solves = float(P) * R * F
    out = {"workload": f"nlte_sphere {raw.npoints} points (Delaunay, density ~ r^-2), {raw.nrays} rays, "
                       f"10-level rotor (9 lines) x nquads {raw.nquads}",
           "iterations": it, "ng": "Default, every 4", "precision": args.precision, "wall_s": wall,
           "s_per_iteration": wall / max(it, 1), "solves_per_iteration": solves,
           "formal_solve_solves_per_s": (solves * it / (ms[0] / 1000.0)) if len(ms) == 4 and ms[0] > 0 else None,
           "phases": phases, "setup_s": setup_s}
    if not args.no_parity:
        out["parity"] = ali_parity(args)
    if not args.no_cpu_baseline:
        out["cpu_formal_solve"] = ali_cpu_formal_solve(raw)
    return out


def ali_cpu_formal_solve(raw, target_solves=6.0e6):
    """The formal solve that dominates each ALI iteration, timed on the host cores: the
    oracle port of the reference's formal solve (glibc erff, all threads) on every
    k-th origin of the same non-LTE model (LTE line data, every ray pair and frequency),
    k chosen for about ``target_solves`` solves."""
    import numpy as np
    oracle = _oracle()
    a = oracle.reference_setup(raw)
    orc = oracle.Oracle(a)
    per_origin = a["hnrays"] * a["nfreqs"]
    stride = max(1, int(a["npoints"] * per_origin / target_solves))
    origins = np.arange(0, a["npoints"], stride, dtype=np.uint32)
    nthreads = os.cpu_count() or 1
    oracle.set_erf_mode(0)
    t0 = time.perf_counter()
    orc.formal_solve_fo2_origins(origins, nthreads=nthreads)
    dt = time.perf_counter() - t0
    solves = len(origins) * per_origin
    return {"solves_per_s": solves / dt, "cores": nthreads, "kind": "port",
            "sample": f"every {stride}th origin ({len(origins)}) x all ray pairs x all frequencies ({solves} "
                      f"solves), {dt:.2f} s"}


class _Handle:
    """A core.Model's device handle with the sizes the batch wrapper reads."""

    def __init__(self, model):
        import ctypes as C
        prm = model.parameters
        self.h = C.c_void_p(model.upload())
        self.P, self.F, self.L, self.R = prm.npoints(), prm.nfreqs(), prm.nlines(), prm.hnrays()


def run_batch(args):
    """Many-model batch: independent models (sphere cutouts, P log-uniform in
    [2k, 60k], 12 or 48 rays, 2-5-level rotors, nquads 11/21/31, random T and v)
    solved by one persistent launch per step."""
    import numpy as np
    import torch
    from magritte_gb300 import _abi, loader, synthetic

    t_setup = time.perf_counter()
    specs = synthetic.many_models(args.batch_models)
    models, devs = [], []
    for sp in specs:
        m = loader.to_core(synthetic.batch_model(**sp), precision=args.precision)
        m.compute_spectral_discretisation()
        m.compute_inverse_line_widths()
        m.compute_LTE_level_populations()
        models.append(m)
        devs.append(_Handle(m))
    setup_s = time.perf_counter() - t_setup
    dev = torch.device("cuda", torch.cuda.current_device())
    Js = [torch.empty(d.P * d.F, dtype=torch.float64, device=dev) for d in devs]
    Ls = [torch.empty(d.P * d.L, dtype=torch.float64, device=dev) for d in devs]
    solves = float(sum(d.P * d.R * d.F for d in devs))
    batch = _abi.Batch(devs)
    stream = torch.cuda.ExternalStream(batch.stream(), device=dev)
    jp, lp = [t.data_ptr() for t in Js], [t.data_ptr() for t in Ls]

    def solve(b):
        b.formal_solve_fo2_device(args.precision, jp, lp)

    # tile shape (CTAs per SM x warps per CTA), timed on a sample of 16 models; the
    # sample's runs also warm the kernels up
    ns = min(16, len(devs))
    sub = _abi.Batch(devs[:ns])
    sub_stream = torch.cuda.ExternalStream(sub.stream(), device=dev)
    best = None
    for minb in (2, 3, 4):
        for warps in (4, 8):
            try:
                sub.set_tuning(minb, warps)
            except _abi.MgrError:
                continue
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            sub.formal_solve_fo2_device(args.precision, jp[:ns], lp[:ns])  # first use of this shape
            e0.record(sub_stream)
            sub.formal_solve_fo2_device(args.precision, jp[:ns], lp[:ns])
            e1.record(sub_stream)
            sub_stream.synchronize()
            ms = e0.elapsed_time(e1)
            if best is None or ms < best[0]:
                best = (ms, minb, warps)
    sub.close()
    batch.set_tuning(best[1], best[2])
    stream.synchronize()
    launches0 = _abi.launch_count()
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
          for _ in range(args.batch_steps)]
    for a, b in ev:
        a.record(stream)
        solve(batch)
        b.record(stream)
    stream.synchronize()
    launches = _abi.launch_count() - launches0
    start, finish = batch.timings()
    step_ms = [a.elapsed_time(b) for a, b in ev]
    batch_s = sum(step_ms) / 1000.0 / len(step_ms)

    # one call per model (each call its own persistent launch) against a batch of the
    # same models, on a sample of 64 models
    ns = min(64, len(devs))
    lib = _abi.load()
    sub = _abi.Batch(devs[:ns])
    sub.set_tuning(best[1], best[2])
    sub_solves = float(sum(d.P * d.R * d.F for d in devs[:ns]))
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    sub.formal_solve_fo2_device(args.precision, jp[:ns], lp[:ns])
    _abi._check(lib.mgr_sync(devs[0].h))
    torch.cuda.ExternalStream(sub.stream(), device=dev).synchronize()
    sub_s = time.perf_counter() - t0
    sub.close()
    t0 = time.perf_counter()
    for d, j, l in zip(devs[:ns], jp[:ns], lp[:ns]):
        _abi._check(lib.mgr_formal_solve_fo2_device(d.h, _abi.PRECISION[args.precision], C_void(j), None,
                                                    C_void(l)))
    for d in devs[:ns]:
        _abi._check(lib.mgr_sync(d.h))
    seq_s = time.perf_counter() - t0
    batch.close()
    for m in models:
        m.release_device()
    lat = finish
    flight = finish - start
    pct = lambda x, q: float(np.percentile(x, q))
    return {"workload": f"{len(devs)} models, sphere cutouts P {min(d.P for d in devs)}-{max(d.P for d in devs)} "
                        f"(mean {np.mean([d.P for d in devs]):.0f}), 12/48 rays, 2-5-level rotors, nquads 11/21/31",
            "solves_per_step": solves, "value": solves / batch_s, "unit": UNIT, "ms_per_step": 1000 * batch_s,
            "steps": len(step_ms), "step_ms": step_ms, "gpu_launches": int(launches),
            "tuning": {"min_blocks_per_sm": best[1], "warps_per_block": best[2]},
            "latency_ms": {"p50": pct(lat, 50), "p99": pct(lat, 99), "max": float(lat.max()),
                           "definition": "model's last origin finished, since the launch began"},
            "in_flight_ms": {"p50": pct(flight, 50), "p99": pct(flight, 99),
                             "definition": "model's last origin finished minus its origin 0 started"},
            "sample_64": {"batch_solves_per_s": sub_solves / sub_s, "one_call_per_model_solves_per_s":
                          sub_solves / seq_s, "note": "host wall clock, first 64 models"},
            "setup_s": setup_s, "precision": args.precision}


def run_adjoint(args):
    """Differentiable new imager: the non-LTE sphere family at 100k points (LTE level
    populations), images of 256 x 256 pixels at inclinations 0, 45 and 90 degrees
    over 41 frequencies spanning +-20 km/s about the J=1-0 line; loss = sum of
    squared differences to the images of perturbed fields (velocity x (1 + 0.05 N),
    temperature x 1.1); gradients with respect to velocity, temperature, turbulence
    and abundance; checked against FP64 central differences (Richardson-extrapolated)
    along a random direction of each of 64 random points' parameters."""
    import numpy as np
    import torch
    from magritte_gb300 import adjoint, loader, synthetic

    t_setup = time.perf_counter()
    raw = synthetic.nlte_sphere(npoints=args.adjoint_points, nside=1)
    f0 = raw.linedata[0].frequency[0]
    dd = 20.0e3 / 2.99792458e8
    model = loader.to_core(raw, precision="fp64")
    model.compute_spectral_discretisation(f0 * (1 - dd), f0 * (1 + dd), 41)
    model.compute_inverse_line_widths()
    model.compute_LTE_level_populations()
    npx = args.adjoint_pixels
    imager = adjoint.NewImager(model, npx, npx)
    setup_s = time.perf_counter() - t_setup
    dev = dict(dtype=torch.float64, device="cuda")
    rng = np.random.default_rng(0)
    v0 = torch.tensor(raw.velocity, **dev)
    T0 = torch.tensor(raw.temperature, **dev)
    vt0 = torch.tensor(raw.vturb2, **dev)
    ab0 = torch.tensor(raw.abundance, **dev)
    dirs = [adjoint.inclination_direction(a) for a in (0.0, 45.0, 90.0)]
    with torch.no_grad():
        vt = v0 * (1.0 + 0.05 * torch.tensor(rng.normal(size=(raw.npoints, 1)), **dev))
        targets = [imager(d, vt, T0 * 1.10, vt0, ab0) for d in dirs]

    def loss_of(v, T, vtu, ab):
        return sum(((imager(d, v, T, vtu, ab) - t) ** 2).sum() for d, t in zip(dirs, targets))

    # warm-up, then timed forward and forward + backward
    params = [t.clone().requires_grad_(True) for t in (v0, T0, vt0, ab0)]
    loss_of(*params).backward()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    with torch.no_grad():
        loss_of(v0, T0, vt0, ab0)
    torch.cuda.synchronize()
    fwd_s = time.perf_counter() - t0
    params = [t.clone().requires_grad_(True) for t in (v0, T0, vt0, ab0)]
    t0 = time.perf_counter()
    loss = loss_of(*params)
    loss.backward()
    torch.cuda.synchronize()
    fb_s = time.perf_counter() - t0
    grads = [p.grad.detach() for p in params]
    # finite-difference check on random interior points
    interior = np.setdiff1d(np.arange(raw.npoints), raw.boundary2point)
    pts = rng.choice(interior, size=min(args.adjoint_fd_points, len(interior)), replace=False)
    errs, flips, worst, t_fd = [], 0, [], time.perf_counter()
    for p in pts:
        dirv = [torch.zeros_like(t) for t in (v0, T0, vt0, ab0)]
        u = rng.normal(size=6)
        dirv[0][p] = torch.tensor(u[:3], **dev) * 1e-4 * v0.abs().max()
        dirv[1][p] = u[3] * 1e-4 * T0[p]
        dirv[2][p] = u[4] * 1e-4 * vt0[p]
        dirv[3][p, 0] = u[5] * 1e-4 * ab0[p, 0]
        an = sum(float((g * dv).sum()) for g, dv in zip(grads, dirv))

        def central(eps):
            with torch.no_grad():
                lp = loss_of(*[t + eps * dv for t, dv in zip((v0, T0, vt0, ab0), dirv)])
                lm = loss_of(*[t - eps * dv for t, dv in zip((v0, T0, vt0, ab0), dirv)])
            return float(lp - lm) / (2 * eps)

        # Richardson estimates from steps (1, 1/2) and (1/2, 1/4): where they disagree the
        # steps straddle a branch of the held structure (large-shift test, line bracket),
        # where the trace-fixed derivative and the differences of the full forward part
        # ways, and the point is counted, not compared; otherwise the finer estimate is
        # the reference
        c1, c2, c4 = central(1.0), central(0.5), central(0.25)
        r1, r2 = (4.0 * c2 - c1) / 3.0, (4.0 * c4 - c2) / 3.0
        if abs(r1 - r2) > 1e-5 * abs(r2):
            flips += 1
        elif r2 != 0.0:
            errs.append(abs(an - r2) / abs(r2))
            worst.append((errs[-1], int(p), an, r2, r1))
    fd_s = time.perf_counter() - t_fd
    solves = float(npx * npx * 41 * len(dirs))
    return {"workload": f"nlte_sphere {raw.npoints} points (LTE), {npx}x{npx} pixels x 41 frequencies "
                        f"(+-20 km/s), inclinations 0/45/90 deg",
            "forward_s": fwd_s, "forward_backward_s": fb_s,
            "forward_pixel_freq_solves_per_s": solves / fwd_s,
            "forward_backward_pixel_freq_solves_per_s": solves / fb_s,
            "fd_check": {"points": len(errs), "branch_crossings_skipped": flips,
                         "max_rel_err": max(errs) if errs else None,
                         "median_rel_err": float(np.median(errs)) if errs else None, "bar": 1e-4,
                         "worst": [dict(zip(("rel_err", "point", "adjoint", "fd", "fd_coarse"), w))
                                   for w in sorted(worst, reverse=True)[:3]],
                         "method": "Richardson-extrapolated central differences (steps 1, 1/2, 1/4) along a "
                                   "random direction of each point's (v_x, v_y, v_z, T, vturb2, abundance)",
                         "s": fd_s},
            "setup_s": setup_s, "loss": float(loss.detach())}


def run_adjoint_j(args):
    """Differentiable formal solve: the benchmarked grid-sphere family reduced to about
    100k points (n = 58), J of every origin as a smooth function of the per-point
    velocity, temperature, turbulence and abundance (LTE level populations, frequencies
    following the line widths); loss = sum of squared differences of J to the J of
    perturbed fields (velocity x (1 + 0.05 N), temperature x 1.1).  Forward and
    forward + backward are timed over every origin.  The gradients are checked against
    FP64 central differences at 64 random interior points, each on a loss localised to
    the point and its neighbours (a random weighting of their J rows), along a random
    direction of the point's six parameters: Richardson extrapolation of the steps
    (1, 1/2) and (1/2, 1/4); a point whose two extrapolations differ by more than 1e-5
    has a held branch inside the steps and is counted, not compared."""
    import numpy as np
    import torch
    from magritte_gb300 import adjoint, loader, synthetic

    t_setup = time.perf_counter()
    raw = synthetic.grid_sphere(n=args.adjoint_j_n)
    model = loader.to_core(raw, precision="fp64")
    model.compute_spectral_discretisation()
    model.compute_inverse_line_widths()
    model.compute_LTE_level_populations()
    solver = adjoint.FormalSolver(model)
    setup_s = time.perf_counter() - t_setup
    dev = dict(dtype=torch.float64, device="cuda")
    rng = np.random.default_rng(0)
    v0 = torch.tensor(raw.velocity, **dev)
    T0 = torch.tensor(raw.temperature, **dev)
    vt0 = torch.tensor(raw.vturb2, **dev)
    ab0 = torch.tensor(raw.abundance, **dev)
    with torch.no_grad():
        vt = v0 * (1.0 + 0.05 * torch.tensor(rng.normal(size=(raw.npoints, 1)), **dev))
        target = solver(vt, T0 * 1.10, vt0, ab0)

    def loss_of(v, T, vtu, ab):
        return ((solver(v, T, vtu, ab) - target) ** 2).sum()

    params = [t.clone().requires_grad_(True) for t in (v0, T0, vt0, ab0)]
    loss_of(*params).backward()  # warm-up
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    with torch.no_grad():
        loss_of(v0, T0, vt0, ab0)
    torch.cuda.synchronize()
    fwd_s = time.perf_counter() - t0
    params = [t.clone().requires_grad_(True) for t in (v0, T0, vt0, ab0)]
    t0 = time.perf_counter()
    loss = loss_of(*params)
    loss.backward()
    torch.cuda.synchronize()
    fb_s = time.perf_counter() - t0
    # finite-difference check on localised losses
    interior = np.setdiff1d(np.arange(raw.npoints), raw.boundary2point)
    pts = rng.choice(interior, size=min(args.adjoint_fd_points, len(interior)), replace=False)
    cum = np.concatenate([np.zeros(1, np.int64), np.cumsum(raw.n_neighbors, dtype=np.int64)])
    errs, flips, worst, t_fd = [], 0, [], time.perf_counter()
    for p in pts:
        S = np.unique(np.concatenate([[p], raw.neighbors[cum[p]:cum[p + 1]]])).astype(np.int32)
        orig = torch.tensor(S, dtype=torch.int32, device="cuda")
        w = torch.tensor(rng.normal(size=(len(S), solver.F)), **dev)
        rows = torch.tensor(S, dtype=torch.long, device="cuda")

        def local(v, T, vtu, ab):
            return (solver(v, T, vtu, ab, origins=orig)[rows] * w).sum()

        prm = [t.clone().requires_grad_(True) for t in (v0, T0, vt0, ab0)]
        local(*prm).backward()
        grads = [q.grad.detach() for q in prm]
        dirv = [torch.zeros_like(t) for t in (v0, T0, vt0, ab0)]
        u = rng.normal(size=6)
        dirv[0][p] = torch.tensor(u[:3], **dev) * 1e-4 * v0.abs().max()
        dirv[1][p] = u[3] * 1e-4 * T0[p]
        dirv[2][p] = u[4] * 1e-4 * vt0[p]
        dirv[3][p, 0] = u[5] * 1e-4 * ab0[p, 0]
        an = sum(float((g * dv).sum()) for g, dv in zip(grads, dirv))

        def central(eps):
            with torch.no_grad():
                lp = local(*[t + eps * dv for t, dv in zip((v0, T0, vt0, ab0), dirv)])
                lm = local(*[t - eps * dv for t, dv in zip((v0, T0, vt0, ab0), dirv)])
            return float(lp - lm) / (2 * eps)

        # Richardson estimates from steps (1, 1/2) and (1/2, 1/4): where they disagree the
        # steps straddle a held branch (large-shift test, line bracket) and the point is
        # skipped; otherwise the better estimate is the reference
        c1, c2, c4 = central(1.0), central(0.5), central(0.25)
        r1, r2 = (4.0 * c2 - c1) / 3.0, (4.0 * c4 - c2) / 3.0
        if abs(r1 - r2) > 1e-5 * abs(r2):
            flips += 1
        elif r2 != 0.0:
            errs.append(abs(an - r2) / abs(r2))
            worst.append((errs[-1], int(p), an, r2, r1))
    fd_s = time.perf_counter() - t_fd
    solves = float(raw.npoints) * (raw.nrays // 2) * solver.F
    return {"workload": f"grid_sphere {args.adjoint_j_n}^3 cutout ({raw.npoints} points), {raw.nrays} rays, "
                        f"5-level rotor (4 lines) x nquads {raw.nquads}, LTE",
            "forward_s": fwd_s, "forward_backward_s": fb_s,
            "forward_solves_per_s": solves / fwd_s, "forward_backward_solves_per_s": solves / fb_s,
            "fd_check": {"points": len(errs), "branch_crossings_skipped": flips,
                         "max_rel_err": max(errs) if errs else None,
                         "median_rel_err": float(np.median(errs)) if errs else None, "bar": 1e-4,
                         "worst": [dict(zip(("rel_err", "point", "adjoint", "fd", "fd_coarse"), w))
                                   for w in sorted(worst, reverse=True)[:3]],
                         "method": "Richardson-extrapolated central differences (steps 1, 1/2, 1/4) of a random weighting of the J "
                                   "rows of the point and its neighbours, along a random direction of the point's "
                                   "(v_x, v_y, v_z, T, vturb2, abundance)", "s": fd_s},
            "setup_s": setup_s, "loss": float(loss.detach())}


def C_void(x):
    import ctypes as C
    return C.c_void_p(x)


def run_reference(args, rank, ws):
    if rank != 0:
        return
    raw, desc = workload(args)
    nthreads = os.cpu_count() or 1
    oracle, orc, origins, solves = cpu_sample(raw)
    oracle.set_erf_mode(0)  # the reference's glibc erff
    for _ in range(args.warmup):
        orc.formal_solve_fo2_origins(origins, nthreads=nthreads)
    times = []
    for _ in range(args.steps):
        t0 = time.perf_counter()
        orc.formal_solve_fo2_origins(origins, nthreads=nthreads)
        times.append(time.perf_counter() - t0)
    total = sum(times)
    value = solves * args.steps / total
    sample = _sample_desc(origins, solves)
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1000 * total / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic", "config": {"workload": desc, "precision": "reference FP64 (CPU)"},
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": nthreads, "kind": "port", "sample": sample},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def run_ours(args, rank, ws):
    import ctypes as C

    import numpy as np
    import torch

    from magritte_gb300 import _abi, loader

    raw, desc = workload(args)
    model = loader.to_core(raw, precision=args.precision)
    model.compute_spectral_discretisation()
    model.compute_inverse_line_widths()
    model.compute_LTE_level_populations()
    lib = _abi.load()
    handle = C.c_void_p(model.upload())
    prm = model.parameters
    P, F, R, L = prm.npoints(), prm.nfreqs(), prm.hnrays(), prm.nlines()
    prec = _abi.PRECISION[args.precision]

    from magritte_gb300 import distributed

    dev = torch.device("cuda", torch.cuda.current_device())
    stream = torch.cuda.ExternalStream(lib.mgr_model_stream(handle), device=dev)
    packed = torch.empty(P * F + P * L, dtype=torch.float64, device=dev)  # [J | ALO diagonal]
    J = packed[:P * F].view(P, F)
    lam = packed[P * F:].view(P, L)
    flush = torch.empty(512 * 1024 * 1024 // 4, dtype=torch.float32, device=dev)  # > 129 MB L2
    tuning = None if args.no_autotune else {p: _abi.autotune(handle, p) for p in sorted({args.precision, "fp64"})}
    rr0, rr1 = distributed.ray_shard(R, rank, ws)
    if ws > 1 and rr1 <= rr0:
        raise SystemExit(f"{ws} ranks for {R} ray pairs: every rank needs at least one")

    def step():
        if ws == 1:
            rc = lib.mgr_formal_solve_fo2_device(handle, prec, C.c_void_p(J.data_ptr()), None,
                                                 C.c_void_p(lam.data_ptr()))
        else:
            rc = lib.mgr_formal_solve_fo2_rays_device(handle, prec, rr0, rr1, C.c_void_p(J.data_ptr()),
                                                      C.c_void_p(lam.data_ptr()))
        if rc != 0:
            raise RuntimeError(lib.mgr_last_error().decode())
        if ws > 1:
            import torch.distributed as dist
            dist.all_reduce(packed, op=dist.ReduceOp.SUM)  # on the current (the model's) stream

    with torch.cuda.stream(stream):
        for _ in range(args.warmup):
            step()
        stream.synchronize()
        _abi._check(lib.mgr_sync(handle))

        ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
        launches0 = _abi.launch_count()
        clocks = Clocks()
        barrier(ws)
        torch.cuda.synchronize()
        clocks.start()
        t_wall0 = time.perf_counter()
        for i in range(args.steps):
            flush.zero_()
            ev[i][0].record(stream)
            step()
            ev[i][1].record(stream)
        stream.synchronize()
        torch.cuda.synchronize()
        barrier(ws)
        wall = time.perf_counter() - t_wall0
        clk = clocks.stop()
        launches = _abi.launch_count() - launches0
        _abi._check(lib.mgr_sync(handle))
    step_ms = [a.elapsed_time(b) for a, b in ev]
    kernel_s = sum(step_ms) / 1000.0
    kernel_s = max_over_ranks(kernel_s, ws)
    solves = float(P) * R * F
    value = solves * args.steps / kernel_s  # the whole job solves one model per step

    # the trace's FP32 filter against the exact FP64 walk on every half ray of the model
    tr_rays, tr_steps, tr_bad = C.c_uint64(), C.c_uint64(), C.c_uint64()
    _abi._check(lib.mgr_trace_self_check(handle, C.byref(tr_rays), C.byref(tr_steps), C.byref(tr_bad)))
    trace_check = {"half_rays": tr_rays.value, "steps": tr_steps.value, "mismatched_half_rays": tr_bad.value,
                   "method": "mgr_trace_self_check: every (origin, ray) walked with the FP32 filter and with the "
                             "exact FP64 argmin; point sequences, edges and dZ compared bit for bit"}

    # work statistics for the algorithmic-bytes roofline
    st_steps, st_nbr, st_elem = C.c_uint64(), C.c_uint64(), C.c_uint64()
    _abi._check(lib.mgr_ray_statistics(handle, C.byref(st_steps), C.byref(st_nbr), C.byref(st_elem)))
    alg_bytes = 28.0 * (st_steps.value + st_nbr.value) + 52.0 * st_elem.value + 32.0 * solves
    alg_bytes *= (rr1 - rr0) / R  # this rank's share of the ray pairs
    mean_launch_s = kernel_s / args.steps
    achieved = alg_bytes / mean_launch_s / 1e9
    peaks_path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(peaks_path):
        peak = json.load(open(peaks_path))["hbm_gbs"]
        peak_src = "measured"
    else:
        peak, peak_src = 6800.0, "fallback"

    # accuracy of this precision against the FP64 path on the full workload
    J_ref = torch.empty_like(J)
    lam_ref = torch.empty_like(lam)
    with torch.cuda.stream(stream):
        rc = lib.mgr_formal_solve_fo2_device(handle, _abi.PRECISION["fp64"], C.c_void_p(J_ref.data_ptr()), None,
                                             C.c_void_p(lam_ref.data_ptr()))
        if rc != 0:
            raise RuntimeError(lib.mgr_last_error().decode())
        step()
        stream.synchronize()
    max_rel = float(((J - J_ref).abs() / J_ref.abs()).max().item())
    gpu_rows = None
    if ws == 1 and not args.no_parity:
        gpu_rows = {"fp64": (J_ref.cpu().numpy(), lam_ref.cpu().numpy())}
        if args.precision != "fp64":
            gpu_rows[args.precision] = (J.cpu().numpy(), lam.cpu().numpy())
    # plain FP64 GPU throughput on the same workload (the comparison path)
    fp64_ms = None
    if args.precision != "fp64":
        with torch.cuda.stream(stream):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            flush.zero_()
            e0.record(stream)
            rc = lib.mgr_formal_solve_fo2_device(handle, _abi.PRECISION["fp64"], C.c_void_p(J_ref.data_ptr()),
                                                 None, None)
            e1.record(stream)
            stream.synchronize()
        fp64_ms = e0.elapsed_time(e1)

    # end to end through the public API: fresh upload, solve, read-back of J and the ALO
    e2e = None
    if not args.no_e2e and ws > 1:
        # sharded: core.Model.upload, this rank's ray pairs, the allreduce, read-back
        e2e_times = []
        for _ in range(max(1, min(args.steps, 3))):
            model.release_device()
            torch.cuda.synchronize()
            barrier(ws)
            t0 = time.perf_counter()
            h = model.upload()
            Jd, ld = distributed.formal_solve_fo2_handle(h, P, F, L, R, args.precision)
            Jh, lh = Jd.cpu(), ld.cpu()
            e2e_times.append(time.perf_counter() - t0)
        h2d = (P * 3 * 8 * 2 + len(raw.neighbors) * 4 + P * 4 * 3 + P * F * 8 + 4 * P * L * 8 + P * 8 * 3
               + F * 4 * 4 + F)
        d2h = P * F * 8 + P * L * 8
        e2e_s = max_over_ranks(sum(e2e_times) / len(e2e_times), ws)
        e2e = {"value": solves / e2e_s, "unit": UNIT, "h2d_bytes_per_step": int(h2d),
               "d2h_bytes_per_step": int(d2h), "s_per_step": e2e_s,
               "path": "core.Model.upload + distributed.formal_solve_fo2_handle (ray-pair shard + NCCL "
                       "allreduce) + J/ALO read-back"}
    elif not args.no_e2e:
        prm.store_u = False
        h2d = (P * 3 * 8 * 2 + len(raw.neighbors) * 4 + P * 4 * 3 + P * F * 8 + 4 * P * L * 8 + P * 8 * 3
               + F * 4 * 4 + F)
        d2h = P * F * 8 + P * L * 8

        def e2e_leg(prec):
            """compute_radiation_field_feautrier_order_2 with a fresh upload each step, and
            its parts: the upload alone, then the call on the resident model."""
            prm.precision = prec
            model.release_device()
            model.compute_radiation_field_feautrier_order_2()  # warm the host paths
            times = []
            for _ in range(max(1, min(args.steps, 3))):
                model.release_device()
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                model.compute_radiation_field_feautrier_order_2()
                times.append(time.perf_counter() - t0)
            model.release_device()
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            model.upload()
            torch.cuda.synchronize()
            t_up = time.perf_counter() - t0
            t0 = time.perf_counter()
            model.compute_radiation_field_feautrier_order_2()
            t_call = time.perf_counter() - t0
            e_s = max_over_ranks(sum(times) / len(times), ws)
            return {"value": solves / e_s, "unit": UNIT, "h2d_bytes_per_step": int(h2d),
                    "d2h_bytes_per_step": int(d2h), "s_per_step": e_s, "precision": prec,
                    "breakdown_s": {"upload (host set-up, copies, tables, ray sizing)": t_up,
                                    "call on the resident model (line-data refresh, solve, read-back)": t_call},
                    "path": "core.Model.compute_radiation_field_feautrier_order_2 (upload + solve + J/ALO "
                            "read-back)"}

        e2e = e2e_leg(args.precision)
        if args.precision != "fp64":
            e2e["fp64"] = e2e_leg("fp64")
        prm.precision = args.precision

    if rank != 0:
        return
    parity = parity_sample(raw, gpu_rows) if gpu_rows is not None else None
    rates = pipe_rates()
    # FP64-pipe roofline: the FP64 thread operations the algorithm needs per launch (the
    # elimination's five per element and frequency; per trace step the exact Zn of the
    # chosen point and Z += Zn - Z (10) and the Doppler shift (11): the FP32 filter picks
    # the points, the exact argmin's 14 per neighbour record runs on the few steps it
    # leaves) over the launch time, against the measured FP64 pipe rate
    fp64_ops = (5.0 * st_elem.value * prm.nquads() + 21.0 * st_steps.value) * (rr1 - rr0) / R
    fp64_peak = rates["dfma"]["thread_ops_per_s"]
    roofline_fp64 = {"bound": "fp64", "achieved": fp64_ops / mean_launch_s, "peak": fp64_peak,
                     "unit": "FP64 thread-ops/s", "frac": fp64_ops / mean_launch_s / fp64_peak,
                     "algorithmic_ops_per_launch": fp64_ops, "peak_source": "measured (mgr_measure_pipe_rate, DFMA)",
                     "note": "algorithmic FP64 ops = 5 per element-frequency (projective elimination row) + 21 per "
                             "trace step (exact Zn and Z of the point the FP32 filter chose, Doppler shift); the pipe "
                             "is busy 16 cycles per warp instruction whatever the active lanes"}
    ali = None if args.no_ali else run_ali(args)
    batch = None if args.no_batch else run_batch(args)
    adj = None if args.no_adjoint else run_adjoint(args)
    adj_j = None if args.no_adjoint_j else run_adjoint_j(args)
    cpu = None
    if not args.no_cpu_baseline:
        cpu = cpu_baseline(raw, os.cpu_count() or 1)
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": ws, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": 1000.0 * kernel_s / args.steps, "higher_is_better": True,
        "scaling": "strong" if ws > 1 else "weak",
        "vs_baseline": None, "dtype": "f32+f64" if args.precision == "split" else "f64", "data": "synthetic",
        "config": {"workload": desc, "npoints": P, "ray_pairs": R, "nfreqs": F, "precision": args.precision,
                   "approx": "CloseLines", "solves_per_step": solves, "l2": "flushed between steps (512 MB write)",
                   "parallelism": f"ray-pair shards x{ws} + NCCL sum-allreduce" if ws > 1 else "1 GPU",
                   "ray_pairs_rank0": [rr0, rr1]},
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                     "traffic": TRAFFIC_BYTES_PER_SOLVE * solves * (rr1 - rr0) / R,
                     "traffic_note": "DRAM read + write bytes per launch from an ncu capture of the staged solve kernel "
                                     "on the 33^3 case (4870.5 MB for 50.8 M solves; ncu flushes the caches between "
                                     "its passes; the kernel that walks the half rays is not in it), scaled by the "
                                     "solves of this launch: the half rays read and the u / L_diag staging written "
                                     "are proportional to solves",
                     "peak_source": peak_src,
                     "algorithmic_bytes_per_launch": alg_bytes,
                     "note": "algorithmic bytes = 28 per trace step and per neighbour record + 52 per ray-pair "
                             "element + 32 per solve"},
        "roofline_fp64": roofline_fp64,
        "cpu_baseline": cpu,
        "e2e": e2e,
        "gpu_launches": int(launches),
        "clocks": clk,
        "wall_s_timed": wall,
        "step_ms": step_ms,
        "max_rel_err_J_vs_fp64_gpu": max_rel,
        "max_rel_err_J_vs_oracle": (max(parity[f"{args.precision}_J_vs_oracle_erf_cr"],
                                        parity[f"{args.precision}_J_vs_oracle_erf_glibc"]) if parity else None),
        "parity": parity,
        "trace_self_check": trace_check,
        "pipe_rates": rates,
        "fp64_gpu_solves_per_s": (solves / (fp64_ms / 1000.0)) if fp64_ms else None,
        "speedup_vs_fp64_gpu": (fp64_ms / (1000.0 * kernel_s / args.steps)) if fp64_ms else None,
        "work": {"trace_steps": st_steps.value, "neighbour_reads": st_nbr.value, "elements": st_elem.value},
        "tuning": tuning,
        "ali": ali,
        "batch": batch,
        "adjoint": adj,
        "adjoint_j": adj_j,
    }
    print(json.dumps(line), flush=True)


def main():
    args = parse()
    if args.ali_full:
        args.ali_points, args.ali_nside = 500_000, 4
    rank, ws = dist_init()
    if args.impl == "reference":
        run_reference(args, rank, ws)
    else:
        run_ours(args, rank, ws)
    if ws > 1:
        import torch.distributed as dist
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
