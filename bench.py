#!/usr/bin/env python
"""
Benchmark of the DFT-D4 dispersion path: energy + forces, structures/s.

Workload (N = 1): ``batch512`` -- 512 structures, N ~ U[8, 200] atoms padded
to 200, 12 elements (H 0.45, C 0.30, others 0.025), density 0.01 atoms/Bohr^3,
total charges in {-1, 0, +1}, BJ parameters s6=1, s8=1.2, a1=0.4, a2=5,
s9=1, float64, seed 1.  One step = energies and forces of the whole batch.

Lines printed by rank 0 (one JSON line):

* ``value``: structures/s of the precision form with inputs resident in HBM
  (device-timed fused energy + gradient call, L2 flushed between steps);
  the plain FP64 kernels are timed on the same workload beside it
  (``plain_fp64``), and both are compared with the float64 oracle;
* ``e2e``: the same metric through the public API ``dftd4()`` + autograd,
  with pinned host inputs copied in and energies / forces copied out every
  step;
* ``roofline``: the dominant kernel (ATM), algorithmic flops per launch
  divided by its CUDA-event duration in the timed steps, against the FP32
  FMA peak measured in this run;
* ``cpu_baseline``: the float64 CPU oracle on a bounded sample;
* ``large16k``: one 16000-atom structure in the precision form (pair / ATM
  cutoffs 50 / 25 Bohr), seconds per energy + force evaluation and stage
  times (``--no-large`` skips it).
* ``diff256``: 256 structures with energies, forces and parameter gradients,
  D4 and D4S, precision form against the plain FP64 kernels;
* ``serving``: the 20000-request stream through the continuous-batching
  server in real time (structures/s, p50 / p99 latency) and saturated, for
  the precision form and the plain FP64 kernels (``--serve-requests 0``
  skips it).

``--impl reference`` times the CPU restatement of tad-dftd4 (the oracle) on
the host cores for the same workload and metric.
"""

from __future__ import annotations

import argparse
import ctypes
import importlib
import json
import os
import subprocess
import sys
import threading
import time
from pathlib import Path

import numpy as np

REPO = Path(__file__).resolve().parent
sys.path.insert(0, str(REPO))

METRIC = "energy+force structures/s"
UNIT = "structures/s"
ATM_FLOPS_PER_TRIPLE = 180.0  # forward 60 + backward 120 (flop convention of the path)
PAIR_FLOPS = 92.0 + 30.0


def parse_args():
    ap = argparse.ArgumentParser(description=__doc__.split("\n\n")[0])
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=("ours", "reference"), default="ours")
    ap.add_argument("--nstruct", type=int, default=512)
    ap.add_argument("--e2e-steps", type=int, default=None)
    ap.add_argument("--cpu-seconds", type=float, default=15.0)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-large", action="store_true",
                    help="skip the one-structure 16000-atom measurement")
    ap.add_argument("--large-n", type=int, default=0,
                    help="only run the large-structure measurement, with this many "
                         "atoms (no FP64 check), and print its JSON")
    ap.add_argument("--serve-requests", type=int, default=20000,
                    help="requests of the serving stream (0 skips it)")
    ap.add_argument("--serve-plain-requests", type=int, default=3000,
                    help="requests of the saturated plain-FP64 serving run")
    return ap.parse_args()


def dist_setup(ngpus: int):
    import torch

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch.distributed as dist

        backend = "nccl" if torch.cuda.is_available() else "gloo"
        dist.init_process_group(backend=backend)
    if torch.cuda.is_available():
        torch.cuda.set_device(local)
    return world, rank, local


def barrier(world):
    if world > 1:
        import torch.distributed as dist

        dist.barrier()


def max_over_ranks(x: float, world: int) -> float:
    if world == 1:
        return x
    import torch
    import torch.distributed as dist

    t = torch.tensor([x], dtype=torch.float64,
                     device="cuda" if torch.cuda.is_available() else "cpu")
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def structure_counts(numbers: np.ndarray, positions: np.ndarray, cut2: float, cut3: float):
    """Unordered pairs within cut2 and triples with >= 2 sides within cut3."""
    pairs = 0
    triples = 0
    for z, r in zip(numbers, positions):
        real = z != 0
        rr = r[real]
        n = len(rr)
        if n < 2:
            continue
        d = np.sqrt(((rr[:, None, :] - rr[None, :, :]) ** 2).sum(-1))
        np.fill_diagonal(d, np.inf)
        pairs += int((d <= cut2).sum()) // 2
        m = (d <= cut3).astype(np.float64)
        deg = m.sum(1)
        tri = np.trace(m @ m @ m) / 6.0
        triples += int(round((deg * (deg - 1) / 2).sum() - 2 * tri))
    return pairs, triples


class ClockSampler:
    """nvidia-smi clock / throttle samples while the timed region runs."""

    QUERY = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.lines: list[str] = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.QUERY}",
                 "--format=csv,noheader,nounits", "-lms", "100"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except (FileNotFoundError, OSError):
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in self.lines:
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx = float(parts[2])
            except ValueError:
                continue
            for name, flag in zip(names, parts[5:9]):
                if flag.lower().startswith("active"):
                    reasons.add(name)
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": mx,
                "reasons": sorted(reasons), "samples": len(sm)}


def cpu_oracle_rate(batch, param, seconds: float, threads: int):
    """Structures/s of the float64 CPU oracle (energy + autograd forces)."""
    import torch

    import oracle

    torch.set_num_threads(threads)
    order = np.random.default_rng(0).permutation(len(batch.numbers))
    done, t0, sizes = 0, time.perf_counter(), []
    for k in order:
        z = batch.numbers[k]
        n = int((z != 0).sum())
        nt = torch.from_numpy(z[:n])
        pt = torch.from_numpy(batch.positions[k, :n])
        oracle.dftd4_energy_and_grad(nt, pt, torch.tensor(float(batch.charge[k])), param)
        done += 1
        sizes.append(n)
        if time.perf_counter() - t0 >= seconds and done >= 3:
            break
    dt = time.perf_counter() - t0
    return done / dt, done, dt, sizes


def oracle_errors(batch, param, energy: np.ndarray, grad: np.ndarray, count: int = 3):
    """Max |dE| per structure and max |dF| against the oracle on a few structures."""
    import torch

    import oracle

    sizes = (batch.numbers != 0).sum(-1)
    order = np.argsort(sizes)
    pick = sorted(set(order[: count - 1].tolist() + [int(order[-1])]))
    de, df = 0.0, 0.0
    for k in pick:
        n = int(sizes[k])
        nt = torch.from_numpy(batch.numbers[k, :n])
        pt = torch.from_numpy(batch.positions[k, :n])
        e_ref, g_ref = oracle.dftd4_energy_and_grad(nt, pt, torch.tensor(float(batch.charge[k])),
                                                    param)
        de = max(de, abs(float(energy[k, :n].sum() - e_ref.sum())))
        df = max(df, float(np.abs(grad[k, :n] - g_ref.numpy()).max()))
    return {"structures_checked": [int(k) for k in pick], "max_abs_dE_eh": de,
            "max_abs_dF_eh_bohr": df}


def run_reference(args, world, rank):
    """--impl reference: the CPU restatement on the host cores."""
    if rank != 0:
        return
    pkg = importlib.import_module("tad-dftd4_gb300")
    batch = pkg.workloads.batch512(1, args.nstruct)
    param = dict(pkg.workloads.BJ_PARAMS)
    threads = os.cpu_count() or 1
    per_step = max(1.0, args.cpu_seconds / max(1, args.steps))
    for _ in range(args.warmup):
        cpu_oracle_rate(batch, param, 0.0, threads)
    rates, total_n, total_t = [], 0, 0.0
    for _ in range(args.steps):
        rate, n, dt, _ = cpu_oracle_rate(batch, param, per_step, threads)
        rates.append(rate)
        total_n += n
        total_t += dt
    value = total_n / total_t
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT,
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": 1e3 * total_t / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": "batch512: 512 structures, N~U[8,200] padded to 200, "
                               "12 elements, density 0.01/Bohr^3, charges {-1,0,1}, seed 1",
                   "model": "D4", "step": "bounded sample of the batch per step"},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port",
                         "sample": f"{total_n} structures drawn from the batch, "
                                   f"energy + autograd forces, torch float64 CPU"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def time_steps(lib, pkg, runner, positions, steps, flush, timing: bool):
    """Per-step CUDA-event times of the fused energy + gradient call."""
    import torch

    nstage = lib.d4_stage_count()
    starts = [torch.cuda.Event(enable_timing=True) for _ in range(steps)]
    ends = [torch.cuda.Event(enable_timing=True) for _ in range(steps)]
    if timing:
        pkg._lib.check(lib.d4_timing_begin(steps), "timing")
    for k in range(steps):
        flush.zero_()
        starts[k].record()
        runner.run(positions, gradient=True)
        ends[k].record()
    torch.cuda.synchronize()
    stages = None
    if timing:
        ms_stage = (ctypes.c_float * nstage)()
        ncalls = ctypes.c_int32(0)
        pkg._lib.check(lib.d4_timing_end(ms_stage, nstage, ncalls), "timing")
        stages = {lib.d4_stage_name(i).decode(): ms_stage[i] / max(1, ncalls.value)
                  for i in range(nstage)}
    return [s.elapsed_time(e) for s, e in zip(starts, ends)], stages


def probe_peak(lib, pkg, dev, fp64: bool) -> float:
    """Best of three FMA-chain probes, TFLOP/s."""
    import torch

    blocks, iters = 152 * 8, (4096 if fp64 else 65536)
    sink = torch.empty(blocks * 256, dtype=torch.float64, device=dev)
    ms = ctypes.c_float(0.0)
    best = 0.0
    for _ in range(3):
        pkg._lib.check(lib.d4_probe_fma(int(fp64), blocks, iters, sink.data_ptr(), ms,
                                        torch.cuda.current_stream(dev).cuda_stream), "probe")
        best = max(best, blocks * 256 * iters * 8 * 2 / (ms.value * 1e-3) / 1e12)
    return best


# Kernels of one precision-form energy + gradient call of the D4 model with
# EEQ charges on structures that fit the one-CTA EEQ and have no neighbour
# lists (N <= 234): prep with the element tables, size order, CN, EEQ (matrix
# and solve), weights, pair (tensor-core C6), ATM (task plan, triples, mirror
# of the pair sums), ATM / C6 adjoint (tensor cores), EEQ adjoint, CN adjoint,
# finish.
KERNELS_PER_CALL = 13


def run_large(pkg, disp, lib, dev, steps: int = 3, natoms: int = 16000,
              fp64_check: bool = True):
    """One large structure (16000 atoms by default; H/C/N/O/S, density 0.01,
    neutral, pair and ATM cutoffs 50 / 25 Bohr), precision form, energy +
    forces: milliseconds per structure and per-stage times (the inputs, 10 GB
    of workspace at 16000 atoms, are far larger than L2).  Then the errors
    against a float64 reference of the same structure (the neighbour-list
    restatement of the oracle, run on the GPU as the checker; not timed) and
    the EEQ residual of the returned charges in float64."""
    import torch

    batch = pkg.workloads.large16k(2, natoms)
    n = batch.numbers.shape[1]
    nt, pt, ct = (torch.from_numpy(x).to(dev) for x in (batch.numbers, batch.positions,
                                                        batch.charge))
    cutoff = pkg.Cutoff(disp2=50.0, disp3=25.0)
    param = dict(pkg.workloads.BJ_PARAMS)
    runner, _, _ = disp._prepare(nt, pt, ct, param, "d4", None, None, None, None, cutoff,
                                 None, None, None, "mixed")
    runner.run(pt, gradient=True)
    torch.cuda.synchronize()
    nstage = lib.d4_stage_count()
    pkg._lib.check(lib.d4_timing_begin(steps), "timing")
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(steps + 1)]
    ev[0].record()
    for k in range(steps):
        e, g, _, _, _ = runner.run(pt, gradient=True)
        ev[k + 1].record()
    torch.cuda.synchronize()
    ms_stage = (ctypes.c_float * nstage)()
    ncalls = ctypes.c_int32(0)
    pkg._lib.check(lib.d4_timing_end(ms_stage, nstage, ncalls), "timing")
    ms = [ev[k].elapsed_time(ev[k + 1]) for k in range(steps)]
    fsum = g[0].sum(0).abs().max().item()
    res = runner.eeq_residuals()  # final refinement residuals of the last timed call
    _, _, _, q, _ = runner.run(pt, gradient=False, charges_out=True)
    torch.cuda.synchronize()
    out = {
        "workload": f"large{natoms // 1000}k: 1 structure, N={natoms} H/C/N/O/S "
                    "(0.45/0.3/0.1/0.1/0.05), density 0.01/Bohr^3, neutral, seed 2, "
                    "cutoffs disp2=50 disp3=25",
        "method": "precision form, energy + forces",
        "ms_per_structure": float(np.median(ms)), "structures_per_s": 1e3 / float(np.median(ms)),
        "atom_pairs_per_s": n * (n - 1) / 2 / (float(np.median(ms)) * 1e-3),
        "stage_ms": {lib.d4_stage_name(i).decode(): ms_stage[i] / max(1, ncalls.value)
                     for i in range(nstage)},
        "energy_eh": float(e.sum()),
        "max_abs_sum_of_forces_eh_bohr": fsum,
        "eeq_refinement_residual": {"charges": float(res[0, 0]), "adjoint": float(res[0, 1]),
                                    "tolerance": 1e-10},
        "peak_device_gb": torch.cuda.max_memory_allocated(dev) / 1e9,
    }
    e_prod = e[0].detach().clone()
    g_prod = g[0].detach().clone()
    q_prod = q[0].detach().clone()
    del runner, e, g, q
    torch.cuda.empty_cache()
    if fp64_check:
        out["error_vs_fp64_reference"] = large_fp64_errors(nt[0], pt[0], e_prod, g_prod,
                                                           q_prod, param)
    return out


def large_fp64_errors(numbers, positions, e_prod, g_prod, q_prod, param):
    """|dE|, max |dF| and the charges' EEQ residual of a large structure
    against the float64 neighbour-list restatement (oracle/d4_nbr.py),
    evaluated on the GPU; checker only, outside every timed region."""
    import torch

    from oracle import d4_nbr

    t0 = time.perf_counter()
    cutoff = {"disp2": 50.0, "disp3": 25.0}
    e_ref, g_ref, extra = d4_nbr.dftd4_large(numbers, positions, 0.0, param, cutoff=cutoff)
    res_prod = d4_nbr.eeq_residual(numbers, positions, 0.0, q_prod)
    res_ref = d4_nbr.eeq_residual(numbers, positions, 0.0, extra["q"])
    out = {
        "reference": "float64 neighbour-list restatement of the oracle (dense pair terms, "
                     "factorised C6, ATM over neighbour triples, dense float64 EEQ solve), "
                     "cross-checked against the dense oracle in tests/test_oracle_nbr.py",
        "abs_dE_total_eh": abs(float(e_prod.sum() - e_ref.sum())),
        "max_abs_dE_atom_eh": float((e_prod - e_ref).abs().max()),
        "max_abs_dF_eh_bohr": float((g_prod - g_ref).abs().max()),
        "max_abs_dq": float((q_prod - extra["q"]).abs().max()),
        "eeq_residual_precision_form": res_prod,
        "eeq_residual_fp64_solve": res_ref,
        "energy_fp64_eh": float(e_ref.sum()),
        "atm_triples": extra["triples"],
        "checker_seconds": time.perf_counter() - t0,
    }
    del e_ref, g_ref, extra
    torch.cuda.empty_cache()
    return out


def run_diff(pkg, disp, dev, steps: int = 5):
    """The differentiation form: 256 structures, N ~ U[20, 150] padded to
    150, 12 elements, neutral, with the damping parameters drawn for the
    first structure (s8, a1, a2; s6 = s9 = 1), energies + forces + the
    gradient with respect to (s6, s8, a1, a2, s9) in one call, D4 and D4S,
    precision form; structures/s and the largest differences to the plain
    FP64 kernels on the same inputs."""
    import torch

    batch, params = pkg.workloads.diff256(3)
    param = params[0]
    nt, pt, ct = (torch.from_numpy(x).to(dev) for x in (batch.numbers, batch.positions,
                                                        batch.charge))
    B = nt.shape[0]
    out = {"workload": "diff256: 256 structures, N~U[20,150] padded to 150, 12 elements, "
                       "neutral, seed 3; energy + forces + parameter gradients",
           "params": param}
    for model in ("d4", "d4s"):
        runs = {}
        for precision in ("mixed", "fp64"):
            r, _, _ = disp._prepare(nt, pt, ct, param, model, None, None, None, None, None,
                                    None, None, None, precision)
            res = r.run(pt, gradient=True, param_grad=True)
            torch.cuda.synchronize()
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            ev[0].record()
            for _ in range(steps):
                res = r.run(pt, gradient=True, param_grad=True)
            ev[1].record()
            torch.cuda.synchronize()
            ms = ev[0].elapsed_time(ev[1]) / steps
            runs[precision] = (ms, res)
        (ms_m, rm), (ms_p, rp) = runs["mixed"], runs["fp64"]
        out[model] = {
            "precision_form_structures_per_s": B / (ms_m * 1e-3),
            "plain_fp64_structures_per_s": B / (ms_p * 1e-3),
            "max_abs_dE_eh": (rm[0].sum(-1) - rp[0].sum(-1)).abs().max().item(),
            "max_abs_dF_eh_bohr": (rm[1] - rp[1]).abs().max().item(),
            "max_rel_dparam": ((rm[2][:, :7].sum(0) - rp[2][:, :7].sum(0)).abs() /
                               rp[2][:, :7].sum(0).abs().clamp(min=1e-12)).max().item(),
        }
    return out


def run_serving(pkg, param, nreq: int, plain_nreq: int):
    """The serving form: a Poisson stream of ``nreq`` single-structure
    energy + force requests at 2000 req/s, log-normal sizes (median 60 atoms,
    sigma 1.0) clipped to [5, 4000], 12 elements, charges in {-1, 0, 1},
    through the continuous-batching server (CUDA graphs per size bucket,
    40 GB HBM budget).  Every request of a given size uses the one seeded
    structure generated for that size.  Reported: the real-time stream
    (structures/s, p50 / p99 latency) and the saturated throughput of the
    precision form and of the plain FP64 kernels on the same requests."""
    import torch

    sv = importlib.import_module("tad-dftd4_gb300.serving")
    wl = pkg.workloads
    sizes, arrivals = wl.stream_sizes(4, nreq)
    rng = np.random.default_rng(5)
    charges = rng.integers(-1, 2, size=nreq).astype(np.float64)
    pool = {int(n): wl.structure(40000 + int(n), int(n)) for n in np.unique(sizes)}
    reqs = [sv.Request(k, pool[int(n)][0], pool[int(n)][1], float(charges[k]), float(t))
            for k, (n, t) in enumerate(zip(sizes, arrivals))]
    out = {"workload": f"stream: {nreq} requests, Poisson at 2000 req/s, log-normal sizes "
                       "(median 60, sigma 1.0) in [5, 4000], 12 elements, seed 4",
           "server": "continuous batching, CUDA graph per (bucket, batch size), "
                     "max_wait 1 ms, HBM budget 40 GB"}
    res = {}
    for precision, count, realtime in (("mixed", nreq, True), ("mixed", nreq, False),
                                       ("fp64", plain_nreq, False)):
        srv = sv.Server(param, precision=precision, max_wait=1e-3, hbm_budget=40e9)
        srv.warmup()
        torch.cuda.synchronize()
        sub = reqs[:count]
        if not realtime:
            sub = [sv.Request(r.rid, r.numbers, r.positions, r.charge, 0.0) for r in sub]
        results, stats = sv.serve_stream(srv, sub, realtime=realtime)
        key = ("realtime_" if realtime else "saturated_") + precision
        out[key] = {k: stats[k] for k in ("requests", "structures_per_s", "atoms_per_s",
                                          "p50_ms", "p99_ms", "max_ms", "batches", "failed")}
        res[key] = results
        del srv
        torch.cuda.empty_cache()
    m, f = res["saturated_mixed"], res["saturated_fp64"]
    out["precision_vs_plain_max_abs_dE_eh"] = max(abs(m[k].energy - f[k].energy)
                                                  for k in range(plain_nreq))
    out["precision_vs_plain_max_abs_dF_eh_bohr"] = max(
        float(np.abs(m[k].gradient - f[k].gradient).max()) for k in range(plain_nreq))
    out["speedup_saturated_precision_vs_plain"] = (out["saturated_mixed"]["structures_per_s"] /
                                                   out["saturated_fp64"]["structures_per_s"])
    return out


def run_ours(args, world, rank, local):
    import torch

    pkg = importlib.import_module("tad-dftd4_gb300")
    disp = importlib.import_module("tad-dftd4_gb300.disp")
    lib = pkg._lib.load()
    dev = torch.device("cuda", local)
    batch = pkg.workloads.batch512(1, args.nstruct)
    param = dict(pkg.workloads.BJ_PARAMS)
    B, N = batch.numbers.shape
    numbers = torch.from_numpy(batch.numbers).to(dev)
    positions = torch.from_numpy(batch.positions).to(dev)
    charge = torch.from_numpy(batch.charge).to(dev)

    def make_runner(precision):
        r, _, _ = disp._prepare(numbers, positions, charge, param, "d4", None, None, None,
                                None, None, None, None, None, precision)
        return r

    mixed = make_runner("mixed")
    plain = make_runner("fp64")
    flush = torch.empty(256 * 1024 * 1024, dtype=torch.uint8, device=dev)
    disp.CHECK_STATUS = False
    for _ in range(args.warmup):
        mixed.run(positions, gradient=True)
        plain.run(positions, gradient=True)
    torch.cuda.synchronize()

    # ---- device-resident timed region: the precision form (headline)
    barrier(world)
    torch.cuda.synchronize()
    with ClockSampler(local) as clocks:
        step_ms, _ = time_steps(lib, pkg, mixed, positions, args.steps, flush, False)
    barrier(world)
    total_s = max_over_ranks(sum(step_ms) / 1e3, world)
    value = world * B * args.steps / total_s
    # the stage split in a pass of its own: its events sit between the kernels,
    # where they hold back the next kernel's early launch
    _, stages = time_steps(lib, pkg, mixed, positions, max(3, min(args.steps, 10)), flush, True)

    # ---- the plain FP64 kernels on the same workload (comparison point)
    plain_steps = max(3, min(args.steps, 10))
    plain_ms, plain_stages = time_steps(lib, pkg, plain, positions, plain_steps, flush, True)
    plain_total = max_over_ranks(sum(plain_ms) / 1e3, world)
    plain_value = world * B * plain_steps / plain_total

    # ---- error of both forms against the float64 oracle
    disp.CHECK_STATUS = True
    e_m, g_m, _, _, _ = mixed.run(positions, gradient=True)
    e_p, g_p, _, _, _ = plain.run(positions, gradient=True)
    err_m = oracle_errors(batch, param, e_m.cpu().numpy(), g_m.cpu().numpy())
    err_p = oracle_errors(batch, param, e_p.cpu().numpy(), g_p.cpu().numpy())
    e_all = (e_m.sum(-1) - e_p.sum(-1)).abs().max().item()
    f_all = (g_m - g_p).abs().max().item()
    res_m = mixed.eeq_residuals()  # final refinement residuals of that call

    # ---- end to end through the public API, host buffers
    e2e_steps = args.e2e_steps or max(3, args.steps // 2)
    h_num = torch.from_numpy(batch.numbers).pin_memory()
    h_pos = torch.from_numpy(batch.positions).pin_memory()
    h_chg = torch.from_numpy(batch.charge).pin_memory()
    h_e = torch.empty((B, N), dtype=torch.float64).pin_memory()
    h_g = torch.empty((B, N, 3), dtype=torch.float64).pin_memory()

    def e2e_step():
        d_num = h_num.to(dev, non_blocking=True)
        d_pos = h_pos.to(dev, non_blocking=True).requires_grad_(True)
        d_chg = h_chg.to(dev, non_blocking=True)
        energy = pkg.dftd4(d_num, d_pos, d_chg, param, precision="mixed")
        (grad,) = torch.autograd.grad(energy.sum(), d_pos)
        h_e.copy_(energy.detach(), non_blocking=True)
        h_g.copy_(grad, non_blocking=True)
        torch.cuda.synchronize()

    for _ in range(2):
        e2e_step()
    lat = []
    barrier(world)
    for _ in range(e2e_steps):
        flush.zero_()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        e2e_step()
        lat.append(time.perf_counter() - t0)
    e2e_total = max_over_ranks(sum(lat), world)
    e2e_value = world * B * e2e_steps / e2e_total
    h2d = h_num.numel() * 8 + h_pos.numel() * 8 + h_chg.numel() * 8
    d2h = h_e.numel() * 8 + h_g.numel() * 8

    # ---- roofline of the dominant kernel (ATM, FP32 arithmetic)
    pairs, triples = structure_counts(batch.numbers, batch.positions, 60.0, 40.0)
    fp32_peak = probe_peak(lib, pkg, dev, fp64=False)
    fp64_peak = probe_peak(lib, pkg, dev, fp64=True)
    top = max(stages, key=stages.get)
    atm_ms = stages["atm"]
    achieved = ATM_FLOPS_PER_TRIPLE * triples / (atm_ms * 1e-3) / 1e12
    plain_achieved = ATM_FLOPS_PER_TRIPLE * triples / (plain_stages["atm"] * 1e-3) / 1e12
    traffic = {}
    tfile = REPO / "profiles" / "traffic.txt"
    if tfile.exists():
        for line in tfile.read_text().splitlines():
            parts = line.split()
            if len(parts) >= 2 and not line.startswith("#"):
                traffic[parts[0]] = float(parts[1])
    peaks = {}
    pfile = REPO / "MEASURED_PEAKS.json"
    if pfile.exists():
        peaks = json.loads(pfile.read_text())

    # ---- CPU baseline (rank 0, bounded sample)
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        threads = os.cpu_count() or 1
        rate, n, dt, sizes = cpu_oracle_rate(batch, param, args.cpu_seconds, threads)
        cpu = {"value": rate, "unit": UNIT, "cores": threads, "kind": "port",
               "sample": f"{n} structures of the batch (mean N {np.mean(sizes):.0f}), "
                         f"energy + autograd forces, float64 torch CPU oracle, {dt:.1f} s"}

    large = None
    if rank == 0 and not args.no_large:
        large = run_large(pkg, disp, lib, dev)
    diff = run_diff(pkg, disp, dev) if rank == 0 and not args.no_large else None
    serve = None
    if rank == 0 and args.serve_requests > 0:
        serve = run_serving(pkg, param, args.serve_requests,
                            min(args.serve_plain_requests, args.serve_requests))

    clk = clocks.summary()
    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": total_s * 1e3 / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32+f64", "data": "synthetic",
            "config": {
                "workload": "batch512: 512 structures, N~U[8,200] padded to 200, 12 elements, "
                            "density 0.01/Bohr^3, charges {-1,0,1}, seed 1",
                "model": "D4", "method": "precision form (FP32 pair/triple maths, "
                                         "compensated sums, FP32 EEQ + FP64 refinement)",
                "global_batch": B, "n_pad": N,
                "params": param, "cutoffs": {"disp2": 60.0, "disp3": 40.0, "cn_eeq": 25.0},
                "l2": "flushed between steps (256 MiB write)",
                "parallelism": f"replicas x{world}",
            },
            "atom_pairs_per_s": world * pairs * args.steps / total_s,
            "latency_ms": {"p50": float(np.percentile(step_ms, 50)),
                           "p99": float(np.percentile(step_ms, 99))},
            "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": h2d,
                    "d2h_bytes_per_step": d2h,
                    "latency_ms": {"p50": 1e3 * float(np.percentile(lat, 50)),
                                   "p99": 1e3 * float(np.percentile(lat, 99))},
                    "api": "dftd4(precision='mixed') + torch.autograd.grad, pinned host buffers"},
            "roofline": {
                "kernel": "atm32_kernel<GRAD> (FP32 arithmetic)", "bound": "fp32",
                "achieved": achieved, "peak": fp32_peak, "unit": "TFLOP/s",
                "frac": achieved / fp32_peak if fp32_peak else None,
                "traffic": traffic.get("atm32_batch512"),
                "peak_source": "FP32 FMA-chain probe (d4_probe_fma) measured in this run; "
                               "MEASURED_PEAKS.json holds only HBM and bf16 peaks",
                "algorithmic": f"{ATM_FLOPS_PER_TRIPLE:.0f} flop x {triples} triples per launch",
                "avg_launch_ms": atm_ms,
                "hbm_peak_gbs": peaks.get("hbm_gbs"),
            },
            "stage_ms": stages, "top_stage": top,
            "gpu_launches": KERNELS_PER_CALL * args.steps,
            "clocks": {k: clk[k] for k in ("sm_mhz", "sm_max_mhz", "reasons")},
            "cpu_baseline": cpu,
            "large16k": large,
            "diff256": diff,
            "serving": serve,
            # last, so that a record that keeps only the end of the line keeps them
            "plain_fp64": {"value": plain_value, "unit": UNIT,
                           "ms_per_step": plain_total * 1e3 / plain_steps,
                           "speedup_of_precision_form": value / plain_value,
                           "stage_ms": plain_stages,
                           "atm_achieved_tflops": plain_achieved, "fp64_peak_tflops": fp64_peak},
            "error_vs_fp64_oracle": err_m,
            "error_plain_fp64_vs_oracle": err_p,
            "error_precision_vs_plain_all_structures": {"max_abs_dE_eh": e_all,
                                                        "max_abs_dF_eh_bohr": f_all},
            "eeq_refinement_residual_max": {"charges": float(res_m[:, 0].max()),
                                            "adjoint": float(res_m[:, 1].max()),
                                            "tolerance": 1e-10},
            "large16k_error_vs_fp64": (large or {}).get("error_vs_fp64_reference"),
            "large16k_eeq_refinement_residual": (large or {}).get("eeq_refinement_residual"),
        }
        print(json.dumps(line), flush=True)


def main():
    args = parse_args()
    world, rank, local = dist_setup(args.gpus)
    if args.large_n > 0:
        import torch

        pkg = importlib.import_module("tad-dftd4_gb300")
        disp = importlib.import_module("tad-dftd4_gb300.disp")
        out = run_large(pkg, disp, pkg._lib.load(), torch.device("cuda", local),
                        steps=max(1, args.steps), natoms=args.large_n, fp64_check=False)
        print(json.dumps(out), flush=True)
        return
    if args.impl == "reference":
        run_reference(args, world, rank)
    else:
        run_ours(args, world, rank, local)
    if world > 1:
        import torch.distributed as dist

        dist.destroy_process_group()


if __name__ == "__main__":
    main()
