#!/usr/bin/env python
"""Benchmark of the B200 sweep: person-steps/s of whole CovidSim realisations.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Workload (default, --workload c1_240): 10,000,000 synthetic people on a 2 x 2 degree
region of 240 x 240 cells (10 x 10 microcells each, lognormal density), household /
age / four place types from the generator, power-law spatial kernel, R0 = 2.4, 100
seed infections, 365 days at 0.25-day steps, with the global ICU-trigger
interventions (case isolation 0.7, household quarantine 0.5, school/university
closure, social distancing) switched on for 90 days.  The 240 x 240 grid is the
largest whose dense cell tables the reference can hold, so the reference arm runs
the same population; the config's own 600 x 600 grid is measured in the same run
(the c1_600x600 key).  One "step" of this benchmark is one whole realisation (1460
model timesteps, InfectSweep + IncubRecoverySweep each); K timed realisations run
after W untimed ones, each with its own seed.

value = people x timesteps x realisations (all ranks) / device time (max over
ranks), timed with CUDA events on the sweep's own stream.  The population (0.6 GB
of structure plus dynamic state) is far larger than L2, so no flush is needed.
e2e runs the realisations through the drop-in (the reference executable with the
GPU sweep linked in) on the reference arm's network file, timing the sweep calls as
the reference arm does, with the state upload at each realisation's start, the
waits for the device and the copies back inside; e2e_python_host repeats them
through the C ABI from host buffers.  Multi-GPU (torchrun) runs independent
realisations per rank (replicas, weak scaling): only the barrier and the max of the
timings cross ranks.

--impl reference times the reference's own CPU sweep (oracle/_ref/CovidSim_timed,
built from the reference sources by oracle/Makefile) on this host's cores, on the
same 10M people: one warm-up realisation at most and at most three timed ones
(about 40 s of run loop each).
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
sys.path.insert(0, os.path.join(ROOT, "covid-sim_b200"))

import numpy as np  # noqa: E402

WORKLOADS = {
    # name: (preset, days, interventions, description, initial infections)
    "c1": ("c1", 365, True, "10M people, 600x600 cells, interventions, 365 d", 100),
    "c0": ("c0", 120, False, "1M people, 240x240 cells, no interventions, 120 d", 100),
    # the same 10M people on the 240x240 grid (coarser cells, as the reference's
    # own grid limit would force)
    "c1_240": ("c1_240", 365, True, "10M people, 240x240 cells, interventions, 365 d", 100),
    # a short case whose sweeps run at epidemic-peak load after a few hundred
    # launches: the profiling case for the spatial and place kernels
    "c1_peak": ("c1", 8, False, "10M people, 600x600 cells, 500k initial infections, 8 d", 500000),
    # 66 M people, 1500x1500 cells, 30 urban blobs, 100 admin units whose triggers
    # fire on their own admissions (staggered)
    "c3": ("c3", 365, "adunit", "66M people, 1500x1500 cells, 100 admin units, staggered triggers, 365 d", 100),
}
METRIC = "person-steps/s"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="c1_240", choices=sorted(WORKLOADS) + ["c2", "c4"])
    ap.add_argument("--no-extra", action="store_true",
                    help="skip the extra measurement of the 600x600-cell grid in the default run")
    ap.add_argument("--c2-scale", type=float, default=1.0,
                    help="c2 only: population sizes times this factor (1.0 = 1/4/10/20 M)")
    ap.add_argument("--c2-per-size", type=int, default=16, help="c2 only: realisations per population size")
    ap.add_argument("--c2-days", type=int, default=365, help="c2 only: days per realisation")
    ap.add_argument("--c4-train", type=int, default=2500, help="c4 only: training scenarios")
    ap.add_argument("--c4-seeds", type=int, default=8, help="c4 only: seeds per training scenario")
    ap.add_argument("--c4-epochs", type=int, default=800, help="c4 only: training epochs")
    ap.add_argument("--c4-sweep", type=int, default=100_000, help="c4 only: scenarios screened")
    ap.add_argument("--c4-rerun", type=int, default=1000, help="c4 only: top scenarios re-run by the simulator")
    ap.add_argument("--c4-ensemble", type=int, default=4, help="c4 only: networks averaged")
    ap.add_argument("--c4-check", type=int, default=100,
                    help="c4 only: scenarios drawn at random from the sweep to measure accuracy on")
    ap.add_argument("--c4-save", default=None, help="c4 only: write the simulated data sets to this .npz")
    ap.add_argument("--c4-people", type=int, default=1_000_000, help="c4 only: population size")
    ap.add_argument("--setup", default="host", choices=["host", "gpu"],
                    help="build the population with the host generator or the set-up kernels on the GPU")
    ap.add_argument("--population-cache", default=None,
                    help="directory keeping generated populations (.npz) for later runs")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--profile-out", default=None, help="write per-kernel times to this JSON file")
    ap.add_argument("--no-tune", action="store_true",
                    help="skip the launch-shape autotuner (use --lanes and --blocks-per-sm), so that the timed "
                         "realisation's k-th timestep is each kernel's k-th launch (profiling runs)")
    ap.add_argument("--lanes", type=int, default=2, help="with --no-tune: lanes per spatial contact")
    ap.add_argument("--blocks-per-sm", type=int, default=8, help="with --no-tune: blocks per SM of the sweep kernels")
    return ap.parse_args()


# ------------------------------------------------------------------- clocks
class ClockSampler:
    """nvidia-smi clock / throttle samples every 200 ms while the timed region runs."""
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device):
        self.device = device
        self.proc = None
        self.path = tempfile.mktemp(prefix="clocks_", suffix=".csv")

    def __enter__(self):
        try:
            self.f = open(self.path, "w")
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.device), "--query-gpu=" + self.FIELDS,
                                          "--format=csv,noheader,nounits", "-lms", "200"], stdout=self.f,
                                         stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None
        return self

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()
        self.f.close()

    def summary(self):
        sm, smax, reasons = [], None, set()
        try:
            for line in open(self.path):
                parts = [x.strip() for x in line.split(",")]
                if len(parts) < 9:
                    continue
                try:
                    sm.append(float(parts[1]))
                    smax = float(parts[2])
                except ValueError:
                    continue
                names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
                for name, v in zip(names, parts[5:9]):
                    if v.lower().startswith("active"):
                        reasons.add(name)
        except OSError:
            pass
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": smax, "reasons": sorted(reasons), "samples": len(sm)}


# ------------------------------------------------------------------ roofline
def peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        d = json.load(open(path))
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


def kernel_bytes(name, w, n_cells_steps):
    """Algorithmic bytes a kernel moved over the timed region, from the work counters
    (per-unit costs, the shared counting convention: transition scan 16 B per
    latent/infectious person -- the kernel itself reads 6 B of it, the list entry and
    the next-event time -- and 16 B per cell, infector record 40 B, household member 12 B, place candidate 20 B, spatial
    draw 33 B, accepted infection 24 B, infector-list entry 12 B, per-cell counts
    16 B)."""
    if name == "k_household":
        return 40 * w["work_infectors"] + 12 * w["work_hh_members"]
    if name == "k_places":
        return 20 * w["work_place_candidates"] + 16 * w["work_infectors"]
    if name == "k_spatial":
        return 33 * w["work_spatial_draws"]
    if name in ("k_apply_infections", "k_partition_S", "k_infections"):
        return 12 * w["work_new_infections"]
    if name == "k_scan":   # the infector list, the transition scan and the cells' counts, one pass
        return 12 * w["work_infectors"] + 16 * w["work_incub_people"] + 16 * n_cells_steps
    if name in ("k_onsets", "k_progress"):   # the transitions, counted once for the two
        return 16 * w["work_transitions"]
    if name == "k_moves":
        return 8 * w["work_transitions"] + 12 * w["work_new_infections"]
    return None


def load_traffic():
    """Per-unit DRAM traffic of the captured kernels from the committed ncu summary
    (bytes per work unit, e.g. per spatial contact), when present."""
    path = os.path.join(ROOT, "profiles", "ncu_traffic.json")
    try:
        return json.load(open(path))
    except Exception:
        return {}


# --------------------------------------------------------------------- ours
def replica_seed(rank):
    """Run seed of rank `rank`: every rank simulates its own realisations."""
    return 17389101 + 7919 * rank


def max_over_ranks(value, dist, device):
    """The largest of the ranks' values (the job's time is its slowest rank's)."""
    if dist is None:
        return value
    import torch
    t = torch.tensor([value], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def ensemble_share(n_members, rank, world):
    """Indices of the ensemble members rank `rank` simulates: every world-th one,
    so each rank gets the same mix of population sizes."""
    return list(range(rank, n_members, world))


def gather_series(local, n_members, rank, world, dist, device):
    """The ensemble's daily series on every rank: `local` is this rank's members'
    [members of the rank, days] array (ensemble_share order); the result is
    [n_members, days] in member order.  One all-gather (NCCL on the GPUs)."""
    local = np.asarray(local, np.float64)
    days = local.shape[1]
    if dist is None:
        return local
    import torch
    per = (n_members + world - 1) // world
    buf = np.zeros((per, days))
    buf[:len(local)] = local
    t = torch.tensor(buf, dtype=torch.float64, device=device)
    parts = [torch.empty_like(t) for _ in range(world)]
    dist.all_gather(parts, t)
    out = np.zeros((n_members, days))
    for r, part in enumerate(parts):
        idx = ensemble_share(n_members, r, world)
        out[idx] = part.cpu().numpy()[:len(idx)]
    return out


def run_ours(args):
    import torch
    rank = int(os.environ.get("RANK", 0))
    world = int(os.environ.get("WORLD_SIZE", 1))
    local = int(os.environ.get("LOCAL_RANK", 0))
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=900))
    else:
        torch.cuda.set_device(local)
    from covidsim_b200 import population, params as prm, sim

    preset, days, with_iv, desc, n_seed = WORKLOADS[args.workload]
    t_setup = time.perf_counter()
    if args.setup == "gpu":
        pop = population.cached(args.population_cache, preset + "_gpu", lambda: population.preset(preset, device=local))
    else:
        pop = population.cached(args.population_cache, preset, lambda: population.preset(preset))
    t_setup = time.perf_counter() - t_setup
    P, lk, hr = prm.build_params(pop.grid)
    beta, r0parts = sim.calibrate_local_beta(pop, P, 2.4)
    P.LocalBeta = beta
    s = sim.Simulation(pop, P, lk, hr, device=local)
    be = s.backend
    policy = (sim.InterventionPolicy(per_adunit=True) if with_iv == "adunit" else
              sim.InterventionPolicy() if with_iv else None)
    steps_per_run = int(days * P.TimeStepsPerDay)
    base_seed = replica_seed(rank)

    from covidsim_b200 import tune
    n_sm = torch.cuda.get_device_properties(local).multi_processor_count
    if args.no_tune:
        be.set_grid(n_sm * args.blocks_per_sm)
        be.set_spatial_lanes(args.lanes)
        tuned = {"grid": n_sm * args.blocks_per_sm, "spatial_lanes": args.lanes, "ms": None}
    else:
        tuned = tune.autotune(s, n_sm=n_sm)
    for w in range(args.warmup):
        s.run(seed=base_seed + 1000 + w, days=days, n_seed=n_seed, policy=policy)
    be.sync()

    def barrier():
        if dist:
            dist.barrier()
        torch.cuda.synchronize()

    stream = torch.cuda.ExternalStream(be.stream())
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    finals = []
    barrier()
    launches0 = be.launches()
    with ClockSampler(local) as clk:
        ev0.record(stream)
        for k in range(args.steps):
            ser = s.run(seed=base_seed + k, days=days, n_seed=n_seed, policy=policy)
            finals.append((int(ser["cumI"][-1]), int(ser["D"][-1]), int(ser["I"].argmax())))
        ev1.record(stream)
        be.sync()
        torch.cuda.synchronize()
    barrier()
    launches = be.launches() - launches0
    ms = ev0.elapsed_time(ev1)
    ms = max_over_ranks(ms, dist, "cuda")
    person_steps = pop.n_people * steps_per_run * args.steps * world
    value = person_steps / (ms / 1e3)
    runs_per_hour = args.steps * world / (ms / 1e3) * 3600.0

    # per-kernel device times: one more realisation of the same workload with every
    # launch bracketed by CUDA events on the sweep's stream (eager launches)
    be.profile(2)
    work_daily = []

    def _daily(step, c):
        work_daily.append({k: int(getattr(c, k)) for k in ("work_infectors", "work_hh_members", "work_place_candidates",
                                                            "work_spatial_contacts", "work_spatial_draws",
                                                            "work_new_infections", "work_transitions",
                                                            "work_incub_people")})
    s.run(seed=base_seed, days=days, n_seed=n_seed, policy=policy, callback=_daily)
    be.sync()
    kernels = be.profile_entries()
    be.profile(0)
    work = sim.abi.counters_to_dict(be.counters())
    prof_runs = 1

    # roofline of the dominant kernel
    peak, peak_kind = peaks()
    traffic = load_traffic()
    n_cells_steps = pop.n_cells * steps_per_run * prof_runs
    rows = []
    merged = {}
    for name, (kms, n) in kernels.items():          # k_spatial<8> and the like under one name
        base = name.split("<")[0]
        a = merged.get(base, (0.0, 0))
        merged[base] = (a[0] + kms, a[1] + n)
    kernels = merged
    for name, (kms, n) in sorted(kernels.items(), key=lambda kv: -kv[1][0]):
        b = kernel_bytes(name, work, n_cells_steps)
        rows.append(dict(kernel=name, ms=kms, launches=n, share=kms / sum(v[0] for v in kernels.values()),
                         bytes=b, gbs=(b / (kms / 1e3) / 1e9) if b else None))
    dom = rows[0]
    # ncu traffic of the same kernel, captured at peak load on the smaller profiling
    # case and scaled to this workload's average launch by the units it processed
    dom_traffic = None
    tr = traffic.get(dom["kernel"])
    if tr and work.get(tr["unit"]):
        dom_traffic = round(tr["dram_bytes_per_unit"] * work[tr["unit"]] / dom["launches"])
    roofline = {
        "bound": "hbm", "kernel": dom["kernel"], "achieved": round(dom["gbs"], 2) if dom["gbs"] else None,
        "peak": peak, "unit": "GB/s", "frac": round(dom["gbs"] / peak, 4) if dom["gbs"] else None,
        "traffic": dom_traffic, "peak_source": peak_kind + " (MEASURED_PEAKS.json hbm_gbs)" if peak_kind == "measured" else peak_kind,
        "algorithmic_bytes_per_launch": round(dom["bytes"] / dom["launches"]) if dom["bytes"] else None,
        "avg_launch_us": round(dom["ms"] / dom["launches"] * 1e3, 3),
        "share_of_kernel_time": round(dom["share"], 4),
        "timing": "CUDA events around each launch on the sweep's stream, over one extra realisation of the workload",
    }
    # the whole realisation: every kernel's algorithmic bytes over the timed time of one realisation
    total_bytes = sum(r["bytes"] for r in rows if r["bytes"])
    realisation_gbs = total_bytes / (ms / args.steps / 1e3) / 1e9
    roofline["realisation"] = {"algorithmic_bytes": int(total_bytes), "achieved": round(realisation_gbs, 2),
                               "frac": round(realisation_gbs / peak, 4),
                               "what": "sum of the kernels' algorithmic bytes in one realisation / ms_per_step"}
    if args.profile_out and rank == 0:
        json.dump(dict(rows=rows, work=work, work_daily=work_daily, timed_ms=ms, steps=args.steps,
                       workload=args.workload, profiled_runs=prof_runs, tuned=tuned),
                  open(args.profile_out, "w"), indent=1)

    # end to end through the reference-facing drop-in: the reference executable with
    # the GPU sweep linked in, on the same network file the reference arm loads
    # (the reference's own set-up and host code, the sweeps on this rank's GPU)
    e2e = None
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import refrun
    dropin = (not args.no_e2e) and refrun.SAMPLES.get(args.workload, {}).get("network")
    if dropin:
        e2e = e2e_dropin(args, local, world, dist, pop.n_cells)
    # end to end through the C ABI from host buffers (the Python host)
    e2e_py = None
    if not args.no_e2e:
        # the prepared start state (input) and the final state (output) in separate
        # pinned host buffers, so every realisation starts from the same input
        arrs, view = sim.state_arrays(pop.n_people, pop.n_cells)
        arrs_out, view_out = sim.state_arrays(pop.n_people, pop.n_cells)
        be.begin_run(base_seed, s.choose_seeds(base_seed, n_seed))
        be.download(view)
        cudart = torch.cuda.cudart()
        pinned = list(arrs.values()) + list(arrs_out.values())
        for a in pinned:
            cudart.cudaHostRegister(a.ctypes.data, a.nbytes, 0)
        state_bytes = sum(a.nbytes for a in arrs.values())
        barrier()
        t0 = time.perf_counter()
        for k in range(args.steps):
            s.run(seed=base_seed + k, days=days, n_seed=n_seed, policy=policy, initial_state=view)
            be.download(view_out)
        be.sync()
        barrier()
        dt = time.perf_counter() - t0
        dt = max_over_ranks(dt, dist, "cuda")
        for a in pinned:
            cudart.cudaHostUnregister(a.ctypes.data)
        import ctypes
        e2e_py = {"value": round(person_steps / dt, 1), "unit": METRIC, "h2d_bytes_per_step": state_bytes,
                  "d2h_bytes_per_step": state_bytes + days * ctypes.sizeof(sim.abi.cs_counters),
                  "what": "Python host through the C ABI: upload prepared start state, run, daily counters, "
                          "download final state"}
        if e2e is None:
            e2e = e2e_py

    # CPU baseline: the oracle port on a bounded sample of the same workload
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        cpu = cpu_baseline_port(s, pop, P, lk, hr, days)
    s.close()

    # the same measurement on the 600x600-cell grid of the 10M workload
    extra = None
    if args.workload == "c1_240" and not args.no_extra:
        extra = extra_600(args, local, world, dist)

    if dist:
        dist.barrier()
        dist.destroy_process_group()
    if rank != 0:
        return None
    clocks = clk.summary()
    return {
        "metric": METRIC, "value": round(value, 1), "unit": METRIC, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": round(ms / args.steps, 3), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64/f32 (f64 infection probabilities, f32 normaliser sums and person state)",
        "data": "synthetic (seeded generator, reference parameter set)",
        "config": {"workload": desc, "people": pop.n_people, "cells": pop.n_cells, "timesteps_per_step": steps_per_run,
                   "realisations_per_rank": args.steps, "parallelism": "replicas x%d" % world,
                   "l2": "inputs larger than L2 (%.0f MB resident)" % (pop.nbytes() / 1e6),
                   "local_beta": round(beta, 6), "r0_parts": {k: round(float(v), 4) for k, v in r0parts.items()},
                   "tuned": {"grid": tuned["grid"], "spatial_lanes": tuned["spatial_lanes"]},
                   "setup": {"kind": args.setup, "seconds": round(t_setup, 2),
                             "device_ms": round(pop.setup_info["device_ms"], 1) if pop.setup_info else None}},
        "runs_per_hour": round(runs_per_hour, 1),
        "outcomes": [{"cumI": a, "deaths": b, "peak_day": c} for a, b, c in finals],
        "clocks": clocks, "e2e": e2e, "e2e_python_host": e2e_py if e2e is not e2e_py else None,
        "c1_600x600": extra, "roofline": roofline, "cpu_baseline": cpu,
        "gpu_launches": int(launches),
        "kernels": [{k: (round(v, 4) if isinstance(v, float) else v) for k, v in r.items()} for r in rows[:8]],
    }


E2E_MAX_STEPS = 3   # realisations the drop-in's end-to-end figure times at most


def e2e_dropin(args, local, world, dist, n_cells):
    """e2e through the drop-in: warm-up 1 and up to three timed realisations of the
    reference executable with the GPU sweep linked in, loading the workload's
    network file; value = people x timesteps / wall time of the sweep calls (state
    upload at each realisation's start, the launch of every timestep's graph, the
    wait for the device at the last timestep of each output step -- the timesteps
    before it run on while the host runs TreatSweep --, the copy of the cell counts
    and counters back to the reference's host structures there, the hand-over of the
    host's interventions).  run_loop_ms_per_step is RunModel's whole loop per
    realisation, the host code between sweeps included."""
    import ctypes
    import refrun
    from covidsim_b200 import abi, sim
    # the host's thread count, as the reference arm: the reference's set-up, and so the
    # population the network file fits, depends on it
    # a realisation through the drop-in runs the reference's RunModel loop, about
    # 30 s of host code (TreatSweep's microcell loop) around 0.2 s of sweeps: at most
    # E2E_MAX_STEPS realisations are timed (one per rank when several ranks share the
    # host's cores), after one warm-up, so the run stays within a few minutes
    steps = max(1, min(args.steps, E2E_MAX_STEPS if world == 1 else 1))
    res = refrun.time_dropin(args.workload, steps=steps, warmup=1, device=local, threads=os.cpu_count())
    if "unavailable" in res:
        return {"unavailable": res["unavailable"]}
    rows = res["rows"]
    person_steps = sum(r["pop"] * r["steps"] for r in rows)
    secs = sum(r["infect_s"] + r["incub_s"] for r in rows)
    secs = max_over_ranks(secs, dist, "cuda")
    n, steps = rows[0]["pop"], rows[0]["steps"]
    arrs, _ = sim.state_arrays(n, n_cells)   # the grid's populated cells (every cell at 10M people)
    h2d = sum(a.nbytes for a in arrs.values())
    days = refrun.SAMPLES[args.workload]["days"]   # one copy back per output step (a day)
    # the cell counts travel as 16-bit values when every cell fits (cell_bytes 2)
    d2h = days * (5 * int(rows[0].get("cell_bytes", 4)) * n_cells + ctypes.sizeof(abi.cs_counters))
    parts = {k: round(1e3 * sum(r.get(k, 0.0) for r in rows) / len(rows), 3)
             for k in ("upload_s", "copyback_s", "wait_s", "scatter_s", "handover_s", "infect_s", "incub_s",
                       "upload_device_s")}
    scans = sum(r.get("mcell_scans", 0) for r in rows) / len(rows)
    return {"value": round(person_steps * world / secs, 1), "unit": METRIC, "h2d_bytes_per_step": h2d,
            "d2h_bytes_per_step": d2h, "ms_per_step": round(1e3 * secs / len(rows), 3),
            "ms_per_step_parts": {"state_upload": parts["upload_s"], "state_upload_device": parts["upload_device_s"],
                                  "copy_back": parts["copyback_s"],
                                  "copy_back_into_cells": parts["scatter_s"], "wait_for_device": parts["wait_s"],
                                  "handover_after_treatsweep": parts["handover_s"], "infect_calls": parts["infect_s"],
                                  "incub_calls": parts["incub_s"]},
            "handover_microcell_scans_per_step": scans,
            # RunModel's time stepping per realisation with the host code between the
            # sweeps (TreatSweep, RecordSample, output), beside the sweep calls alone
            "run_loop_ms_per_step": round(1e3 * sum(r.get("loop_s", 0.0) for r in rows) / len(rows), 3),
            "what": "the reference executable with the GPU sweep linked in (oracle/_ref/CovidSim_b200), the same "
                    "network file as the reference arm; wall time of the sweep calls per realisation: state upload "
                    "from the reference's host structures at its start, device sweeps (one graph per timestep; "
                    "the host waits for the device at the last timestep of each output step, the timesteps "
                    "before it run on while the host runs TreatSweep), copy of cell counts and counters back "
                    "at each output step, intervention hand-over; run_loop_ms_per_step is RunModel's whole "
                    "time stepping, the host code between sweeps included, as the reference arm reports it",
            "realisations": len(rows), "host_threads": rows[0]["threads"], "process_wall_s": round(res["wall"], 1),
            "network_file": res.get("network_file")}


def extra_600(args, local, world, dist):
    """value of the 10M workload on its own 600x600-cell grid (device time, 1 warm-up
    and 2 timed realisations)."""
    import torch
    from covidsim_b200 import population, params as prm, sim, tune
    preset, days, with_iv, desc, n_seed = WORKLOADS["c1"]
    pop = population.cached(args.population_cache, preset, lambda: population.preset(preset))
    P, lk, hr = prm.build_params(pop.grid)
    P.LocalBeta, _ = sim.calibrate_local_beta(pop, P, 2.4)
    s = sim.Simulation(pop, P, lk, hr, device=local)
    n_sm = torch.cuda.get_device_properties(local).multi_processor_count
    tuned = tune.autotune(s, n_sm=n_sm)
    policy = sim.InterventionPolicy()
    base_seed = replica_seed(int(os.environ.get("RANK", 0)))
    s.run(seed=base_seed + 999, days=days, n_seed=n_seed, policy=policy)
    stream = torch.cuda.ExternalStream(s.backend.stream())
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    ev0.record(stream)
    for k in range(2):
        s.run(seed=base_seed + k, days=days, n_seed=n_seed, policy=policy)
    ev1.record(stream)
    s.backend.sync()
    torch.cuda.synchronize()
    ms = max_over_ranks(ev0.elapsed_time(ev1), dist, "cuda")
    s.close()
    return {"workload": desc, "value": round(pop.n_people * int(days * P.TimeStepsPerDay) * 2 * world / (ms / 1e3), 1),
            "unit": METRIC, "ms_per_step": round(ms / 2, 3), "realisations_per_rank": 2,
            "tuned": {"grid": tuned["grid"], "spatial_lanes": tuned["spatial_lanes"]}}


def cpu_baseline_port(s, pop, P, lk, hr, days, budget_s=20.0):
    """The CPU oracle (a single-threaded C restatement of the sweep) timed on a
    bounded sample: a few timesteps around the epidemic peak of the same
    population, interventions off, started from the GPU's state at that day."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle_py
    from covidsim_b200 import sim
    seed = 4242
    be = s.backend
    be.begin_run(seed, s.choose_seeds(seed, 100))
    # advance on the GPU to the peak region of an intervention-free epidemic
    peak_day = None
    I_prev = -1
    for step in range(int(days * 4)):
        be.step(step * P.ModelTimeStep, 0)
        if step % 4 == 3:
            c = be.counters()
            if c.I < I_prev and c.I > 0.02 * pop.n_people:
                peak_day = (step + 1) // 4
                break
            I_prev = c.I
    start_step = step + 1
    arrs, view = sim.state_arrays(pop.n_people, pop.n_cells)
    be.download(view)
    o = oracle_py.OracleBackend(s._pop_c, P)
    o.upload(seed, view)
    n = 0
    t0 = time.perf_counter()
    while n < 40:
        o.step((start_step + n) * P.ModelTimeStep, 0)
        n += 1
        if time.perf_counter() - t0 > budget_s:
            break
    dt = time.perf_counter() - t0
    o.close()
    return {"value": round(pop.n_people * n / dt, 1), "unit": METRIC, "cores": 1, "kind": "port",
            "sample": "%d timesteps from day %s (epidemic peak, no interventions) of the same population, "
                      "oracle/cs_oracle.c single-threaded" % (n, peak_day)}


# ---------------------------------------------------------------- reference
REF_MAX_STEPS = 3   # realisations the reference arm times at most


def run_reference(args):
    rank = int(os.environ.get("RANK", 0))
    if rank != 0:
        return None
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import refrun
    if args.workload not in refrun.SAMPLES:
        return {"impl": "reference", "unavailable": "no reference sample defined for workload %s" % args.workload}
    # a CPU realisation needs no warm-up beyond touching its memory once: one
    # warm-up realisation at most.  A realisation of the 10M-person workload runs
    # about 40 s of RunModel's loop on the reference (10 s of it in the sweeps), so at
    # most REF_MAX_STEPS realisations are timed, which bounds the run to a few
    # minutes; the metric is a rate, per realisation
    steps = max(1, min(args.steps, REF_MAX_STEPS))
    res = refrun.time_reference(args.workload, steps=steps, warmup=min(args.warmup, 1))
    if "unavailable" in res:
        return {"impl": "reference", "unavailable": res["unavailable"]}
    preset, days, with_iv, desc, n_seed = WORKLOADS[args.workload]
    v = res["value"]
    return {
        "impl": "reference", "metric": METRIC, "value": round(v, 1), "unit": METRIC, "n_gpus": args.gpus,
        "steps": steps, "steps_requested": args.steps, "warmup": args.warmup, "ms_per_step": res["ms_per_step"],
        "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": desc, "reference_sample": res["sample"], "network_file": res.get("network_file"),
                   "process_wall_s": round(res["wall"], 1), "run_loop_ms_per_step": res.get("run_loop_ms_per_step")},
        "cpu_baseline": {"value": round(v, 1), "unit": METRIC, "cores": res["cores"], "kind": "reference",
                         "sample": res["sample"]},
        "e2e": {"value": round(v, 1), "unit": METRIC, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }


# ------------------------------------------------------------ batched ensemble
C2_SIZES = (1_000_000, 4_000_000, 10_000_000, 20_000_000)


def run_c2(args):
    """Ensemble of uneven populations stepped together (cs_gpu_batch): per size,
    `c2-per-size` realisations sharing that population's static device arrays,
    each with its own seed and R0 drawn uniformly in [1.8, 3.2], C1 interventions.
    One step = the whole ensemble for c2-days days, one CUDA graph per day.  Under
    torchrun the realisations are split across the ranks (every world-th member to
    each), the members' daily series are all-gathered at the end, and the time is the
    slowest rank's (strong scaling: the ensemble's size is fixed)."""
    import torch
    rank = int(os.environ.get("RANK", 0))
    world = int(os.environ.get("WORLD_SIZE", 1))
    local_rank = int(os.environ.get("LOCAL_RANK", 0))
    torch.cuda.set_device(local_rank)
    dist = None
    if world > 1:
        # the ensemble is split by realisation: each rank simulates its share, only
        # the timing and the final series cross ranks
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=900))
    from covidsim_b200 import population, params as prm, sim
    grid = population.make_grid(cell_deg=1.0 / 120, nmcl=10)
    rng = np.random.default_rng(2024)
    n_members = len(C2_SIZES) * args.c2_per_size
    mine = set(ensemble_share(n_members, rank, world))
    members, people, people_all, j = [], 0, 0, 0
    for size in C2_SIZES:
        n = int(size * args.c2_scale)
        draws = [float(rng.uniform(1.8, 3.2)) for _ in range(args.c2_per_size)]   # the same draws on every rank
        people_all += n * args.c2_per_size
        idx = [j + k for k in range(args.c2_per_size)]
        j += args.c2_per_size
        if not any(i in mine for i in idx):
            continue
        pop = population.cached(args.population_cache, "c2_%d" % n,
                                lambda n=n: population.generate(n, grid, sigma=1.2, seed=98798150 + n))
        P, lk, hr = prm.build_params(pop.grid)
        beta24, _ = sim.calibrate_local_beta(pop, P, 2.4)
        base = None
        for k, i in enumerate(idx):
            if i not in mine:
                continue
            Pk = type(P).from_buffer_copy(P)
            Pk.LocalBeta = beta24 * draws[k] / 2.4   # the coefficient scales R0 linearly
            if base is None:
                base = sim.Simulation(pop, Pk, lk, hr)
                members.append(base)
            else:
                members.append(base.replica(Pk))
            people += n
    order = sorted(mine)   # member indices of this rank, in the order of `members`
    if not members:
        raise SystemExit("c2: %d ranks for %d realisations leaves rank %d without any" % (world, n_members, rank))
    batch = sim.Batch(members)
    from covidsim_b200 import tune
    tuned = tune.autotune_batch(batch, n_sm=torch.cuda.get_device_properties(local_rank).multi_processor_count)
    days = args.c2_days
    policy = sim.InterventionPolicy()
    stream = torch.cuda.ExternalStream(batch.stream())
    for w in range(args.warmup):
        batch.run([9000 + 100 * w + i for i in order], min(days, 20), policy=policy)
    batch.sync()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    last = None
    if dist:
        dist.barrier()
    with ClockSampler(local_rank) as clk:
        ev0.record(stream)
        for k in range(args.steps):
            last = batch.run([17389101 + 1000 * k + i for i in order], days, policy=policy)
        ev1.record(stream)
        batch.sync()
        torch.cuda.synchronize()
    ms = max_over_ranks(ev0.elapsed_time(ev1), dist, "cuda")
    # the ensemble's daily cumulative infections, gathered from the ranks
    ens = gather_series(np.stack([o["cumI"] for o in last]), n_members, rank, world, dist, "cuda")
    finals = [int(ens[:, -1].sum())]
    steps_per_run = int(days * members[0].params.TimeStepsPerDay)
    person_steps = people_all * steps_per_run * args.steps
    nreal = n_members * args.steps
    batch.close()
    for m in members:
        m.close()
    if dist:
        dist.barrier()
        dist.destroy_process_group()
    if rank != 0:
        return None
    return {
        "metric": METRIC, "value": round(person_steps / (ms / 1e3), 1), "unit": METRIC, "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms / args.steps, 3),
        "higher_is_better": True, "scaling": "strong", "vs_baseline": None,
        "dtype": "f64/f32 (f64 infection probabilities, f32 normaliser sums and person state)",
        "data": "synthetic (seeded generator, reference parameter set)",
        "config": {"workload": "batched ensemble: %d realisations, %d each of %s people on 240x240 cells, "
                               "R0 ~ U[1.8, 3.2], interventions, %d d"
                               % (n_members, args.c2_per_size,
                                  "/".join("%g" % (x * args.c2_scale) for x in C2_SIZES), days),
                   "realisations_per_step": n_members, "people_total": people_all,
                   "timesteps_per_realisation": steps_per_run,
                   "parallelism": "realisations split across %d GPU(s), daily series all-gathered at the end; "
                                  "per GPU one graph per day, each kernel launched once for all of its "
                                  "realisations (one grid row each); static arrays shared per population" % world,
                   "tuned": tuned},
        "runs_per_hour": round(nreal / (ms / 1e3) * 3600.0, 1),
        "ensemble_new_infections": finals,
        "clocks": clk.summary(), "e2e": None, "gpu_launches": None,
    }


# -------------------------------------------------------- surrogate sweep
def run_c4(args):
    """Scenario sweep with the surrogate: simulate training scenarios (batched,
    several seeds each), train the network, screen the sweep, re-run the
    scenarios ranked best (lowest critical-care peak) with 8 seeds each, and
    report the network's error on those against the simulator's ensemble mean.
    The plain method (every sweep scenario simulated one realisation at a time
    with 8 seeds) is timed on a sample and extrapolated."""
    import torch
    torch.cuda.set_device(0)
    from covidsim_b200 import population, params as prm, sim, surrogate
    grid = population.make_grid(cell_deg=1.0 / 120, nmcl=10)
    pop = population.generate(args.c4_people, grid, sigma=1.2, seed=98798150)
    P, lk, hr = prm.build_params(pop.grid)
    t_all = time.perf_counter()
    # 1. training trajectories
    train = surrogate.sample_scenarios(args.c4_train, seed=101)
    t0 = time.perf_counter()
    idx, ys = surrogate.simulate(pop, P, lk, hr, train, args.c4_seeds, batch_size=64)
    t_sim = time.perf_counter() - t0
    # targets: log1p of each scenario's mean over its seeds (the quantity the
    # simulator's ensemble mean estimates; a mean of logs would sit below it)
    ym = np.stack([np.log1p(np.expm1(ys[idx == k]).mean(axis=0)) for k in range(len(train))]).astype(np.float32)
    xs = surrogate.to_unit(train).astype(np.float32)
    ys = ym
    # 2. training: an ensemble of networks, minibatches of 64, 10 % held out per member
    net = surrogate.Ensemble(args.c4_ensemble, max_batch=256, seed=5)
    t0 = time.perf_counter()
    hists = net.fit(xs, ys, epochs=args.c4_epochs, lr=1e-3, batch=64, holdout=0.1, weight_decay=1e-4)
    t_train = time.perf_counter() - t0
    # 3. screening
    sweep = surrogate.sample_scenarios(args.c4_sweep, seed=202)
    t0 = time.perf_counter()
    pred = net.predict(surrogate.to_unit(sweep).astype(np.float32))
    t_screen = time.perf_counter() - t0
    top = np.argsort(np.expm1(pred[:, :, 2]).max(axis=1))[:args.c4_rerun]
    # 4. the simulator judges the top scenarios: 8 seeds each
    t0 = time.perf_counter()
    ridx, rys = surrogate.simulate(pop, P, lk, hr, sweep[top], 8, batch_size=64, seed0=777)
    t_rerun = time.perf_counter() - t0
    t_pipeline = time.perf_counter() - t_all

    def icu_errors(sel, idx_r, ys_r):
        ens = np.stack([np.expm1(ys_r[idx_r == k]).mean(axis=0) for k in range(len(sel))])   # per million
        pr = np.expm1(pred[sel])
        num = np.linalg.norm(pr[:, :, 2] - ens[:, :, 2], axis=1)
        den = np.linalg.norm(ens[:, :, 2], axis=1)
        rel = num / np.maximum(den, 1e-12)
        return {"median": round(float(np.median(rel)), 4), "mean": round(float(rel.mean()), 4),
                "p90": round(float(np.quantile(rel, 0.9)), 4),
                "ensemble_icu_peak_per_million_median": round(float(np.median(ens[:, :, 2].max(axis=1))), 2)}
    err_top = icu_errors(top, ridx, rys)
    # accuracy on scenarios drawn at random from the sweep (not part of the timed pipeline)
    rnd = np.random.default_rng(303).choice(len(sweep), args.c4_check, replace=False)
    qidx, qys = surrogate.simulate(pop, P, lk, hr, sweep[rnd], 8, batch_size=64, seed0=888)
    err_rnd = icu_errors(rnd, qidx, qys)
    # the simulator against itself: a second, independent 8-seed ensemble of the same
    # random scenarios (the error floor any surrogate of the ensemble mean meets)
    q2idx, q2ys = surrogate.simulate(pop, P, lk, hr, sweep[rnd], 8, batch_size=64, seed0=999)
    e1 = np.stack([np.expm1(qys[qidx == k]).mean(axis=0) for k in range(len(rnd))])
    e2 = np.stack([np.expm1(q2ys[q2idx == k]).mean(axis=0) for k in range(len(rnd))])
    floor = np.linalg.norm(e1[:, :, 2] - e2[:, :, 2], axis=1) / np.maximum(np.linalg.norm(e2[:, :, 2], axis=1), 1e-12)
    err_rnd["simulator_vs_itself_median"] = round(float(np.median(floor)), 4)
    err_rnd["simulator_vs_itself_mean"] = round(float(floor.mean()), 4)
    if args.c4_save:
        def ens(sel, i_r, y_r):   # per-scenario ensemble means, log1p
            return np.stack([np.log1p(np.expm1(y_r[i_r == k]).mean(axis=0)) for k in range(len(sel))]).astype(np.float32)
        np.savez_compressed(args.c4_save, train=train, train_targets=ym, sweep_top=sweep[top],
                            top_mean=ens(top, ridx, rys), sweep_rnd=sweep[rnd], rnd_mean=ens(rnd, qidx, qys),
                            rnd_mean2=ens(rnd, q2idx, q2ys))
    # 5. the plain method: one realisation at a time, timed on a sample
    s1 = sim.Simulation(pop, P, lk, hr)
    beta24, _ = sim.calibrate_local_beta(pop, P, 2.4)
    n_plain = 8
    t0 = time.perf_counter()
    for k in range(n_plain):
        q, pol = surrogate.scenario_params(P, beta24, sweep[k])
        s1.backend.set_params(q)
        s1.params = q
        s1.run(9000 + k, surrogate.DAYS, policy=pol)
    s1.backend.sync()
    t_one = (time.perf_counter() - t0) / n_plain
    s1.close()
    t_plain = t_one * args.c4_sweep * 8
    heldout = [round(float(min(v for _, v in m.val_history)), 5) for m in net.nets if m.val_history]
    net.close()
    return {
        "metric": "scenario-sweep speed-up over one-at-a-time simulation", "value": round(t_plain / t_pipeline, 1),
        "unit": "x", "n_gpus": 1, "higher_is_better": True, "dtype": "bf16 network (fp32 accumulate), f64/f32 simulator",
        "data": "synthetic (seeded generator, reference parameter set)",
        "config": {"workload": "surrogate sweep: %d people, %d training scenarios x %d seeds, %d screened, top %d "
                               "re-run x 8 seeds" % (args.c4_people, args.c4_train, args.c4_seeds, args.c4_sweep,
                                                     args.c4_rerun)},
        "seconds": {"simulate_training": round(t_sim, 2), "train": round(t_train, 2), "screen": round(t_screen, 3),
                    "rerun_top": round(t_rerun, 2), "pipeline": round(t_pipeline, 2),
                    "one_realisation_plain": round(t_one, 4), "plain_sweep_estimate": round(t_plain, 1)},
        "train_loss": [round(float(np.mean([h[0] for h in hists])), 5), round(float(np.mean([h[-1] for h in hists])), 5)],
        "heldout_loss_best": heldout,
        "ensemble": args.c4_ensemble,
        "icu_rel_l2_vs_ensemble_mean": {"top_ranked": err_top, "random_sweep_sample": err_rnd},
    }


def main():
    args = parse()
    if args.impl == "ours" and args.workload == "c2":
        out = run_c2(args)
        if out is not None:
            print(json.dumps(out))
        return
    if args.impl == "ours" and args.workload == "c4":
        print(json.dumps(run_c4(args)))
        return
    out = run_reference(args) if args.impl == "reference" else run_ours(args)
    if out is not None:
        print(json.dumps(out))


if __name__ == "__main__":
    main()
