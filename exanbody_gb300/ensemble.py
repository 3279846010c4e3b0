"""Batched ensemble of independent LJ systems in one batch, and its autotuner.

All systems of a batch advance together: every kernel of a step covers the
packed particle and cell tables of every system (uneven sizes, empty cells
included), and the step sequence is captured as a CUDA graph
(xnb_step_graph_create) so a chunk of steps costs one launch on the host.

The autotuner times short trials of the batch over the tunables the library
exposes -- the neighbour-build kernel (lane per candidate or lane per particle
with bulk-copied rows), its staging capacity, force-traversal threads per
block and threads per particle, the force traversal itself (full lists or
Newton half lists) and the Verlet skin -- and keeps the fastest.

  python -m exanbody_gb300.ensemble [--count 1024] [--steps 500] [--autotune] [--no-tune-skin]
"""
import argparse
import ctypes
import itertools
import json
import time

import numpy as np

from . import replicas, workloads, xnb

DEFAULTS = dict(build_form="warp", stage_cap=640, force_block=128, force_lanes=1, skin=0.3, newton=False)
FORMS = {"warp": xnb.BUILD_WARP, "rows": xnb.BUILD_ROWS, "half": xnb.BUILD_HALF}


def make_systems(specs, rcut=2.5, skin=0.3):
    return [workloads.lj_fcc_system(sp["n"], sp["rho"], sp["T"], sp["seed"], rcut, skin) for sp in specs]


def geometry_for(w, rcut, skin):
    """The system's periodic box with the cell grid of neighbour distance rcut + skin
    (the same box and positions; the cell size follows the skin)."""
    g = w["geom"]
    return workloads.geometry(tuple(e - o for e, o in zip(g["extent"], g["origin"])), rcut, skin)


def build_batch(systems, stage_cap=640, force_block=128, skin=0.3, rcut=2.5, dt=0.005, stream=None,
                precision=xnb.PREC_MIXED, list_per_atom=None, build_form="warp", force_lanes=1):
    n_atoms = sum(w["n_atoms"] for w in systems)
    n_cells = sum(int(np.prod(w["geom"]["dims"])) for w in systems)
    if list_per_atom is None:
        # neighbours within rc + skin at the densest state point of the batch, with margin
        rho = max(w["rho"] for w in systems)
        list_per_atom = 1.6 * (4.0 / 3.0) * np.pi * (rcut + skin) ** 3 * rho + 24
    b = xnb.Batch(n_atoms + 64 * len(systems), n_cells + 64, int(list_per_atom * n_atoms) + 4096,
                  max_systems=len(systems), stage_cap=stage_cap, force_block=force_block)
    if stream is not None:
        b.stream = ctypes.c_void_p(stream)
    b.set_build_form(FORMS[build_form])
    b.set_force_lanes(force_lanes)
    ids = [b.add_system(xnb.lj_params(geometry_for(w, rcut, skin), rcut=rcut, rcut_inc=skin, dt=dt), w["r"], w["v"],
                        w["id"], list_factor=1.25) for w in systems]
    b.init_particles(-1, precision)
    return b, ids, n_atoms


def timed_steps(batch, stream, steps, precision, chunk=10):
    """Run `steps` MD steps as replays of a captured `chunk`-step graph; seconds."""
    import torch

    g = batch.graph(chunk, precision, 0)
    g.launch()  # warm
    stream.synchronize()
    reps = max(1, steps // chunk)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(reps):
        g.launch()
    e1.record(stream)
    e1.synchronize()
    batch.check_errors()
    g.close()
    return e0.elapsed_time(e1) * 1e-3, reps * chunk


def trial(systems, cfg, steps, precision, stream):
    prec = precision | (xnb.PREC_NEWTON if cfg["newton"] else 0)
    b, ids, n = build_batch(systems, cfg["stage_cap"], cfg["force_block"], cfg["skin"], stream=stream.cuda_stream,
                            precision=prec, build_form=cfg["build_form"], force_lanes=cfg["force_lanes"])
    try:
        secs, done = timed_steps(b, stream, steps, prec)
    finally:
        b.close()
    return n * done / secs


def autotune(systems, precision=xnb.PREC_MIXED, steps=40, tune_skin=False, stream=None):
    """Coordinate search over the tunables on the given systems (a sample of the batch). The force settings that
    their forces do not read (FP64, and mixed up to MIXED_SPLIT_MAX particles) keep their defaults."""
    import torch

    stream = stream or torch.cuda.Stream()
    space = {
        "build_form": ["warp", "rows"],
        "stage_cap": [384, 640, 1024],
        "force_block": [64, 128, 256],
        "force_lanes": [1, 2, 4],
        "newton": [False, True],
        "skin": [0.3, 0.4, 0.5] if tune_skin else [0.3],
    }
    if systems and (precision != xnb.PREC_MIXED or sum(w["n_atoms"] for w in systems) <= xnb.MIXED_SPLIT_MAX):
        space["force_block"], space["force_lanes"] = [DEFAULTS["force_block"]], [DEFAULTS["force_lanes"]]
    best = dict(DEFAULTS)
    best_rate = trial(systems, best, steps, precision, stream)
    log = [dict(best, rate=best_rate)]
    for key in ("build_form", "stage_cap", "force_block", "force_lanes", "newton", "skin"):
        measured = best[key]  # this knob's value in the configuration already timed
        for v in space[key]:
            if v == measured:
                continue
            cand = dict(best, **{key: v})
            rate = trial(systems, cand, steps, precision, stream)
            log.append(dict(cand, rate=rate))
            if rate > best_rate:
                best, best_rate = cand, rate
    return best, best_rate, log


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--count", type=int, default=1024)
    ap.add_argument("--steps", type=int, default=500)
    ap.add_argument("--seed", type=int, default=2024)
    ap.add_argument("--autotune", action="store_true")
    ap.add_argument("--no-tune-skin", action="store_true", help="keep the Verlet skin at 0.3")
    ap.add_argument("--tune-sample", type=int, default=128, help="systems used for the autotuner trials")
    args = ap.parse_args()
    import torch

    rank, world, local = replicas.dist_env()
    dev = None
    if world > 1:
        # replicas: each GPU advances every world-th system of the ensemble
        import torch.distributed as dist

        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
        torch.cuda.set_device(local)
        dev = torch.device("cuda", local)
    specs = replicas.shard(workloads.ensemble_specs(args.count, seed=args.seed), rank, world)
    systems = make_systems(specs)
    stream = torch.cuda.Stream()
    cfg = dict(DEFAULTS)
    tune_log = None
    t0 = time.perf_counter()
    if args.autotune:
        sample = systems[: args.tune_sample]
        cfg, _, tune_log = autotune(sample, xnb.PREC_MIXED, tune_skin=not args.no_tune_skin, stream=stream)
    tune_s = time.perf_counter() - t0
    out = {"workload": "ensemble_%d_fcc_n4-25_rho0.70-1.00_T0.7-1.5" % args.count, "gpus": world,
           "atoms": int(replicas.gather_values([sum(w["n_atoms"] for w in systems)], device=dev).sum()),
           "systems": args.count, "steps": args.steps,
           "config": cfg, "autotune_seconds": tune_s}
    # the mixed path runs the tuned configuration; the FP64 path is timed with both
    # traversals (full lists, Newton half lists) at the tuned skin and at the
    # default one (the skin was tuned on the mixed path), and reported at its
    # fastest: the speedup is against FP64 at its own best
    runs = [("mixed", xnb.PREC_MIXED | (xnb.PREC_NEWTON if cfg["newton"] else 0), cfg["skin"]),
            ("fp64_full", xnb.PREC_FP64, cfg["skin"]), ("fp64_newton", xnb.PREC_FP64 | xnb.PREC_NEWTON, cfg["skin"])]
    if cfg["skin"] != DEFAULTS["skin"]:
        runs += [("fp64_full_skin%.1f" % DEFAULTS["skin"], xnb.PREC_FP64, DEFAULTS["skin"]),
                 ("fp64_newton_skin%.1f" % DEFAULTS["skin"], xnb.PREC_FP64 | xnb.PREC_NEWTON, DEFAULTS["skin"])]
    for name, prec, skin in runs:
        b, ids, n = build_batch(systems, cfg["stage_cap"], cfg["force_block"], skin,
                                stream=stream.cuda_stream, precision=prec, build_form=cfg["build_form"],
                                force_lanes=cfg["force_lanes"])
        secs, done = timed_steps(b, stream, args.steps, prec)
        rebuilds = sum(b.info(s).rebuilds for s in ids)
        b.close()
        # whole job: all ranks' atoms over the slowest rank's time
        secs = replicas.max_over_ranks(secs, device=dev)
        n_all = replicas.gather_values([n], device=dev).sum()
        rebuilds = replicas.gather_values([rebuilds], device=dev).sum()
        out[name] = {"atom_steps_per_s": float(n_all) * done / secs, "seconds": secs, "steps": done,
                     "rebuilds_total": int(rebuilds), "skin": skin}
    best = max((r[0] for r in runs if r[0].startswith("fp64")), key=lambda k: out[k]["atom_steps_per_s"])
    out["fp64"] = dict(out[best], traversal=best)
    out["speedup_mixed_vs_fp64"] = out["mixed"]["atom_steps_per_s"] / out["fp64"]["atom_steps_per_s"]
    if tune_log is not None:
        out["autotune_trials"] = tune_log
    if rank == 0:
        print(json.dumps(out))


if __name__ == "__main__":
    main()
