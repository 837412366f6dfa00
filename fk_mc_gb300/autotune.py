"""Autotuner for the Householder reduction's variant and the mixed path's
back-transformation kernel.

For every matrix-size class of the uneven workloads (cubic2d L = 12..32,
triangular L = 12..24: n = 144, 256, 324, 400, 576, 1024) and both
precisions, times every compiled reduction variant (fkg_set_tuning: the
one-stage panel widths and, for the mixed path, the two-stage reduction) on a
batch of random configurations with CUDA events around the launches
(fkg_profile / fkg_stage_time), keeps the fastest and writes the table as
JSON. A variant's time is the sum of all stages of the solve (reduction,
tridiagonal eigenproblem, back-transformation, refinement): the two-stage
reduction moves work into the back-transformation (the band stage's
reflectors). On the mixed path it adds a values-only solve and one with
eigenvectors (the panel widths matter only for the latter; the values-only
one-stage reduction has one width). It then times the mixed path's two back-transformation
kernels (mma.sync with the block of Z in shared memory, tcgen05 with
tensor-memory accumulators; fkg_set_tuning_back) per size class under the
chosen reduction. Where that is the two-stage one, it times the proposal steps of
resident chains, which need eigenvalues only, under both reductions: with few
chains the one-stage kernel gives each several SMs (fkg_set_tuning_chains). `Solver(..., tuning=path)` (default: the table shipped
next to this file, when present) applies it with these setters.

Run on the GPU:  python -m fk_mc_gb300.autotune --out fk_mc_gb300/tuning_gb300.json
"""
import argparse
import json
import os

import numpy as np

DEFAULT_TABLE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "tuning_gb300.json")
CLASSES = [("cubic2d", 12), ("cubic2d", 16), ("triangular", 18), ("cubic2d", 20), ("cubic2d", 24), ("cubic2d", 32)]
VARIANTS = {"mixed": [4, 8, 16, "two-stage"], "f64": [2, 4]}  # panel widths (or two-stage), index = variant
STAGES = ("reduce", "trieig", "back", "refine")
BACK_VARIANTS = {0: "mma.sync", 1: "tcgen05"}       # back-transformation kernels of the mixed path


def _step_ms(s, n, f, most, reps, rng):
    """Stage times of a proposal step of resident chains reduced in one stage (most >= their number) or two."""
    B = len(f)
    s.set_tuning_chains(n, most)
    s.chains_init(np.zeros(B, np.int32), f.ravel(), 2.0, 1.0, 1.0, 4.0)
    step = lambda k: s.propose_accept(rng.integers(0, n, (k, B)), np.full((k, B), 0.5))
    step(1)  # warm
    s.profile(True)
    step(reps)
    ms = sum(s.stage_time(st)[0] for st in STAGES) / reps
    s.profile(False)
    return ms


def tune(batch=None, reps=3, seed=1):
    from .solver import Solver
    table = {"device": None, "entries": []}
    import torch
    table["device"] = torch.cuda.get_device_name(0)
    if batch is None:  # one chain per SM: between the few chains and the many that one choice has to serve
        batch = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(seed)
    for prec, widths in VARIANTS.items():
        s = Solver(max_n=1024, max_batch=batch, precision=prec, tuning=None)
        s.set_graphs(False)
        for kind, L in CLASSES:
            n = s.set_lattice(0, kind, L)
            f = rng.integers(0, 2, (batch, n))
            diag = (-1.0 + 2.0 * f).ravel()
            ids = np.zeros(batch, np.int32)
            def solve():  # values only, and (mixed: another one-stage kernel) with eigenvectors
                s.eigh_logz(ids, diag, 4.0)
                if prec == "mixed":
                    s.free_energy_grad(ids, f.ravel(), 2.0, 1.0, 1.0, 4.0)
            times = []
            for v in range(len(widths)):
                s.set_tuning(prec, n, v)
                solve()  # warm
                s.profile(True)
                for _ in range(reps):
                    solve()
                times.append(sum(s.stage_time(st)[0] for st in STAGES) / reps)
                s.profile(False)
            best = int(np.argmin(times))
            reduction = {"precision": prec, "n_max": n, "variant": best, "panel_width": widths[best],
                         "ms_per_solve": [round(t, 4) for t in times], "batch": batch}
            table["entries"].append(reduction)
            if prec == "mixed":
                s.set_tuning(prec, n, best)
                bt = []
                for v in sorted(BACK_VARIANTS):
                    s.set_tuning_back(n, v)
                    s.eigh_logz(ids, diag, 4.0)  # warm
                    s.profile(True)
                    for _ in range(reps):
                        s.eigh_logz(ids, diag, 4.0)
                    bt.append(s.stage_time("back")[0] / reps)
                    s.profile(False)
                best = int(np.argmin(bt))
                table["entries"].append({"stage": "back", "n_max": n, "variant": best,
                                         "kernel": BACK_VARIANTS[best], "ms_per_solve": [round(t, 4) for t in bt],
                                         "batch": batch})
                if widths[reduction["variant"]] == "two-stage":
                    s.set_tuning_back(n, best)
                    steps = [(b, [_step_ms(s, n, f[:b], most, reps, rng) for most in (b, 0)])
                             for b in (batch // 4, batch // 2, batch)]
                    reduction.update(chains=max([b for b, (one, two) in steps if one < two], default=0),
                                     ms_per_step=[[b, round(one, 4), round(two, 4)] for b, (one, two) in steps])
                s.set_tuning_back(n, -1)
            s.set_tuning(prec, n, -1)
        s.close()
    return table


def apply(solver, path=DEFAULT_TABLE):
    """Apply a tuning table to a Solver (entries for its own sizes; others keep the default)."""
    if not path or not os.path.exists(path):
        return False
    table = json.load(open(path))
    for e in table.get("entries", []):
        if e.get("stage") == "back":
            solver.set_tuning_back(e["n_max"], e["variant"])
        else:
            solver.set_tuning(e["precision"], e["n_max"], e["variant"])
            if "chains" in e:
                solver.set_tuning_chains(e["n_max"], e["chains"])
    return True


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--out", default=DEFAULT_TABLE)
    ap.add_argument("--batch", type=int, default=None)
    args = ap.parse_args()
    t = tune(batch=args.batch)
    with open(args.out, "w") as fh:
        json.dump(t, fh, indent=1)
    print(json.dumps(t))
