"""Autotuner for the radix plans of the transform passes.

For one workload (dimension, N, padded M, precision, batch) it runs SSP-RK3
steps of a Simulation with every kernel variant, times each pass with the
library's per-pass CUDA events (az_profile_*), and keeps, for each pass kind
that has variants there (pass_kinds), the fastest.
Results go into a JSON tuning table that ``azeban_b200`` loads at import
(``tuning.json`` beside this file) and applies with az_tune_set.

The reference's closest counterpart picks the padded FFT size from a
benchmark file (src/azeban/operations/fft.cpp:63-108).

Usage on a GPU: ``python -m azeban_b200.tune --out azeban_b200/tuning.json``.
"""

from __future__ import annotations

import argparse
import ctypes as ct
import json
import os

import torch

from . import _lib
from .core import SSP_RK3, Grid, IncompressibleEuler, Simulation, make_viscosity, precision_code

TABLE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "tuning.json")
VISC = {"type": "Smooth Cutoff", "eps": 0.05}


# Kernel variants: the radix plan (0 std, 1 wide).
RUNS = (0, 1)
# Padded lengths whose 3-D column passes have the two plans (kRegisterColumns).
REGISTER_COLUMNS = (384,)


def pass_kinds(dim: int, L: int) -> dict:
    """Tuned kinds that the passes of a solve read, with the passes that each one times: the last pass of
    3-D solves (kind 2) and, at some lengths, their column passes (kind 0).  The other passes have one
    form per length.  Kinds 0 and 1 are also the plans of FFT<Dim>'s strided axes and r2c lines, which no
    solve times."""
    if dim != 3:
        return {}
    return {2: (4,), **({0: (0, 1, 3)} if L in REGISTER_COLUMNS else {})}


def _time_passes(eq, u, reps):
    """Per-pass times averaged over SSP-RK3 steps of a Simulation: the first
    pass of stage 1 reads the caller-layout state and those of stages 2 and 3
    the stepper's component-innermost buffers, as in every run (a plain dudt
    times the first layout only)."""
    sim = Simulation(eq.grid, 0.2, SSP_RK3(eq), u)
    sim.steps(2)
    torch.cuda.synchronize()
    _lib.check(_lib.lib.az_profile_enable(1))
    sim.steps(reps)
    torch.cuda.synchronize()
    _lib.check(_lib.lib.az_profile_enable(0))
    ms = (ct.c_double * 5)()
    by = (ct.c_double * 5)()
    nl = (ct.c_longlong * 5)()
    _lib.check(_lib.lib.az_profile_read(ms, by, nl, 5))
    return [ms[i] / nl[i] if nl[i] else 0.0 for i in range(5)]


def autotune(dim: int, N: int, precision="f32", batch: int = 1, M: int | None = None, reps: int = 5):
    """Measures both plan variants of one workload and applies the winners;
    returns the table entries (none where no pass has variants)."""
    prec = precision_code(precision)
    g = Grid(dim, N, M)
    L = g.N_phys_pad
    kinds = pass_kinds(dim, L)
    if not kinds:
        return []
    visc = make_viscosity(VISC, g)
    shape = ((batch,) if batch > 1 else ()) + g.shape_fourier(dim)
    cdt = torch.complex128 if prec == 0 else torch.complex64
    gen = torch.Generator(device="cuda").manual_seed(1234)
    u = (torch.randn(shape, dtype=cdt, device="cuda", generator=gen) * (N ** dim) * 1e-3).contiguous()
    per_run = {}
    for run in RUNS:
        for kind in kinds:
            _lib.check(_lib.lib.az_tune_set(prec, L, kind, run))
        eq = IncompressibleEuler(g, visc, precision, batch)
        per_run[run] = _time_passes(eq, u, reps)
        del eq
    entries = []
    for kind, passes in kinds.items():
        t = {run: sum(times[p] for p in passes) for run, times in per_run.items()}
        best = min(t, key=t.get)
        _lib.check(_lib.lib.az_tune_set(prec, L, kind, best))
        entries.append({"precision": prec, "L": L, "kind": kind, "variant": best,
                        "workload": f"{dim}-D N={N} M={L} batch={batch}",
                        "ms_per_rhs": {str(v): t[v] for v in sorted(t)}})
    return entries


def load_table(path: str = TABLE) -> int:
    """Applies a saved tuning table; returns the number of entries."""
    if not os.path.exists(path):
        return 0
    with open(path) as f:
        entries = json.load(f)
    n = 0
    for e in entries:
        if _lib.lib.az_tune_set(int(e["precision"]), int(e["L"]), int(e["kind"]), int(e["variant"])) == 0:
            n += 1
    return n


WORKLOADS = [
    # (dim, N, precision, batch): the configs' 3-D sizes
    (3, 256, "f32", 4), (3, 256, "f64", 1), (3, 128, "f32", 1), (3, 128, "f64", 1),
    (3, 64, "f32", 4), (3, 64, "f64", 4), (3, 512, "f32", 1),
]


def main(argv=None):
    ap = argparse.ArgumentParser()
    ap.add_argument("--out", default=TABLE)
    ap.add_argument("--reps", type=int, default=5)
    args = ap.parse_args(argv)
    table = {}
    if os.path.exists(args.out):  # keeps the plans that no workload times
        with open(args.out) as f:
            table = {(e["precision"], e["L"], e["kind"]): e for e in json.load(f)}
    for dim, N, prec, batch in WORKLOADS:
        for e in autotune(dim, N, prec, batch, reps=args.reps):
            table[(e["precision"], e["L"], e["kind"])] = e
            print(json.dumps(e), flush=True)
    with open(args.out, "w") as f:
        json.dump(list(table.values()), f, indent=1)


if __name__ == "__main__":
    main()
