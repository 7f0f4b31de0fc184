"""Offline tuner of the GEMM-pass kernels: times the library's pass-kernel
variants (tile shapes: 32 or 16 complex lines per CTA, the register-operand
and persistent forms, the flip-symmetric half-block passes) and the library's
default for a small and a large batch of fields at each grid size and writes
a JSON table keyed by (ny, nz): the default, unless another form is faster at
both.  `Context.apply_tuning()` reads the table back and sets the pass kernel of
the context's size class (ductgpu_set_pass_kernel) and, for rectangular grids,
the form of ductgpu_set_rect_fold.

    python -m duct_b200.tune --square 33,65,129,193 --rect 65x129,49x145,33x129 \\
        --out duct_b200/tuning.json

Square grids: a substep's u, v, w (Dirichlet, lambda = kx^2 + 2/(nu dt))
and p (Neumann, lambda = kx^2) with `--modes` and a sixteenth of `--modes`
Fourier modes, every variant timed over CUDA-graph replays.  Rectangular grids
(my x mz, aspect mz/my): the same four fields through
ductgpu_solve_rect_fields_dev: the default, folded, one launch per pass and
size, folded in one launch, and full operators.
Needs a GPU.
"""
import argparse
import json
import os

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
TABLE = os.path.join(HERE, "tuning.json")

VARIANTS = {"staged-32": 0, "register": 1, "staged-16": 2, "persist": 3, "parity": 4, "parity-queue": 5}
FORMS = {"default": -1, **VARIANTS}
RECT = {"default": -1, "full": 0, "fold": 1, "fold-one-launch": 2}


def _time_graph(ctx, gid, reps):
    for _ in range(3):
        ctx.graph_launch(gid)
    ctx.synchronize()
    best = float("inf")
    for _ in range(3):
        ctx.event_record(0)
        for _ in range(reps):
            ctx.graph_launch(gid)
        ctx.event_record(1)
        best = min(best, ctx.event_elapsed(0, 1) / reps)
    return best


def choose(ms):
    """The form to set for a grid from ms[batch][form], every batch with a
    "default": a table holds for any batch of its grid, so the default stays
    unless another form is faster (by more than 2 %) at every batch timed."""
    forms = [f for f in next(iter(ms.values())) if f != "default"
             and all(f in t and t[f] < 0.98 * t["default"] for t in ms.values())]
    return min(forms, key=lambda f: sum(t[f] / t["default"] for t in ms.values()), default="default")


def _batches(nmodes):
    return sorted({max(1, nmodes // 16), nmodes})


def _time_forms(ctx, forms, select, fields, reps, **graph):
    """ms[form] of one batch; a form that refuses the batch is left out."""
    import duct_b200 as D
    ms = {}
    for name, v in forms.items():
        select(v)
        try:
            gid = ctx.graph_create(fields, **graph)
        except D.DuctGPUError:
            continue
        ms[name] = _time_graph(ctx, gid, reps)
        ctx.graph_destroy(gid)
    select(-1)
    return ms


def _fields(ctx, my, mz, nmodes, xalp, specs):
    from duct_b200 import synth
    fields = []
    for k, spec in enumerate(specs):
        f = synth.chebyshev_rhs(my, mz, nmodes, seed=1 + k, ib=0)
        r, s = ctx.device_array(f.shape), ctx.device_array(f.shape)
        r.upload(f)
        fields.append(dict(rhs=r, sol=s, xalp=xalp, ib=0, **spec))
    return fields


def _free(fields):
    for f in fields:
        f["rhs"].free()
        f["sol"].free()


def tune_square(ctx, m, nmodes, reps=20):
    ctx.pseudomat(m)
    lam = 2.0 / ((1.0 / 2000.0) * 1.0e-3)
    ms = {}
    for nm in _batches(nmodes):
        fields = _fields(ctx, m, m, nm, 0.5 * np.arange(nm),
                         [dict(bound="d", alambda=lam)] * 3 + [dict(bound="n", alambda=0.0)])
        ms[str(nm)] = _time_forms(ctx, FORMS, ctx.set_pass_kernel, fields, reps)
        _free(fields)
    return {"ny": m, "nz": m, "fields": 4, "pass_kernel": choose(ms), "ms_per_batch": ms}


def tune_rect(ctx, my, mz, nmodes, reps=20):
    aspect = (mz - 1) / (my - 1)
    ctx.pseudomat_temp(0, my, mz, 1.0, aspect)
    ctx.pseudomat_temp(1, my, mz, 1.0, aspect, ("n", "n"), ("n", "n"))
    lam = 2.0 / ((1.0 / 4400.0) * 5.0e-4)
    ms = {}
    for nm in _batches(nmodes):
        fields = _fields(ctx, my, mz, nm, 1.0 * np.arange(nm),
                         [dict(slot=0, alambda=lam)] * 3 + [dict(slot=1, alambda=0.0)])
        ms[str(nm)] = _time_forms(ctx, RECT, ctx.set_rect_fold, fields, reps, rect=True)
        _free(fields)
    return {"ny": my, "nz": mz, "fields": 4, "rect_fold": choose(ms), "ms_per_batch": ms}


def apply(ctx, my, mz, path=TABLE):
    """Settings of the table entry for (my, mz) onto ctx; returns the entry
    (None if the table or the entry is missing: the library defaults stay)."""
    if not os.path.exists(path):
        return None
    with open(path) as f:
        table = json.load(f)
    for e in table.get("entries", []):
        if e["ny"] == my and e["nz"] == mz:
            if "pass_kernel" in e:
                n = my - 2
                size_class = 0 if n <= 64 else (1 if n <= 128 else 2)
                ctx.set_pass_kernel(FORMS[e["pass_kernel"]], size_class)
            if "rect_fold" in e:       # a form's name, or its number in older tables
                form = e["rect_fold"]
                ctx.set_rect_fold(form if isinstance(form, int) else RECT[form])
            return e
    return None


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--square", default="33,65,129,193")
    ap.add_argument("--rect", default="65x129,49x145,33x129")
    ap.add_argument("--modes", type=int, default=64)
    ap.add_argument("--out", default=TABLE)
    a = ap.parse_args()
    import duct_b200 as D
    entries = []
    with D.Context(0) as ctx:
        for s in filter(None, a.square.split(",")):
            entries.append(tune_square(ctx, int(s), a.modes))
            print(json.dumps(entries[-1]), flush=True)
        for s in filter(None, a.rect.split(",")):
            my, mz = (int(x) for x in s.split("x"))
            entries.append(tune_rect(ctx, my, mz, a.modes))
            print(json.dumps(entries[-1]), flush=True)
    import subprocess
    dev = subprocess.run(["nvidia-smi", "--query-gpu=name", "--format=csv,noheader"], capture_output=True,
                         text=True).stdout.strip().splitlines()
    with open(a.out, "w") as f:
        json.dump({"device": dev[0] if dev else None, "tuned_with": "python -m duct_b200.tune", "entries": entries},
                  f, indent=1)


if __name__ == "__main__":
    main()
