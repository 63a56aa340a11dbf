"""What this framework is timed on: solves through its public entry points.

Each case is one pass of a program that keeps its handle (a solver context, a
batch, a server, or its own device buffers for the drop-in call):

  solve   a context takes `steps` time steps and its field is read back into
          pinned host memory; with `restart` a new initial field is set first
          (many short solves with one handle), without it the run continues
          where it stood (a long run that writes its field out now and then)
  whole   a context made from host arrays, stepped, read back and closed
  dropin  heat_update_async on the caller's device buffers, swapped by the
          caller each step, as the reference's own time loop calls it
  batch   a batch of uneven grids, half FP64 and half FP32C, advanced together
  serve   a request stream through the continuous-batching server

Fields are seeded versions of the three problems that the tests and the
benchmark use: "bump" (smooth conductivity, Gaussian bump), "random"
(log-normal conductivity, uniform noise) and "source" (the reference's own
problem, with its source term).
"""
from __future__ import annotations

import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "openmp-offloading-intranode-artifact_gb300"))
import heat_ctypes as H  # noqa: E402

FORMS = {"fp64": (H.HEAT_FP64, 0), "fp32c": (H.HEAT_FP32C, 0), "bitexact": (H.HEAT_FP64, H.HEAT_BITEXACT)}


def solve(name, form, problem, nx, ny, nz, steps, restart, kind="solve"):
    return {"name": name, "kind": kind, "form": form, "problem": problem, "nx": nx, "ny": ny, "nz": nz,
            "steps": steps, "restart": restart}


def listed():
    return [
        # the benchmark's headline problem: a long run on 512^3
        solve("fp64_512", "fp64", "bump", 512, 512, 512, 200, False),
        # the reference's own problem at its verify size (256, 100 steps), source term included
        solve("fp64_source_256", "fp64", "source", 256, 256, 256, 100, False),
        # the reference-CPU-sized problem, restarted with new initial fields
        solve("fp64_128", "fp64", "random", 128, 128, 128, 100, True),
        # the smallest calls: launches and latency count
        solve("fp64_small", "fp64", "random", 40, 33, 28, 50, True),
        # ragged axes, none a multiple of a tile or of the row padding
        solve("fp64_ragged", "fp64", "bump", 259, 131, 97, 100, True),
        # the fast reduced-storage form, large
        solve("fp32c_512", "fp32c", "bump", 512, 512, 512, 200, False),
        # the same form on an uneven grid with an odd number of steps
        solve("fp32c_ragged", "fp32c", "random", 150, 101, 83, 51, True),
        # results bit for bit as the reference's serial solver, source term included
        solve("bitexact_source_160", "bitexact", "source", 160, 160, 160, 50, True),
        # a whole call from host arrays to host array: set-up, solve, read-back
        solve("whole_fp64_192", "fp64", "bump", 192, 192, 192, 200, False, kind="whole"),
        # the reference's per-step device call on the caller's buffers
        {"name": "dropin_256", "kind": "dropin", "problem": "source", "nx": 256, "ny": 256, "nz": 256, "steps": 20},
        # many uneven grids at once
        {"name": "batch_12", "kind": "batch", "grids": 12, "min_axis": 48, "max_axis": 192, "steps": 96, "shapes": 7},
        # a burst of requests through the server
        {"name": "serve_16", "kind": "serve", "requests": 16, "min_axis": 32, "max_axis": 160, "steps": 200, "shapes": 5},
    ]


def log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve"] * 7 + ["whole", "dropin", "dropin", "batch", "serve"])
    if kind in ("batch", "serve"):
        c = {"kind": kind, "min_axis": rng.randint(24, 64), "max_axis": rng.randint(96, 192),
             "steps": rng.randint(40, 200), "shapes": rng.randint(0, 999)}
        return {**c, ("grids" if kind == "batch" else "requests"): rng.randint(4, 16)}
    while True:
        nx, ny, nz = (log_uniform(rng, 16, 512) for _ in range(3))
        if nx * ny * nz <= 100_000_000:
            break
    points = nx * ny * nz
    form = rng.choice(["fp64", "fp64", "fp64", "fp32c", "fp32c", "bitexact"])
    problem = rng.choice(["bump", "random", "source"])
    most = max(4, min(200, int(4e9 / points / (1 if form != "bitexact" else 4))))
    steps = log_uniform(rng, 4, most) if most > 4 else 4
    if kind == "dropin":
        return {"kind": kind, "problem": problem, "nx": nx, "ny": ny, "nz": nz, "steps": max(4, steps // 4)}
    c = solve("", form, problem, nx, ny, nz, steps, points < 8_000_000, kind=kind)
    c.pop("name")
    return c


# ---- inputs ---------------------------------------------------------------

def fields(problem, nx, ny, nz, seed):
    """(kappa, u0, rhs or None, h, dt), FP64 on the GPU, shape (nz, ny, nx)."""
    rnd = random.Random(seed)
    h = 1.0 / (max(nx, ny, nz) - 1)
    z, y, x = (torch.arange(n, dtype=torch.float64, device="cuda") * h for n in (nz, ny, nx))
    z, y, x = z[:, None, None], y[None, :, None], x[None, None, :]
    rhs = None
    if problem == "random":
        g = torch.Generator(device="cuda").manual_seed(seed)
        kappa = torch.exp(0.5 * torch.randn((nz, ny, nx), generator=g, device="cuda", dtype=torch.float64))
        u0 = torch.rand((nz, ny, nx), generator=g, device="cuda", dtype=torch.float64)
        dt = 0.9 * h * h / (6.0 * float(kappa.max()))
    elif problem == "bump":
        kappa = 1.0 + 0.9 * torch.sin(2 * math.pi * x) * torch.sin(4 * math.pi * y) * torch.cos(2 * math.pi * z)
        u0 = 1.0
        for a, n in ((x, nx), (y, ny), (z, nz)):
            centre = rnd.uniform(0.3, 0.7) * (n - 1) * h
            u0 = u0 * torch.exp(-((a - centre) ** 2) / (2 * 0.05 ** 2))
        dt = 0.9 * h * h / (6.0 * 1.9)
    else:
        a = rnd.uniform(0.8, 1.2)
        px, py, pz = (math.pi / ((n - 1) * h) for n in (nx, ny, nz))
        kappa = 0.5 + 0.45 * torch.sin(a * px * x) * torch.sin(py * y) * torch.sin(pz * z)
        u0 = a * torch.sin(px * x) * torch.sin(py * y) * torch.sin(pz * z)
        dt = h * h / (12.0 * 0.95)
        rhs = dt * (a + torch.cos(px * x) * torch.cos(py * y) * torch.cos(pz * z))
    u0 = u0.expand(nz, ny, nx).clone()
    u0[0], u0[-1], u0[:, 0], u0[:, -1], u0[:, :, 0], u0[:, :, -1] = 0, 0, 0, 0, 0, 0
    return kappa.expand(nz, ny, nx).contiguous(), u0, rhs, h, dt


def pinned(t):
    """A pinned host copy of t, as numpy."""
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    p.copy_(t)
    return p.numpy()


def context(form, problem, nx, ny, nz, seed):
    precision, flags = FORMS[form]
    kappa, u0, rhs, h, dt = fields(problem, nx, ny, nz, seed)
    args = [pinned(kappa), pinned(u0), h, dt]
    return args, {"rhs": None if rhs is None else pinned(rhs), "precision": precision, "flags": flags}


def grids_of(case, seed):
    """Shapes, problem, form and seed of each grid of a batch."""
    rnd = random.Random(case["shapes"])
    return [(("random", "bump")[k % 3 == 2], "fp64" if k % 2 == 0 else "fp32c",
             [rnd.randint(case["min_axis"], case["max_axis"]) for _ in range(3)], 1000 * seed + k)
            for k in range(case["grids"])]


def requests_of(case, seed):
    rnd = random.Random(case["shapes"])
    return [{"nx": rnd.randint(case["min_axis"], case["max_axis"]), "ny": rnd.randint(case["min_axis"], case["max_axis"]),
             "nz": rnd.randint(case["min_axis"], case["max_axis"]), "steps": rnd.randint(case["steps"] // 4, case["steps"]),
             "precision": H.HEAT_FP64 if k % 2 == 0 else H.HEAT_FP32C, "cfg": 0, "seed": 1000 * seed + k}
            for k in range(case["requests"])]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solve", "whole"):
        args, more = context(case["form"], case["problem"], case["nx"], case["ny"], case["nz"], seed)
        state = {"kind": kind, "steps": case["steps"], "restart": case["restart"], "u0": args[1],
                 "out": pinned(torch.empty(args[1].shape, dtype=torch.float64))}
        if kind == "whole":
            return {**state, "args": args, "more": more}
        return {**state, "solver": H.Solver(*args, **more)}
    if kind == "dropin":
        kappa, u0, rhs, h, dt = fields(case["problem"], case["nx"], case["ny"], case["nz"], seed)
        return {"kind": kind, "steps": case["steps"], "factor": dt / h / h / 2.0, "kappa": kappa, "rhs": rhs,
                "u": [u0, u0.clone()]}
    if kind == "batch":
        solvers, outs = [], []
        for problem, form, shape, s in grids_of(case, seed):
            args, more = context(form, problem, *shape, s)
            solvers.append(H.Solver(*args, **more))
            outs.append(pinned(torch.empty(args[1].shape, dtype=torch.float64)))
        return {"kind": kind, "batch": H.Batch(), "solvers": solvers, "steps": case["steps"], "outs": outs}
    reqs = requests_of(case, seed)
    return {"kind": kind, "server": H.Server(8 << 30, tick_steps=32, prep_threads=4), "requests": reqs,
            "outs": [pinned(torch.empty((r["nz"], r["ny"], r["nx"]), dtype=torch.float64)) for r in reqs]}


def run(state):
    kind = state["kind"]
    if kind == "solve":
        s = state["solver"]
        if state["restart"]:
            s.set_field(state["u0"])
        s.step(state["steps"])
        return s.field(state["out"])
    if kind == "whole":
        with H.Solver(*state["args"], **state["more"]) as s:
            s.step(state["steps"])
            return {"u": s.field(state["out"]), "norm": list(s.norm())}
    if kind == "dropin":
        old, new = state["u"]
        nz, ny, nx = old.shape
        rhs = None if state["rhs"] is None else state["rhs"].data_ptr()
        stream = torch.cuda.current_stream().cuda_stream
        lib = H.lib()
        for _ in range(state["steps"]):
            H.check(lib.heat_update_async(new.data_ptr(), old.data_ptr(), rhs, state["kappa"].data_ptr(),
                                          nz, ny, nx, state["factor"], stream), "heat_update_async")
            old, new = new, old
        state["u"] = [old, new]
        return old
    if kind == "batch":
        b = state["batch"]
        for s in state["solvers"]:
            b.add(s, state["steps"])
        b.run()
        return [s.field(o) for s, o in zip(state["solvers"], state["outs"])]
    srv = state["server"]
    for r, o in zip(state["requests"], state["outs"]):
        srv.submit(**r, field_out=o)
    srv.wait_idle()
    for r in srv.poll():
        H.check(r["status"], "request")
    return state["outs"]


# ---- what a pass cannot do without, and its results in 64 bits --------------

def step_bytes(form, problem):
    """Per point and step: the field read and written and the conductivity read once, and the source term.
    fp64: 8 + 8 + 8 (+ 8); fp32c: value and carry 6 + 6, three face weights 12 (+ 4)."""
    return 24 + ((4 if form == "fp32c" else 8) if problem == "source" else 0)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        per = [(math.prod(s), case["steps"], f, p) for p, f, s, _ in grids_of(case, 0)]
    elif kind == "serve":
        per = [(r["nx"] * r["ny"] * r["nz"], r["steps"], "fp64", "random") for r in requests_of(case, 0)]
    else:
        per = [(case["nx"] * case["ny"] * case["nz"], case["steps"], case.get("form", "fp64"), case["problem"])]
    return {"bytes": sum(n * s * step_bytes(f, p) for n, s, f, p in per),
            "flops": sum(n * s * 14 for n, s, _, _ in per)}


def advance(kappa, u, rhs, factor, steps):
    """`steps` explicit steps in 64 bits, in the reference's expression."""
    c = (slice(1, -1),) * 3

    def at(dim, d):
        return tuple(slice(1 + d, (-1 + d) or None) if a == dim else slice(1, -1) for a in range(3))

    weights = [factor * (kappa[at(dim, d)] + kappa[c]) for dim in range(3) for d in (1, -1)]
    for _ in range(steps):
        uc = u[c]
        acc = torch.zeros_like(uc) if rhs is None else rhs[c].clone()
        for w, (dim, d) in zip(weights, ((a, b) for a in range(3) for b in (1, -1))):
            t = u[at(dim, d)] - uc
            acc.addcmul_(w, t)
        u[c] = uc + acc
    return u


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return None  # the server makes its own inputs
    if kind == "batch":
        out = []
        for problem, _, shape, s in grids_of(case, seed):
            kappa, u0, rhs, h, dt = fields(problem, *shape, s)
            out.append(advance(kappa, u0, rhs, dt / h / h / 2.0, case["steps"]).cpu().numpy())
        return out
    kappa, u, rhs, h, dt = fields(case["problem"], case["nx"], case["ny"], case["nz"], seed)
    u = advance(kappa, u, rhs, dt / h / h / 2.0, case["steps"])
    if kind == "whole":
        return {"u": u.cpu().numpy(), "norm": [float(u.square().sum().sqrt()), float(u.sum())]}
    return u if kind == "dropin" else u.cpu().numpy()
