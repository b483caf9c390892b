"""Performance cases of the rh3t solver: the calls a program makes, over the
sizes, boundary kinds, physics options and arithmetic builds it makes them
with.

  listed()             the fixed cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  geometry, solver and host arrays a program holds before the call
  run(state)           one pass through the public entry points; returns its outputs
  work(case)           bytes and floating-point operations the pass cannot do without
  exact(case, seed)    outputs with a closed form (the CFL time steps), by numpy

The initial fields are developed-looking flows, not uniform ones: a smeared bow
shock (half-cylinder) or the case's own shock, with smooth seeded
perturbations of density, velocity and the three pressures, so that every
term of the operator works on values of the size it meets in a run. A pass of
many steps starts from the same initial field (a program that runs a parameter
study or an ensemble uploads a field, advances it and reads it back); a pass of
one step on host arrays goes on from where the one before it ended, in place, as
a host program's time loop does, and starts over after LOOP steps (the impulsive
flows of the coarsest meshes do not last for ever).

The geometry (Field and GhostGrid) depends on the mesh alone and is kept per
mesh, as a program that runs several flows on one mesh keeps it.
"""
import functools
import importlib
import math

import numpy as np
import torch

rh = importlib.import_module("3t_rh_b200")
flops = importlib.import_module("3t_rh_b200.flops")

CFL = 0.05  # the reference driver's factor on the CFL time step
LOOP = 500  # time steps of a host program's loop


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # One time-loop iteration of a host program on its own value array
        # (the drop-in call), on the coarsest half-cylinder: launch latency.
        {"name": "host step 31x121", "kind": "host_step", "nx": 31, "mach": 3.0, "source": False},
        # The semi-discrete operator alone, with the ghost values, as an
        # implicit or external time integrator calls it.
        {"name": "operator 121x481", "kind": "operator", "nx": 121, "mach": 3.0, "source": True},
        # Translating planar shock: periodic / far-field / outflow sides,
        # diffusion and exchange on, a thin grid that leaves most of the GPU idle.
        {"name": "planar shock 1024x8", "kind": "planar", "nx": 1024, "ny": 8, "steps": 20},
        # Double Mach reflection: the inverse Lax-Wendroff wall, an odd mesh.
        {"name": "double mach 402x283", "kind": "double_mach", "cells": 101, "steps": 10},
        # The half-cylinder at the reference's own mesh, one output interval.
        {"name": "cylinder 121x481", "kind": "cylinder", "nx": 121, "mach": 3.0, "source": False, "steps": 20},
        # The half-cylinder refined: the largest single solver.
        {"name": "cylinder 961x3841", "kind": "cylinder", "nx": 961, "mach": 3.0, "source": False, "steps": 5},
        # Ensembles of half-cylinders of uneven size, Mach number and
        # exchange coefficients: a small one, a large one, and the small one
        # in the contracted (FMA) build, which a program picks for speed.
        {"name": "batch of 24", "kind": "batch", "n": 24, "sizes": "61,91,121", "steps": 10, "exact": True},
        {"name": "batch of 96", "kind": "batch", "n": 96, "sizes": "61,91,121", "steps": 5, "exact": True},
        {"name": "batch of 24, fma", "kind": "batch", "n": 24, "sizes": "61,91,121", "steps": 10, "exact": False},
        # An ensemble whose state lives in host memory: copies in, one step, copies out.
        {"name": "batch host step 48", "kind": "batch_host_step", "n": 48, "sizes": "61,91,121"},
        # Gradient of a functional of the final state: the checkpointed
        # forward run and the reverse sweep.
        {"name": "gradient 8 x 121x481", "kind": "gradient", "n": 8, "sizes": "121", "steps": 10, "ckpt": 5},
        # Vector-Jacobian product of the operator, for an outer solver's own time loop.
        {"name": "operator vjp 61x241", "kind": "vjp", "nx": 61, "mach": 3.0, "source": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host_step", "operator", "planar", "double_mach", "cylinder", "cylinder", "batch", "batch",
                       "batch_host_step", "gradient", "vjp"])
    mach, source = round(rng.uniform(2.0, 4.0), 3), rng.random() < 0.5
    if kind in ("host_step", "operator", "vjp"):
        return {"kind": kind, "nx": _log_int(rng, 31, 181), "mach": mach, "source": source}
    if kind == "planar":
        return {"kind": kind, "nx": _log_int(rng, 128, 2048), "ny": _log_int(rng, 8, 32), "steps": rng.randint(5, 20)}
    if kind == "double_mach":
        return {"kind": kind, "cells": rng.randint(40, 120), "steps": rng.randint(5, 15)}
    if kind == "cylinder":
        nx = _log_int(rng, 31, 641)
        return {"kind": kind, "nx": nx, "mach": mach, "source": source, "steps": rng.randint(5, 20) if nx < 300 else 5}
    sizes = ",".join(str(_log_int(rng, 31, 121)) for _ in range(3))
    n = _log_int(rng, 2, 48)
    if kind == "batch":
        return {"kind": kind, "n": n, "sizes": sizes, "steps": rng.randint(3, 8), "exact": rng.random() < 0.7}
    if kind == "batch_host_step":
        return {"kind": kind, "n": n, "sizes": sizes}
    return {"kind": "gradient", "n": min(n, 8), "sizes": sizes, "steps": rng.randint(4, 10), "ckpt": rng.randint(2, 5)}


# ------------------------------------------------------------------ geometry
@functools.lru_cache(maxsize=16)
def _mesh(kind, nx, ny=0):
    """(Field, GhostGrid) of a mesh; the flow of a case is put on copies of the Field."""
    if kind == "cylinder":
        f = rh.cases.init_cylinder(h=3.0 / (nx - 1))
    elif kind == "double_mach":
        f = rh.cases.init_double_mach(h=1.0 / nx)
    else:
        ly = 4.0 * ny / nx  # square cells
        par = rh.Params(kappa_e=1e-3, kappa_i=1e-3, kappa_r=1e-3, omega_ei=1.0, omega_er=1.0, periodic_ly=ly)
        f = rh.cases.planar_shock(nx, ny, 4.0, ly, params=par)
    return f, rh.GhostGrid.build(f)


def _specs(case):
    """One dict per instance of a case: mesh, Mach number, exchange coefficients."""
    kind = case["kind"]
    if kind == "planar":
        return [dict(mesh=("planar", case["nx"], case["ny"]))]
    if kind == "double_mach":
        return [dict(mesh=("double_mach", case["cells"]))]
    if "sizes" in case:
        sizes = tuple(int(s) for s in case["sizes"].split(","))
        return [dict(mesh=("cylinder", s["nx"]), mach=s["mach"], omega_ei=s["omega_ei"], omega_er=s["omega_er"])
                for s in rh.cases.batch_specs(case["n"], sizes=sizes)]
    omega = 1.0 if case["source"] else 0.0
    return [dict(mesh=("cylinder", case["nx"]), mach=case["mach"], omega_ei=omega, omega_er=omega)]


# ------------------------------------------------------------------ flows
def _flow(spec, rng):
    """A Field on the spec's mesh with a developed, perturbed flow, and its GhostGrid."""
    base, ghosts = _mesh(*spec["mesh"])
    f, g = base.empty_like(), base.grid
    dev = torch.device("cuda")
    x = (g.x0 + g.dx * torch.arange(g.nx, dtype=torch.float64, device=dev))[:, None]
    y = (g.y0 + g.dy * torch.arange(g.ny, dtype=torch.float64, device=dev))[None, :]
    if spec["mesh"][0] == "cylinder":
        f.params = rh.Params(omega_ei=spec["omega_ei"], omega_er=spec["omega_er"])
        inflow = rh.cases.freestream(spec["mach"])
        f.bc_outer = [rh.BCType.FarField(inflow) if b.kind == rh.BCType.FAR_FIELD else b for b in base.bc_outer]
        # a bow shock smeared over 0.1: jumps of 0.8 times the normal shock's
        m2 = spec["mach"] ** 2
        r = torch.sqrt(x * x + y * y)
        cosphi = -x / torch.clamp(r, min=1e-3)
        s = 0.5 * (1.0 - torch.tanh((r - 1.5 - 0.8 * (1.0 - cosphi)) / 0.1)) * cosphi * cosphi
        rho = 1.0 + 0.8 * s * (2.4 * m2 / (0.4 * m2 + 2.0) - 1.0)
        p = 1.0 + 0.8 * s * ((2.8 * m2 - 0.4) / 2.4 - 1.0)
        un = spec["mach"] * math.sqrt(1.4)
        u, v = un * (1.0 - 0.7 * s), 0.3 * un * s * y / torch.clamp(r, min=1e-3)
        pk = [p / 3.0 * (1.0 + a * s) for a in (0.1, 0.05, -0.15)]
    else:
        w = torch.from_numpy(base.value).to(dev).reshape(g.nx, g.ny, 6)
        fl = torch.from_numpy(base.fluid).to(dev).reshape(g.nx, g.ny)
        rho = torch.where(fl, w[..., 0], torch.ones_like(w[..., 0]))
        u, v = w[..., 1] / rho, w[..., 2] / rho
        pk = [0.4 * (w[..., k] - rho * (u * u + v * v) / 6.0) for k in (3, 4, 5)]
    lx, ly = g.dx * g.nx, g.dy * g.ny

    def wave(amp):
        out = torch.ones_like(rho)
        for _ in range(2):
            kx, ky = 2.0 * math.pi * rng.integers(1, 5) / lx, 2.0 * math.pi * rng.integers(1, 4) / ly
            out = out + amp * torch.sin(kx * (x - g.x0) + rng.uniform(0.0, 6.28)) * torch.cos(ky * (y - g.y0))
        return out

    rho, u, pk = rho * wave(0.01), u * wave(0.01), [q * wave(0.01) for q in pk]
    v = v + 0.01 * (wave(1.0) - 1.0)
    k = rho * (u * u + v * v) / 6.0
    w = torch.stack(torch.broadcast_tensors(rho, rho * u, rho * v, *[q / 0.4 + k for q in pk]), dim=-1).reshape(-1, 6)
    w = torch.where(torch.from_numpy(base.fluid).to(dev)[:, None], w, torch.zeros_like(w))
    f.value = _pinned(w.shape)
    torch.from_numpy(f.value).copy_(w)
    f.time = 0.0
    return f, ghosts


def _pinned(shape):
    """A page-locked host array, as a program that moves fields each step holds."""
    return torch.empty(tuple(shape), dtype=torch.float64, pin_memory=True).numpy()


def _flows(case, seed):
    rng = np.random.default_rng(seed)
    return [_flow(s, rng) for s in _specs(case)]


def prepare(case, seed):
    flows = _flows(case, seed)
    fields, grids = [f for f, _ in flows], [g for _, g in flows]
    st = {"case": case, "fields": fields}
    if case["kind"] in ("host_step", "operator", "planar", "double_mach") or \
            (case["kind"] == "cylinder" and case["nx"] <= 300):
        st["solver"] = rh.Solver(fields[0], grids[0])
        st["value"], st["time"], st["passes"] = fields[0].value.copy(), 0.0, 0
        return st
    # ensembles, adjoints, and large single fields in page-locked arrays
    st["solver"] = b = rh.Batch(fields, grids, exact=case.get("exact", True))
    total = int(b.offsets[-1])
    st["values"], st["times"] = _pinned((total, 6)), np.zeros(b.n)
    np.concatenate([f.value for f in fields], out=st["values"])
    st["out"], st["times_out"], st["passes"] = _pinned((total, 6)), np.zeros(b.n), 0
    if case["kind"] in ("gradient", "vjp"):
        gen = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
        lam = torch.randn((total, 6), dtype=torch.float64, device="cuda", generator=gen)
        fluid = torch.from_numpy(np.concatenate([f.fluid for f in fields])).cuda()
        st["cotangent"] = _pinned((total, 6))
        torch.from_numpy(st["cotangent"]).copy_(lam * fluid[:, None])
    return st


# ------------------------------------------------------------------ one pass
def run(st):
    case, s = st["case"], st["solver"]
    kind = case["kind"]
    if kind == "host_step":
        st["passes"] += 1
        if st["passes"] > LOOP:
            st["value"][:], st["time"], st["passes"] = st["fields"][0].value, 0.0, 1
        st["time"], dt = s.step_host(st["value"], st["time"], CFL)
        return {"value": st["value"], "time": st["time"], "dt": dt}
    if kind == "operator":
        rhs, ghosts = s.l(with_ghosts=True)
        return {"rhs": rhs, "ghosts": ghosts}
    if kind == "vjp":
        ubar, pbar = s.l_vjp(0, st["cotangent"])
        return {"ubar": ubar, "pbar": pbar}
    if kind == "batch_host_step":
        if st["passes"] % LOOP == 0:
            st["out"][:], st["times_out"][:] = st["values"], st["times"]
        st["passes"] += 1
        s.step_host(st["out"], st["times_out"], CFL)
        return {"values": st["out"], "times": st["times_out"]}
    if isinstance(s, rh.Solver):
        s.upload(st["fields"][0])
        s.advance(case["steps"], CFL)
        value, t = s.download()
        return {"value": value, "time": t}
    s.upload_values(st["values"], st["times"])
    if kind == "gradient":
        s.adjoint_forward(case["steps"], CFL, ckpt_every=case["ckpt"])
        values, times = s.download_values(st["out"], st["times_out"])
        if "grad" not in st:
            st["grad"] = _pinned(values.shape)
        _, dparams = s.adjoint_backward(st["cotangent"], out=st["grad"])
        return {"values": values, "times": times, "dvalues": st["grad"], "dparams": dparams}
    s.advance(case["steps"], CFL)
    values, times = s.download_values(st["out"], st["times_out"])
    return {"values": values, "times": times}


# ------------------------------------------------------------------ bounds
@functools.lru_cache(maxsize=64)
def _counts(mesh):
    f, g = _mesh(*mesh)
    nfx, nfy = flops.face_counts(f.fluid, f.grid.nx, f.grid.ny)
    return dict(cells=f.grid.len(), fluid=int(f.fluid.sum()), nfx=nfx, nfy=nfy, ghosts=g.len(), heavy=g.n_heavy(),
                planar=mesh[0] == "planar")


def work(case):
    """Bytes: the field in and out and the ghost tables, once. Operations: the
    reference algorithm's, per step; the reverse sweep of a step counts twice
    its forward (the products of a vector-Jacobian product)."""
    kind, specs = case["kind"], _specs(case)
    bytes_, fl = 0.0, 0.0
    for s in specs:
        c = _counts(s["mesh"])
        source = c["planar"] or s.get("omega_ei", 0.0) != 0.0
        step = flops.step_flops(c["fluid"], c["nfx"], c["nfy"], c["ghosts"], c["heavy"], c["planar"], source)
        steps = {"host_step": 1, "batch_host_step": 1, "operator": 1.0 / 3.0, "vjp": 1.0 / 3.0}.get(kind) or case["steps"]
        fl += step * steps * (3.0 if kind in ("gradient", "vjp") else 1.0)
        bytes_ += 2 * 48.0 * c["fluid"] + flops.ghost_launch_bytes(c["heavy"])
        if kind in ("gradient", "vjp"):
            bytes_ += 2 * 48.0 * c["fluid"]
        if kind == "operator":
            bytes_ += 48.0 * c["ghosts"]
    return {"bytes": bytes_, "flops": fl}


def _cfl_dt(f):
    """The reference driver's time step: CFL times the smallest local time
    step lambda / ((|u| + c) / dx + 2 d / (dx^2 + dy^2) + s + (|v| + c) / dy)
    over the fluid nodes, s the larger rate of the linearised exchange terms."""
    P, w = f.params, f.value[f.fluid].astype(np.longdouble)
    rho, u, v = w[:, 0], w[:, 1] / w[:, 0], w[:, 2] / w[:, 0]
    ee, ei, er = (w[:, k] / rho - (u * u + v * v) / 6 for k in (3, 4, 5))
    ge, gi, gr = P.gamma_e, P.gamma_i, P.gamma_r
    c = np.sqrt(ge * (ge - 1) * ee + gi * (gi - 1) * ei + gr * (gr - 1) * er)
    A, oei, oer, ce, ci = P.a_rad, P.omega_ei, P.omega_er, P.cve, P.cvi
    t = A * oei * ce**4 + A * oei * ce**3 * ci + 4 * A * oer * ci * ee**3 + oer * ce**4 * ci * rho
    root = np.sqrt(np.maximum(t * t - 4 * A * oei * oer * ce**4 * ci * (4 * A * ee**3 + ce**4 * rho + ce**3 * ci * rho), 0))
    rate = (t + root) / (2 * A * ce**4 * ci * rho)
    d = np.maximum(np.maximum(P.kappa_e / (ce * rho), P.kappa_i / (ci * rho)), P.kappa_r / A)
    dx, dy = f.grid.dx, f.grid.dy
    return float(CFL * (P.lambda_ / ((abs(u) + c) / dx + 2 * d / (dx * dx + dy * dy) + rate + (abs(v) + c) / dy)).min())


def exact(case, seed):
    """The time and the time step of one-step cases (the operator, the fields
    and the gradients are themselves 64-bit results of long ordered sums: no
    plain formula gives them in wider precision)."""
    if case["kind"] == "host_step":
        dt = _cfl_dt(_flows(case, seed)[0][0])
        return {"value": None, "time": dt, "dt": dt}
    if case["kind"] == "batch_host_step":
        return {"values": None, "times": np.array([_cfl_dt(f) for f, _ in _flows(case, seed)])}
    return None
