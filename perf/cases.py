"""Performance cases of the per-level LBM time step, through the package's
public entry points (Mesh / GpuLattice and the case builders of
octlb_b200.cases).

A pass is what a driver program does between two outputs: a number of
advance_one calls, then the quantities it reads back (fields into pinned host
arrays, the momentum-exchange force, the audit, populations for a restart).
The inputs are seeded smooth fields of the sizes and amplitudes the solver is
used at.  ``listed()`` names the cases, ``draw()`` gives more of the same
ranges, ``exact()`` the FP64 result where plain torch can give it quickly
(the periodic boxes).
"""
import math

import numpy as np
import torch

import octlb_b200 as ob
from octlb_b200 import cases as ob_cases

Q = 19
FLOPS_PER_UPDATE = 250  # moments, equilibrium, relaxation of 19 populations


def listed():
    return [
        # The smallest call: a 32^3 periodic box advanced one step at a time by
        # a program that watches mass / momentum and the fields every step.
        {"name": "monitor_32", "kind": "box", "n": 32, "precision": "fp32", "order": "ab", "steps": 1,
         "io": "audit", "tau": 0.6, "u0": 0.05},
        # The reference's cavity3d example: one 31^3 block, finite-difference
        # velocity faces, ConstRhoBGK (FP32).
        {"name": "cavity3d_31", "kind": "cavity3d", "resolution": 30, "precision": "fp32", "steps": 100},
        # The Taylor-Green accuracy configuration: small box, many steps
        # between outputs.
        {"name": "box_64", "kind": "box", "n": 64, "precision": "fp32", "order": "ab", "steps": 200, "io": "fields",
         "tau": 0.55, "u0": 0.05},
        # A run segment between restart files (populations in and out) on a
        # ragged box edge, FP16-shifted storage.
        {"name": "restart_90_fp16", "kind": "box", "n": 90, "precision": "fp16", "order": "ab", "steps": 200,
         "io": "restart", "tau": 0.56, "u0": 0.04},
        # The throughput configuration, FP32 and FP16-shifted.
        {"name": "box_256", "kind": "box", "n": 256, "precision": "fp32", "order": "ab", "steps": 200, "io": "fields",
         "tau": 0.55, "u0": 0.05},
        {"name": "box_256_fp16", "kind": "box", "n": 256, "precision": "fp16", "order": "ab", "steps": 200,
         "io": "fields", "tau": 0.55, "u0": 0.05},
        # A box chosen for memory: the one-buffer (AA) stream order, an edge
        # that is no power of two.
        {"name": "box_320_aa", "kind": "box", "n": 320, "precision": "fp32", "order": "aa", "steps": 100,
         "io": "fields", "tau": 0.55, "u0": 0.05},
        # Lid-driven cavity with a refined band under the lid (two levels).
        {"name": "amr_cavity_64", "kind": "cavity", "cells": 64, "band": 8, "precision": "fp32", "const_rho": False,
         "coupler": "reference", "steps": 50, "tau": 0.56, "lid": 0.05},
        # Lid-driven cavity on one fine level, ConstRhoBGK.
        {"name": "const_rho_cavity_128", "kind": "cavity", "cells": 128, "band": 0, "precision": "fp32",
         "const_rho": True, "coupler": "reference", "steps": 20, "tau": 0.56, "lid": 0.05},
        # Channel flow past a cylinder (three levels, Bouzidi links, drag).
        {"name": "cylinder_256", "kind": "cylinder", "height": 64, "length": 256, "n": 8, "levels": 3,
         "diameter": 16.0, "precision": "fp32", "steps": 100, "u_max": 0.05, "re": 100.0},
        # The same channel at twice the resolution, FP16-shifted storage.
        {"name": "cylinder_512_fp16", "kind": "cylinder", "height": 128, "length": 512, "n": 8, "levels": 3,
         "diameter": 32.0, "precision": "fp16", "steps": 50, "u_max": 0.05, "re": 100.0},
        # Gradients of the mean drag: forward with checkpoints, then the
        # adjoint sweep back (the adjoint configuration's channel).
        {"name": "adjoint_channel", "kind": "adjoint", "steps": 256, "window": 64, "interval": 16, "u_max": 0.05},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "box", "box", "cavity3d", "cavity", "cavity", "cylinder", "cylinder", "adjoint"])
    precision = rng.choice(["fp32", "fp16"])
    tau = round(rng.uniform(0.52, 0.9), 3)
    u = round(rng.uniform(0.02, 0.08), 4)
    if kind == "box":
        order = rng.choice(["ab", "ab", "aa"])
        n = _log_int(rng, 16, 288)
        if order == "aa":
            n += n % 2
        steps = max(1, min(400, int(1.2e9 / n ** 3)))
        io = rng.choice(["fields", "audit", "restart"]) if n <= 128 else "fields"
        return {"kind": kind, "n": n, "precision": precision, "order": order, "steps": steps, "io": io, "tau": tau,
                "u0": u}
    if kind == "cavity3d":
        return {"kind": kind, "resolution": rng.randint(14, 60), "precision": precision, "steps": rng.randint(20, 150)}
    if kind == "cavity":
        cells = rng.choice([32, 64, 64, 128])
        band = rng.choice([0, 8, 16]) if cells < 128 else 0
        const_rho = rng.random() < 0.4
        return {"kind": kind, "cells": cells, "band": band, "precision": precision, "const_rho": const_rho,
                "coupler": "physical" if band and not const_rho and rng.random() < 0.4 else "reference",
                "steps": rng.randint(5, 20) if cells == 128 else rng.randint(10, 60), "tau": tau, "lid": u}
    if kind == "cylinder":
        height = rng.choice([32, 64, 64, 128])
        n = 16 if height == 64 and rng.random() < 0.25 else 8
        levels = rng.choice([2, 3])
        return {"kind": kind, "height": height, "length": height * rng.choice([2, 4] if height < 128 else [2]), "n": n,
                "levels": levels, "diameter": float(height // 4), "precision": precision,
                "steps": rng.randint(10, 40) if height == 128 else rng.randint(20, 100), "u_max": u,
                "re": round(rng.uniform(20.0, 150.0), 1)}
    steps = rng.randint(32, 256)
    return {"kind": "adjoint", "steps": steps, "window": max(1, steps // 4), "interval": rng.choice([0, 8, 16]),
            "u_max": u}


def _precision(case):
    return ob.FP16_SHIFTED if case.get("precision") == "fp16" else ob.FP32


def _elem(case):
    return 2 if case.get("precision") == "fp16" else 4


def _mesh(case):
    """(mesh, info) of a case, without its initial state."""
    k = case["kind"]
    if k == "box":
        return ob.Mesh(case["n"], [0], [0, 0, 0, 1, 1, 1], periodic=1), {"omega": 1.0 / case["tau"]}
    if k == "cavity3d":
        mesh, _, info = ob_cases.cavity3d(resolution=case["resolution"])
        return mesh, info
    if k == "cavity":
        mesh, _, info = ob_cases.cavity_forest(cells=case["cells"], n=8, lid=case["lid"], tau=case["tau"],
                                               band_cells=case["band"])
        return mesh, info
    if k == "cylinder":
        h = case["height"]
        mesh, _, info = ob_cases.cylinder_forest(length=case["length"], height=h, n=case["n"],
                                                 diameter=case["diameter"], center=(h * 1.0, h / 2.0),
                                                 levels=case["levels"], u_max=case["u_max"], re=case["re"])
        return mesh, info
    mesh, _, info = ob_cases.adjoint_channel(u_max=case["u_max"])
    return mesh, info


def _box_fields(case, seed, device):
    """Seeded Taylor-Green-like fields of a periodic n^3 box: the vortex with
    random phases plus a weaker second harmonic, FP64."""
    n, u0 = case["n"], case["u0"]
    rng = np.random.default_rng(seed)
    ph = rng.uniform(0.0, 2.0 * math.pi, size=6)
    am = rng.uniform(0.7, 1.0)
    c = (torch.arange(n, dtype=torch.float64, device=device) + 0.5) * (2.0 * math.pi / n)
    x, y, z = c[:, None, None], c[None, :, None], c[None, None, :]
    u = torch.empty((n, n, n, 3), dtype=torch.float64, device=device)
    u[..., 0] = am * u0 * torch.sin(x + ph[0]) * torch.cos(y + ph[1]) * torch.cos(z + ph[2])
    u[..., 1] = -am * u0 * torch.cos(x + ph[0]) * torch.sin(y + ph[1]) * torch.cos(z + ph[2])
    u[..., 2] = 0.2 * u0 * torch.sin(2 * x + ph[3]) * torch.cos(2 * y + ph[4])
    rho = 1.0 + 3.0 * u0 * u0 / 16.0 * (torch.cos(2 * x + ph[5]) + torch.cos(2 * y + ph[3])) * (torch.cos(2 * z) + 2.0)
    return rho.contiguous(), u


def _forest_fields(mesh, seed, amplitude):
    """Seeded smooth disturbance of the rest state on every leaf's cells."""
    rng = np.random.default_rng(seed)
    ph = rng.uniform(0.0, 2.0 * math.pi, size=6)
    n, nb = mesh.n, mesh.n_blocks
    lo, hi = mesh.bounds[:, :3], mesh.bounds[:, 3:]
    span = hi.max(axis=0) - lo.min(axis=0)
    s = (np.arange(n) + 0.5) / n
    xyz = [(lo[:, a, None] + s[None, :] * (hi - lo)[:, a, None]) * (2.0 * math.pi / span[a]) for a in range(3)]
    x, y, z = xyz[0][:, :, None, None], xyz[1][:, None, :, None], xyz[2][:, None, None, :]
    u = np.empty((nb, n, n, n, 3))
    u[..., 0] = amplitude * np.sin(x + ph[0]) * np.cos(y + ph[1]) * np.cos(z + ph[2])
    u[..., 1] = -amplitude * np.cos(x + ph[0]) * np.sin(y + ph[1]) * np.cos(z + ph[2])
    u[..., 2] = 0.5 * amplitude * np.sin(x + ph[3]) * np.cos(y + ph[4])
    rho = 1.0 + amplitude * amplitude * np.cos(x + ph[5]) * np.cos(2 * y) * np.ones_like(z)
    return rho, u


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def prepare(case, seed):
    mesh, info = _mesh(case)
    k = case["kind"]
    cells = mesh.n_blocks * mesh.n ** 3
    state = {"case": case, "rho": _pinned((cells,)), "u": _pinned((cells, 3))}
    if k == "box":
        lat = ob.GpuLattice(mesh, info["omega"], precision=_precision(case),
                            stream_order=ob.ORDER_AA if case["order"] == "aa" else ob.ORDER_AB)
        rho, u = _box_fields(case, seed, "cuda")
        torch.from_numpy(state["rho"]).copy_(rho.reshape(-1))
        torch.from_numpy(state["u"]).copy_(u.reshape(-1, 3))
        if case["io"] == "restart":
            state["pops"] = _feq(rho, u).permute(1, 2, 3, 0).contiguous().cpu().numpy()
    else:
        amplitude = 0.01
        if k == "cavity3d":
            lat = ob.GpuLattice(ob.stamp_fd_kinds(mesh, info["types"]), info["omega"], precision=_precision(case))
            lat.set_const_rho(True)
            lat.set_fd_boundary(info["types"], info["u_wall"])
        elif k == "cavity":
            lat = ob.GpuLattice(mesh, info["omega"], precision=_precision(case), coupler_mode=(
                ob.COUPLER_PHYSICAL if case["coupler"] == "physical" else ob.COUPLER_REFERENCE))
            if case["const_rho"]:
                lat.set_const_rho(True)
        else:
            lat = ob.GpuLattice(mesh, info["omega"], precision=_precision(case), stream_mode=ob.STREAM_LINKS,
                                drag=True)
        rho, u = _forest_fields(mesh, seed, amplitude)
        state["rho"][:] = rho.reshape(-1)
        state["u"][:] = u.reshape(-1, 3)
    lat.set_equilibrium(state["rho"], state["u"])
    state["lat"] = lat
    return state


def run(state):
    case, lat = state["case"], state["lat"]
    k = case["kind"]
    if k == "adjoint":
        J, du, dtau, dforce = lat.adjoint(case["steps"], case["window"], case["interval"])
        return {"J": J, "dJ_du": du, "dJ_dtau": dtau, "dJ_dF": dforce}
    if k == "box" and case["io"] == "restart":
        lat.set_populations(state["pops"])
        lat.advance(case["steps"])
        return {"pops": lat.get_populations()}
    lat.advance(case["steps"])
    out = {}
    if k == "cylinder":
        out["force"] = lat.force()
    if k == "box" and case["io"] == "audit":
        out["audit"] = lat.audit()
    out["rho"], out["u"] = lat.get_fields(state["rho"], state["u"])
    return out


_updates = {}


def _updates_per_call(case):
    """Lattice updates of one advance_one, and cells."""
    key = tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "steps", "precision")))
    if key not in _updates:
        mesh, _ = _mesh(case)
        _updates[key] = (mesh.lattice_updates_per_coarse_step(), mesh.n_blocks * mesh.n ** 3)
    return _updates[key]


def work(case):
    """Every level step reads and writes its populations once; the outputs
    are written once.  The adjoint's reverse sweep touches the step's input
    and the two cotangent states of every step, on top of the forward."""
    lups, cells = _updates_per_call(case)
    lups *= case["steps"]
    per_update = 2 * Q * _elem(case)
    if case["kind"] == "adjoint":
        return {"bytes": lups * (per_update + 3 * Q * 4) + cells * 24, "flops": lups * 3 * FLOPS_PER_UPDATE}
    io = cells * (2 * Q * 8 if case.get("io") == "restart" else 32)
    return {"bytes": lups * per_update + io, "flops": lups * FLOPS_PER_UPDATE}


# ---- FP64 in plain torch: BGK on a periodic box

_C = [(0, 0, 0), (-1, 0, 0), (0, -1, 0), (0, 0, -1), (-1, -1, 0), (-1, 1, 0), (-1, 0, -1), (-1, 0, 1), (0, -1, -1),
      (0, -1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, -1, 0), (1, 0, 1), (1, 0, -1), (0, 1, 1), (0, 1, -1)]
_W = [1 / 3 if c == (0, 0, 0) else (1 / 18 if sum(abs(v) for v in c) == 1 else 1 / 36) for c in _C]


def _feq(rho, u):
    """Shifted equilibrium [19][n][n][n]."""
    out = torch.empty((Q,) + tuple(rho.shape), dtype=torch.float64, device=rho.device)
    usq = 1.5 * (u * u).sum(-1)
    for i, (c, w) in enumerate(zip(_C, _W)):
        cu = c[0] * u[..., 0] + c[1] * u[..., 1] + c[2] * u[..., 2]
        out[i] = rho * w * (1.0 + 3.0 * cu + 4.5 * cu * cu - usq) - w
    return out


def _moments(f):
    rho = 1.0 + f.sum(0)
    u = torch.empty(tuple(rho.shape) + (3,), dtype=torch.float64, device=f.device)
    for a in range(3):
        j = torch.zeros_like(rho)
        for i, c in enumerate(_C):
            if c[a]:
                j += c[a] * f[i]
        u[..., a] = j / rho
    return rho, u


def _collide(f, omega):
    rho, u = _moments(f)
    usq = 1.5 * (u * u).sum(-1)
    for i, (c, w) in enumerate(zip(_C, _W)):
        cu = c[0] * u[..., 0] + c[1] * u[..., 1] + c[2] * u[..., 2]
        f[i] += omega * (rho * w * (1.0 + 3.0 * cu + 4.5 * cu * cu - usq) - w - f[i])
    return f


def exact(case, seed):
    if case["kind"] != "box":
        return None  # the forests' couplers and boundary passes are no few lines of torch
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["n"] ** 3 * case["steps"] > (4e9 if device == "cuda" else 1e8):
        return None
    rho, u = _box_fields(case, seed, device)
    f = _feq(rho, u)
    omega = 1.0 / case["tau"]
    for _ in range(case["steps"]):
        _collide(f, omega)
        for i, c in enumerate(_C):
            if i:
                f[i] = torch.roll(f[i], shifts=c, dims=(0, 1, 2))
    if case["io"] == "restart":
        g = _collide(f, omega).permute(1, 2, 3, 0).contiguous().cpu().numpy()
        return {"pops": g[None]}
    rho, u = _moments(f)
    out = {}
    if case["io"] == "audit":
        out["audit"] = torch.stack([rho.sum()] + [(rho * u[..., a]).sum() for a in range(3)]).cpu().numpy()
    out["rho"], out["u"] = rho.cpu().numpy()[None], u.cpu().numpy()[None]
    return out
