"""Timed work of the solver: the calls that a program makes through ``exasim_b200.HDGSolver``.

A case names one step of the solver on one of the package's models:

* ``krylov``    w = P A v: one application of the condensed operator (``evalMatVec``) and of the
                preconditioner (``ApplyPreconditioner``), for a program with its own Krylov method
* ``residual``  q from the trace and the residual vectors and norm at the current state
                (``hdgGetQ``, ``hdgAssembleResidual``; LDG: ``evalResidual``)
* ``assemble``  the condensed system and its preconditioner (``hdgAssembleLinearSystem``)
* ``gmres``     the solve of the assembled system (``GMRES``; LDG: of J(u) x = -R(u))
* ``solve``     one whole Newton solve from pinned host buffers to host buffers (``solve``)

``listed`` gives the fixed cases, ``draw`` further ones of the same ranges, ``prepare`` the inputs and
the context that a program holds before the call, ``run`` one pass, ``work`` what a pass cannot do
without, ``tolerance`` how far two right implementations may differ, and ``exact`` the results in
64 bits by plain torch: a restatement of the discretisation on dense blocks that takes from the
package only the input tables (nodes, shape functions, mesh) and the numbering of the faces.
"""
from __future__ import annotations

import functools
import math
import os
import tempfile

import numpy as np
import torch

from exasim_b200 import HDGSolver, cases, inputs, read_datain
from exasim_b200.serve import with_params

DEV = "cuda"


def listed():
    return [
        # an external Krylov method on the smallest mesh of the served stream: launches and
        # synchronisation count
        {"name": "krylov_cdsin2d_q8_p2", "step": "krylov", "model": "cdsin2d", "n": 8, "p": 2, "form": "plain"},
        # the same on large blocks (480 x 480) in the mixed form's 32-bit matrices
        {"name": "krylov_euler3d_h12_p3_mixed", "step": "krylov", "model": "euler3d", "n": 12, "p": 3, "form": "mixed"},
        # the residual of a Newton line search: a system with q on an odd 2D mesh
        {"name": "residual_ns2d_q33_p3", "step": "residual", "model": "ns2d", "n": 33, "p": 3, "form": "plain"},
        # the LDG residual, which explicit and matrix-free drivers evaluate over and over
        {"name": "residual_ldg_euler3d_h20_p3", "step": "residual", "model": "euler3d_ldg", "n": 20, "p": 3, "form": "plain"},
        # assembly on 512 perturbed triangles with the additive Schwarz preconditioner
        {"name": "assemble_poisson2d_t16_p3", "step": "assemble", "model": "poisson2d", "n": 16, "p": 3, "form": "plain"},
        # assembly with q elimination in 3D: both forms, an odd mesh and the benchmark's mesh
        {"name": "assemble_convdiff3d_h11_p4", "step": "assemble", "model": "convdiff3d", "n": 11, "p": 4, "form": "plain"},
        {"name": "assemble_convdiff3d_h16_p4_mixed", "step": "assemble", "model": "convdiff3d", "n": 16, "p": 4, "form": "mixed"},
        # assembly of large blocks without q (320 x 320 element inverses)
        {"name": "assemble_euler3d_h10_p3", "step": "assemble", "model": "euler3d", "n": 10, "p": 3, "form": "plain"},
        # the linear solve of a Navier-Stokes stage: GMRES(100) with block ILU(0)
        {"name": "gmres_ns2d_q32_p3", "step": "gmres", "model": "ns2d", "n": 32, "p": 3, "form": "plain"},
        # the matrix-free linear solve of a pseudo-transient step: the longest call of the list
        {"name": "gmres_ldg_euler3d_h12_p3", "step": "gmres", "model": "euler3d_ldg", "n": 12, "p": 3, "form": "plain"},
        # one request of the served stream, from host buffers to host buffers
        {"name": "solve_cdsin2d_q24_p3", "step": "solve", "model": "cdsin2d", "n": 24, "p": 3, "form": "plain"},
        # one DIRK stage of the benchmark workload, from host buffers to host buffers
        {"name": "solve_convdiff3d_h16_p4_mixed", "step": "solve", "model": "convdiff3d", "n": 16, "p": 4, "form": "mixed"},
    ]


# (step, model, form, elements per side, orders): n is drawn over its logarithm; the upper ends cost no
# more than the longest listed case.  Block ILU(0) wants n in sub-domains of 4 x 4 elements.
RANGES = [
    ("krylov", "cdsin2d", "plain", (8, 64), (2, 3, 4)),
    ("krylov", "convdiff3d", "plain", (5, 15), (3, 4)),
    ("krylov", "convdiff3d", "mixed", (5, 15), (4,)),
    ("krylov", "euler3d", "mixed", (4, 11), (2, 3)),
    ("residual", "ns2d", "plain", (9, 64), (2, 3)),
    ("residual", "convdiff3d", "plain", (5, 15), (2, 3, 4)),
    ("residual", "euler3d_ldg", "plain", (5, 22), (2, 3)),
    ("assemble", "poisson2d", "plain", (6, 32), (2, 3)),
    ("assemble", "convdiff3d", "plain", (5, 14), (3, 4)),
    ("assemble", "convdiff3d", "mixed", (6, 15), (4,)),
    ("assemble", "euler3d", "plain", (4, 9), (2, 3)),
    ("assemble", "euler3d", "mixed", (4, 11), (3,)),
    ("gmres", "ns2d", "plain", (8, 40), (2, 3)),
    ("gmres", "convdiff3d", "plain", (5, 15), (3, 4)),
    ("gmres", "euler3d_ldg", "plain", (4, 10), (2, 3)),
    ("solve", "cdsin2d", "plain", (8, 48), (2, 3, 4)),
    ("solve", "cdsin2d", "mixed", (8, 32), (2, 3, 4)),
    ("solve", "convdiff3d", "mixed", (6, 15), (4,)),
    ("solve", "convdiff3d", "plain", (6, 14), (3, 4)),
]


def draw(rng):
    step, model, form, (lo, hi), orders = rng.choice(RANGES)
    n = min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))
    if step == "gmres" and model == "ns2d":
        n = 4 * max(2, round(n / 4))
    return {"step": step, "model": model, "n": n, "p": rng.choice(orders), "form": form}


# ------------------------------------------------------------------ inputs
PARAMS = {"ns2d": [1.4, 1600.0, 0.72, 0.1], "euler3d": [1.4, 0.5], "poisson2d": [1.0]}


@functools.lru_cache(maxsize=4)
def _datain(step, model, n, p, mesh_seed):
    """The app, master, mesh and sol blobs of a mesh, as the package's preprocessor writes them."""
    with tempfile.TemporaryDirectory() as tmp:
        d = os.path.join(tmp, "datain")
        if model == "poisson2d":
            cases.poisson2d_tri(d, n=n, porder=p, seed=mesh_seed, preconditioner=1)
        elif model == "cdsin2d":
            cases.cdsin2d_quad(d, n=n, porder=p, gmres_tol=1e-11 if step == "solve" else 1e-8)
        elif model == "convdiff3d":
            cases.convdiff3d_hex(d, n=n, porder=p)
        elif model == "ns2d":
            cases.ns2d_tgv_quad(d, n=n, porder=p, preconditioner=2 if step == "gmres" else 0)
        else:
            cases.euler3d_vortex_hex(d, n=n, porder=p, hybrid=0 if model == "euler3d_ldg" else 1)
        return read_datain(d)


def _smooth(x, length, rng):
    """A seeded sum of eight waves over the domain, of size one."""
    s = np.zeros(x.shape[0])
    for _ in range(8):
        k = rng.integers(1, 4, x.shape[1]) * rng.choice([-1, 1], x.shape[1])
        s += np.sin(2 * np.pi / length * (x @ k) + rng.uniform(0, 2 * np.pi))
    return s / 4.0


def _inputs(case, seed):
    """What the call starts from: blobs with seeded parameters and state, and the DIRK stage's
    time, factor and source.  x [ne, npe, nd] are the element nodes, u [ne, ncu, npe] the state."""
    model, n, p = case["model"], case["n"], case["p"]
    rng = np.random.default_rng(seed)
    blobs = list(_datain(case["step"], model, n, p, seed if model == "poisson2d" else 0))
    master = inputs.read_blob(blobs[1].tobytes())
    nd, npe = int(master[1][0]), int(master[1][5])
    sol = inputs.read_blob(blobs[3].tobytes())
    x = sol[2].reshape(-1, nd, npe).transpose(0, 2, 1)
    ne = x.shape[0]
    X = x.reshape(-1, nd)
    dtf = 0.0
    if model in ("poisson2d", "cdsin2d"):
        # steady linear problems from a rough guess of the solution
        if model == "cdsin2d":
            th = rng.uniform(0, 2 * np.pi)
            params = [0.03, math.cos(th), math.sin(th), float(rng.integers(1, 4)), float(rng.integers(1, 4))]
        else:
            params = PARAMS["poisson2d"]
        u = 0.1 * (np.prod(np.sin(np.pi * X), axis=1) * (1 + 0.3 * _smooth(X, 1.0, rng)))[:, None]
    elif model == "convdiff3d":
        # a later step of the transport: the source's plume, carried and spread
        c = rng.normal(size=3)
        c *= 1.15 / np.linalg.norm(c)
        x0 = rng.uniform(0.35, 0.65, 3)
        params = [0.01, *c, *x0, 0.1]
        u = sum(0.02 * np.exp(-((X - x0 - t * c) ** 2).sum(1) / (2 * (0.01 + 0.02 * t))) for t in (0.0, 0.05, 0.1, 0.15))
        u = (u * (1 + 0.05 * _smooth(X, 1.0, rng)))[:, None]
        dtf = 2.294280360323567 / 0.01
    elif model == "ns2d":
        params = PARAMS["ns2d"]
        gam, M = params[0], params[3]
        s = 1 + 0.02 * _smooth(X, 2 * np.pi, rng)
        ux, uy = np.sin(X[:, 0]) * np.cos(X[:, 1]) * s, -np.cos(X[:, 0]) * np.sin(X[:, 1]) * s
        rho = 1 + 1e-3 * _smooth(X, 2 * np.pi, rng)
        pr = 1 / (gam * M * M) + (np.cos(2 * X[:, 0]) + np.cos(2 * X[:, 1])) / 4
        u = np.stack([rho, rho * ux, rho * uy, pr / (gam - 1) + 0.5 * rho * (ux**2 + uy**2)], 1)
        dtf = 2.294280360323567 / 0.05
    else:
        params = PARAMS["euler3d"]
        gam, M = params
        r2 = X[:, 0] ** 2 + X[:, 1] ** 2
        rho = (1 - (gam - 1) / (16 * np.pi**2) * 25 * np.exp(2 * (1 - r2))) ** (1 / (gam - 1))
        a = 5 * np.exp(1 - r2) / (2 * np.pi * M)
        v = np.stack([1 - a * X[:, 1], a * X[:, 0], 0.05 * _smooth(X, 10.0, rng)], 1)
        pr = rho**gam / (gam * M * M)
        rho = rho * (1 + 5e-3 * _smooth(X, 10.0, rng))
        u = np.concatenate([rho[:, None], rho[:, None] * v, (pr / (gam - 1) + 0.5 * rho * (v**2).sum(1))[:, None]], 1)
        dtf = 3.414213562373096 / 0.05
    u = np.ascontiguousarray(u.reshape(ne, npe, -1).transpose(0, 2, 1))
    if model in ("cdsin2d", "convdiff3d"):
        blobs[0] = with_params(blobs[0], params)
    with tempfile.TemporaryDirectory() as tmp:
        fn = os.path.join(tmp, "sol.bin")
        app = inputs.read_blob(blobs[0].tobytes())
        inputs.write_sol_bin(fn, sol[2].reshape(npe, nd, ne, order="F"), udg=u.transpose(2, 1, 0), nc=int(app[1][5]),
                             ncu=u.shape[1])
        blobs[3] = np.fromfile(fn)
    return {"blobs": blobs, "params": params, "u": u, "time": 0.4 / dtf if dtf else 0.0, "dtfactor": dtf,
            "sdg": dtf * u if dtf else None, "tau": float(app[9][0]), "seed": seed}


def _trace(uh, seed):
    """A trace in the midst of a Newton solve: not quite the elements' own values."""
    return uh * (1.0 + 1e-4 * np.random.default_rng(seed + 1).standard_normal(uh.size))


def _library(model):
    return "euler3d" if model == "euler3d_ldg" else model


class _Device:
    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner  # the tensor made of this keeps the solver, and so its memory
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 3}


def _view(s, name, typestr="<f8"):
    """A solver field as a torch tensor on its own device memory."""
    ptr, n = s.field_ptr(name)
    return torch.as_tensor(_Device(s, ptr, n, typestr), device=DEV)


def _vector(case, seed, N):
    """A Krylov vector: entries of one sign and size are not met there."""
    g = torch.Generator().manual_seed(seed)
    return torch.randn(N, generator=g, dtype=torch.float64)


def prepare(case, seed):
    i = _inputs(case, seed)
    step, mixed, ldg = case["step"], case["form"] == "mixed", case["model"] == "euler3d_ldg"
    s = HDGSolver("", _library(case["model"]), blobs=i["blobs"])
    if mixed:
        # the inner tolerance of the package's benchmark for its serving requests and its stages
        s.set_precision(1, 1e-2 if case["model"] == "cdsin2d" else 1e-4, 1e-8)
    if i["sdg"] is not None:
        s.set_time(i["time"], i["dtfactor"])
        s.set("sdg", i["sdg"].ravel())
    state = {"step": step, "s": s}
    if not ldg:
        s.set("uh", _trace(s.get("uh"), i["seed"]))
        s.hdgGetQ()
    if step in ("krylov", "gmres") and not ldg:
        s.hdgAssembleLinearSystem()
    if step == "krylov":
        state["v"] = _vector(case, seed, s.sizes["ndofuhat"]).to(DEV)
        state["w"] = torch.empty_like(state["v"])
        state["y"] = torch.empty_like(state["v"])
        torch.cuda.synchronize()
    elif step == "residual":
        state["out"] = [_view(s, k) for k in (("Ru",) if ldg else ("udg", "Ru", "Rh", "b"))]
    elif step == "assemble":
        names = ("Ru", "Rh", "b") + (() if mixed else ("H", "F", "P"))
        state["out"] = [_view(s, k) for k in names] + [_view(s, k, "<f4") for k in (("H32", "F32") if mixed else ())]
    elif step == "gmres":
        if ldg:
            s.evalResidual()
            s.set("b", -s.get("Ru"))
        state["out"] = [_view(s, "x")]
    else:
        pin = lambda a: torch.from_numpy(np.array(a, dtype=np.float64).ravel()).pin_memory()  # noqa: E731
        state["udg"], state["uh"] = pin(s.get("udg")), pin(s.get("uh"))
        state["udg_out"], state["uh_out"] = torch.empty_like(state["udg"]).pin_memory(), torch.empty_like(state["uh"]).pin_memory()
        state["sdg"] = pin(i["sdg"]) if i["sdg"] is not None else None
        state["sdg_dev"] = _view(s, "sdg") if i["sdg"] is not None else None
    return state


def run(state):
    s, step = state["s"], state["step"]
    if step == "krylov":
        s.evalMatVec(state["v"].data_ptr(), state["w"].data_ptr())
        s.ApplyPreconditioner(state["w"].data_ptr(), state["y"].data_ptr())
        return [state["w"], state["y"]]
    if step == "residual":
        s.hdgGetQ()
        return [*state["out"], s.hdgAssembleResidual()]
    if step == "assemble":
        s.hdgAssembleLinearSystem()
        return state["out"]
    if step == "gmres":
        s.GMRES()
        return state["out"]
    if state["sdg"] is not None:
        state["sdg_dev"].copy_(state["sdg"])
    s.solve(*(state[k].numpy() for k in ("udg", "uh", "udg_out", "uh_out")))
    return [state["udg_out"], state["uh_out"]]


# ------------------------------------------------------------------ work and tolerance
def _sizes(case):
    model, n, p = case["model"], case["n"], case["p"]
    nd = 2 if model in ("poisson2d", "cdsin2d", "ns2d") else 3
    ncu = {"ns2d": 4, "euler3d": 5, "euler3d_ldg": 5}.get(model, 1)
    if model == "poisson2d":
        ne, npe, npf, nfe = 2 * n * n, (p + 1) * (p + 2) // 2, p + 1, 3
        nf, nge, ngf = 3 * n * n + 2 * n, {2: 6, 3: 12}[p], p + 1
    else:
        ne, npe, npf, nfe = n**nd, (p + 1) ** nd, (p + 1) ** (nd - 1), 2 * nd
        nf, nge, ngf = nd * n**nd + (0 if model in ("ns2d", "euler3d", "euler3d_ldg") else nd * n ** (nd - 1)), npe, npf
    nq = 0 if ncu == 5 else nd
    return dict(nd=nd, ncu=ncu, ne=ne, npe=npe, npf=npf, nfe=nfe, nf=nf, nge=nge, ngf=ngf, nq=nq, n=npe * ncu,
                m=ncu * npf * nfe, N=ncu * npf * nf, nc=ncu * (1 + nq))


# Krylov steps of a solve at the listed sizes' order, to count the work that cannot be left out
STEPS = {"ns2d": 60, "euler3d_ldg": 120, "cdsin2d": 300, "convdiff3d": 18}


def work(case):
    z = _sizes(case)
    step, ldg, es = case["step"], case["model"] == "euler3d_ldg", 4 if case["form"] == "mixed" else 8
    nd, ne, npe, nge, n, m, N, nc, ncu = (z[k] for k in ("nd", "ne", "npe", "nge", "n", "m", "N", "nc", "ncu"))
    ncf, geom = ncu * z["npf"], 8 * ne * (nge * (nd * nd + nd + 1) + z["nfe"] * z["ngf"] * (2 * nd + 1))
    blocks = z["nf"] * ncf * ncf if case["model"] != "poisson2d" else ne * m * m
    res = {"bytes": geom + 8 * ne * (2 * npe * nc + 2 * n + m) + 16 * N,
           "flops": 2 * ne * (npe * nge * (nc + ncu + (nd + 1) * ncu) + z["nq"] * npe * ncu * (2 * nge * nd + npe))}
    if ldg:
        kry = {"bytes": res["bytes"] - 16 * N, "flops": res["flops"]}
        vec = n * ne
        res = kry
    else:
        kry = {"bytes": es * (m * m * ne + blocks) + 24 * N, "flops": 2 * (m * m * ne + blocks)}
        vec = N
    k = npe * z["nq"] * ncu
    asm = {"bytes": res["bytes"] + es * ((m + n) * m * ne + blocks),
           "flops": res["flops"] + ne * (2 * npe * npe * nge * ncu * nc + 2 * (n + m) ** 2 * k // max(1, ncu) + 2 * n**3
                                         + 2 * n * n * m + 2 * m * m * n) + 2 * blocks * (ncf if blocks != ne * m * m else m)}
    if step == "residual":
        return res
    if step == "krylov":
        return kry
    if step == "assemble":
        return asm
    its = STEPS[case["model"]]
    basis = sum(min(j % 50, 50) for j in range(its))
    gm = {"bytes": its * kry["bytes"] + 16 * vec * basis, "flops": its * kry["flops"] + 4 * vec * basis}
    if step == "gmres":
        return gm
    return {k: gm[k] + asm[k] + res[k] for k in gm}


def tolerance(case):
    """About four times the distance from ``exact`` that the ranges showed, more where a right
    implementation may invert or stop differently."""
    step, mixed, model = case["step"], case["form"] == "mixed", case["model"]
    if step == "krylov":
        return {"rel": 4e-6} if mixed else {"rel": 1e-12}   # seen 8e-7, 4e-15
    if step in ("residual", "assemble"):
        return {"rel": 8e-6} if mixed else {"rel": 2e-12}   # seen 2e-6, 5e-13
    if step == "gmres":
        return {"rel": 5e-6} if model == "euler3d_ldg" else {"rel": 2e-7}   # seen 1.3e-6, 4e-8
    if mixed:
        return {"rel": 4e-8}                                # seen 6e-9
    return {"rel": 1e-10} if model == "cdsin2d" else {"rel": 1e-7}   # seen 1.4e-11; stops at 1e-8


# ------------------------------------------------------------------ the same in 64 bits by plain torch
def _flux(model, params):
    """Pointwise flux [ncu, nd] of the state U = (u, q)."""
    def linear(U):
        nd = U.shape[0] - 1
        c = params[1:1 + nd] if model != "poisson2d" else [0.0] * nd
        return torch.stack([params[0] * U[1 + d] + c[d] * U[0] for d in range(nd)])[None]

    def ns2d(U):
        gam, Re, Pr, M = params
        r, m1, m2, E = U[:4]
        (rx, ux_, vx_, Ex), (ry, uy_, vy_, Ey) = U[4:8], U[8:12]
        u, v = m1 / r, m2 / r
        ke = (u * u + v * v) / 2
        P = (gam - 1) * (E - r * ke)
        ux, vx, uy, vy = (ux_ - rx * u) / r, (vx_ - rx * v) / r, (uy_ - ry * u) / r, (vy_ - ry * v) / r
        Px = (gam - 1) * (Ex - rx * ke - r * (u * ux + v * vx))
        Py = (gam - 1) * (Ey - ry * ke - r * (u * uy + v * vy))
        k = gam / ((gam - 1) * Re * Pr) / (r * r)
        txx, txy, tyy = (2 * ux - vy) * 2 / 3 / Re, (uy + vx) / Re, (2 * vy - ux) * 2 / 3 / Re
        h = (E + P) / r
        fx = [m1, m1 * u + P + txx, m2 * u + txy, m1 * h + u * txx + v * txy + k * (Px * r - P * rx)]
        fy = [m2, m1 * v + txy, m2 * v + P + tyy, m2 * h + u * txy + v * tyy + k * (Py * r - P * ry)]
        return torch.stack([torch.stack(fx), torch.stack(fy)], 1)

    def euler(U):
        r, mom, E = U[0], U[1:4], U[4]
        v = mom / r
        P = (params[0] - 1) * (E - (mom * v).sum() / 2)
        return torch.cat([mom[None], mom[:, None] * v[None] + P * torch.eye(3, dtype=U.dtype, device=U.device),
                          ((E + P) * v)[None]])

    return {"ns2d": ns2d, "euler3d": euler, "euler3d_ldg": euler}.get(model, linear)


def _source(model, params, x):
    """Pointwise source [..., ncu] at the points x [..., nd]."""
    if model == "poisson2d":
        return (2 * math.pi**2 * torch.sin(math.pi * x).prod(-1))[..., None]
    if model == "cdsin2d":
        return (torch.sin(params[3] * math.pi * x[..., 0]) * torch.sin(params[4] * math.pi * x[..., 1]))[..., None]
    if model == "convdiff3d":
        d = x - torch.tensor(params[4:7], dtype=x.dtype, device=x.device)
        return torch.exp(-(d * d).sum(-1) / (2 * params[7] ** 2))[..., None]
    return torch.zeros(*x.shape[:-1], 4 if model == "ns2d" else 5, dtype=x.dtype, device=x.device)


class _Dense:
    """The discretisation on dense element blocks: index order [element, row, column]."""

    def __init__(self, case, i):
        self.model, self.params, self.tau, self.dtf = case["model"], i["params"], i["tau"], i["dtfactor"]
        T = lambda a: torch.from_numpy(np.array(a)).to(DEV)  # noqa: E731
        ma, me, so = (inputs.read_blob(i["blobs"][k].tobytes()) for k in (1, 2, 3))
        nd, npe, npf, nge, ngf = (int(ma[1][k]) for k in (0, 5, 6, 7, 8))
        self.ne, self.nfe = int(me[1][1]), int(me[1][4])
        self.nd, self.npe, self.npf = nd, npe, npf
        phi = T(ma[2].reshape(nge, npe, nd + 1, order="F"))
        self.phi, self.w = phi[:, :, 0], T(ma[3].reshape(npe, nge, nd + 1, order="F"))
        pf = T(ma[4].reshape(ngf, npf, nd, order="F"))
        self.pf, self.wf = pf[:, :, 0], T(ma[5].reshape(npf, ngf, nd, order="F"))[:, :, 0]
        self.perm = T(me[24].reshape(npf, self.nfe, order="F").astype(np.int64)).T          # [l, a]
        self.bf = T(me[25].reshape(self.nfe, self.ne, order="F").astype(np.int64)).T > 0      # [e, l]
        s = HDGSolver("", _library(case["model"]), blobs=i["blobs"])
        f2e, con = s.connectivity()
        s.close()
        self.f2e, self.con = T(f2e.astype(np.int64)), T(con.T.astype(np.int64)).reshape(self.ne, self.nfe, npf)
        self.nf = f2e.shape[1]
        x = T(so[2].reshape(self.ne, nd, npe))
        self.u = T(i["u"])                                                              # [e, k, i]
        self.ncu = self.u.shape[1]
        self.nc = int(inputs.read_blob(i["blobs"][0].tobytes())[1][5])
        self.nq = nd if self.nc > self.ncu else 0
        self.sdg = T(i["sdg"]) if i["sdg"] is not None else None
        J = torch.einsum("gir,eci->egcr", phi[:, :, 1:], x)
        self.jac = torch.linalg.det(J)
        self.Xx = self.jac[..., None, None] * torch.linalg.inv(J)                       # [e, g, r, d]
        self.xg = torch.einsum("gi,eci->egc", self.phi, x)
        xf = x[:, :, self.perm]                                                         # [e, c, l, a]
        t = torch.einsum("gar,ecla->elgcr", pf[:, :, 1:], xf)
        nl = torch.stack([t[..., 1, 0], -t[..., 0, 0]], -1) if nd == 2 else torch.linalg.cross(t[..., 0], t[..., 1])
        self.jf = nl.norm(dim=-1)
        self.nl = nl / self.jf[..., None]                                               # [e, l, g, d]
        # the trace starts from the state of each face's first element
        e1, l1 = self.f2e[0], self.f2e[1]
        uh = self.u[e1][torch.arange(self.nf, device=DEV)[:, None], :, self.perm[l1]]
        self.uh = T(_trace(uh.flatten().cpu().numpy(), i["seed"])).reshape(-1, self.ncu)
        if self.nq:
            Mi = torch.linalg.inv(torch.einsum("ig,gj,eg->eij", self.w[:, :, 0], self.phi, self.jac))
            C = torch.einsum("igr,gj,egrd->edij", self.w[:, :, 1:], self.phi, self.Xx)
            E = torch.zeros(self.ne, nd, npe, self.nfe, npf, dtype=torch.float64, device=DEV)
            mf = torch.einsum("ag,gb,elgd,elg->elabd", self.wf, self.pf, self.nl, self.jf)
            for l in range(self.nfe):
                E[:, :, self.perm[l], l] += mf[:, l].permute(0, 3, 1, 2)
            self.MC, self.ME = Mi[:, None] @ C, Mi[:, None] @ E.flatten(3)

    def getq(self):
        """u and q at the nodes, [e, c, i]."""
        if not self.nq:
            return self.u
        q = (torch.einsum("edij,ekj->edki", self.MC, self.u)
             - torch.einsum("edij,ejk->edki", self.ME, self.uh[self.con].flatten(1, 2)))
        return torch.cat([self.u, q.flatten(1, 2)], 1)

    def _points(self, U, jac):
        """Flux [.., k, d] at the points U [.., c] and, with jac, its derivatives [.., k, d, c]."""
        f, shape = _flux(self.model, self.params), U.shape[:-1]
        U = U.reshape(-1, U.shape[-1])
        out = torch.vmap(f)(U)
        df = torch.vmap(torch.func.jacfwd(f), chunk_size=1 << 17)(U) if jac else None
        return out.reshape(*shape, *out.shape[1:]), df.reshape(*shape, *df.shape[1:]) if jac else None

    def volume(self, U, jac):
        Ug = torch.einsum("gi,eci->egc", self.phi, U)
        f, df = self._points(Ug, jac)
        s = _source(self.model, self.params, self.xg)
        if self.sdg is not None:
            s = s + torch.einsum("gi,eki->egk", self.phi, self.sdg) - self.dtf * Ug[..., :self.ncu]
        rg = torch.cat([(s * self.jac[..., None])[:, :, None], torch.einsum("egkd,egrd->egrk", f, self.Xx)], 2)
        Ru = torch.einsum("igr,egrk->eki", self.w, rg)
        if not jac:
            return Ru, None
        ds = torch.zeros_like(df[..., 0, :])
        for k in range(self.ncu):
            ds[..., k, k] = -self.dtf
        rj = torch.cat([(ds * self.jac[..., None, None])[:, :, None], torch.einsum("egkdc,egrd->egrkc", df, self.Xx)], 2)
        DB = torch.empty(self.ne, self.ncu, self.npe, self.nc, self.npe, dtype=torch.float64, device=DEV)
        for k in range(self.ncu):
            for c in range(self.nc):
                DB[:, k, :, c] = -torch.einsum("igr,egr->eig", self.w, rj[..., k, c]) @ self.phi
        return Ru, DB

    def faces(self, U, jac):
        """Node residuals and blocks of the numerical flux on every element face; the trace equation's."""
        ncu = self.ncu
        Uf = torch.einsum("ga,ecla->elgc", self.pf, U[:, :, self.perm])
        Hf = torch.einsum("ga,elak->elgk", self.pf, self.uh[self.con])
        f, df = self._points(torch.cat([Hf, Uf[..., ncu:]], -1), jac)
        fh = torch.einsum("elgkd,elgd->elgk", f, self.nl) + self.tau * (Uf[..., :ncu] - Hf)
        bou = self.bf[:, :, None, None]
        fb = torch.where(bou, -self.tau * Hf, fh)
        r = [torch.einsum("ag,elgk->elak", self.wf, v * self.jf[..., None]) for v in (fh, fb)]
        if not jac:
            return r, None
        d = torch.einsum("elgkdc,elgd->elgkc", df, self.nl)
        eye = self.tau * torch.eye(ncu, dtype=torch.float64, device=DEV)
        dU, dH = d.clone(), d[..., :ncu] - eye
        dU[..., :ncu] = eye
        bU, bH = torch.where(bou[..., None], 0.0, dU), torch.where(bou[..., None], -eye, dH)
        mats = [torch.einsum("ag,gb,elgkc->elkacb", self.wf, self.pf, v * self.jf[..., None, None]) for v in (dU, dH, bU, bH)]
        return r, mats

    def residual(self, U):
        Ru, _ = self.volume(U, False)
        (rf, rb), _ = self.faces(U, False)
        for l in range(self.nfe):
            Ru[:, :, self.perm[l]] -= rf[:, l].transpose(1, 2)
        return Ru.flatten(1), -rb.flatten(1)                                            # [e, n], [e, (l a k)]

    def scatter(self, we):
        """Element trace vectors [e, (l a k)] summed on the faces."""
        w = torch.zeros(self.nf * self.npf, self.ncu, dtype=torch.float64, device=DEV)
        return w.index_add_(0, self.con.flatten(), we.reshape(-1, self.ncu)).flatten()

    def assemble(self, U):
        ne, ncu, npe, npf, nfe, nc = self.ne, self.ncu, self.npe, self.npf, self.nfe, self.nc
        Ru, Rh = self.residual(U)
        _, DB = self.volume(U, True)
        _, (dU, dH, bU, bH) = self.faces(U, True)
        Z = lambda *s: torch.zeros(*s, dtype=torch.float64, device=DEV)  # noqa: E731
        F, KG, H = Z(ne, ncu, npe, nfe, npf, ncu), Z(ne, nfe, npf, ncu, nc, npe), Z(ne, nfe, npf, ncu, nfe, npf, ncu)
        for l in range(nfe):
            p = self.perm[l]
            for k in range(ncu):
                for c in range(nc):
                    DB[:, k, p[:, None], c, p[None]] += dU[:, l, k, :, c]
                    KG[:, l, :, k, c, p] += bU[:, l, k, :, c]
                for c in range(ncu):
                    F[:, k, p, l, :, c] += dH[:, l, k, :, c]
                    H[:, l, :, k, l, :, c] += bH[:, l, k, :, c]
        n, m = ncu * npe, nfe * npf * ncu
        D, K = DB[:, :, :, :ncu].reshape(ne, n, n), KG[..., :ncu, :].reshape(ne, m, n)
        F, H = F.reshape(ne, n, m), H.reshape(ne, m, m)
        for d in range(self.nq):
            for c in range(ncu):
                j = ncu * (1 + d) + c
                B, G = DB[:, :, :, j].reshape(ne, n, npe), KG[..., j, :].reshape(ne, m, npe)
                D[:, :, c * npe:(c + 1) * npe] += B @ self.MC[:, d]
                F[:, :, c::ncu] -= B @ self.ME[:, d]
                K[:, :, c * npe:(c + 1) * npe] += G @ self.MC[:, d]
                H[:, :, c::ncu] -= G @ self.ME[:, d]
        del DB, KG
        Di = torch.linalg.inv(D)
        F = -(Di @ F)
        H = H + K @ F
        Ru = (Di @ Ru[..., None])[..., 0]
        Rh = Rh - (K @ Ru[..., None])[..., 0]
        self.H, self.F, self.Ru, self.Rh, self.b = H, F, Ru, Rh, self.scatter(Rh)
        return self

    def faceblocks(self):
        """H summed into one block per face [f, (a k), (b c)], and each element's own."""
        npf, ncu, nfe = self.npf, self.ncu, self.nfe
        n1 = npf * ncu
        P = torch.zeros(self.nf, n1, n1, dtype=torch.float64, device=DEV)
        H = self.H.reshape(self.ne, nfe, n1, nfe, n1)
        f, a = self.con // npf, self.con % npf                                          # [e, l, a]
        idx = (a[..., None] * ncu + torch.arange(ncu, device=DEV)).flatten(2)           # [e, l, (a k)]
        for l in range(nfe):
            P.index_put_((f[:, l, 0][:, None, None], idx[:, l][:, :, None], idx[:, l][:, None]), H[:, l, :, l], accumulate=True)
        return P, f[:, :, 0], idx

    def precond(self):
        """The preconditioner's blocks: of faces, or (additive Schwarz) of elements."""
        P, f, idx = self.faceblocks()
        if self.model != "poisson2d":
            return torch.linalg.inv(P)
        n1 = self.npf * self.ncu
        A = self.H.reshape(self.ne, self.nfe, n1, self.nfe, n1).clone()
        for l in range(self.nfe):
            A[:, l, :, l] = P[f[:, l][:, None, None], idx[:, l][:, :, None], idx[:, l][:, None]]
        return torch.linalg.inv(A.reshape(self.H.shape))

    def gather(self, v):
        return v.reshape(-1, self.ncu)[self.con].flatten(1)

    def matvec(self, v):
        return self.scatter((self.H @ self.gather(v)[..., None])[..., 0])

    def pre(self, P, v):
        if self.model != "poisson2d":
            return (P @ v.reshape(self.nf, -1, 1)).flatten()
        return self.scatter((P @ self.gather(v)[..., None])[..., 0])

    def ldg_residual(self, u):
        Ru, _ = self.volume(u, False)
        e1, l1, e2, l2 = self.f2e
        u1 = u[e1][torch.arange(self.nf, device=DEV)[:, None], :, self.perm[l1]]         # [f, a, k]
        nodes = self._second_nodes()
        u2 = u[e2][torch.arange(self.nf, device=DEV)[:, None], :, nodes]
        g1, g2 = (torch.einsum("ga,fak->fgk", self.pf, v) for v in (u1, u2))
        nl, jf = self.nl[e1, l1], self.jf[e1, l1]
        fl = [self._points(g, False)[0] for g in (g1, g2)]
        fh = torch.einsum("fgkd,fgd->fgk", (fl[0] + fl[1]) / 2, nl) + self.tau * (g1 - g2)
        r = torch.einsum("ag,fgk->fak", self.wf, fh * jf[..., None])
        R = Ru.transpose(1, 2).reshape(-1, self.ncu).clone()
        R.index_add_(0, (e1[:, None] * self.npe + self.perm[l1]).flatten(), -r.flatten(0, 1))
        R.index_add_(0, (e2[:, None] * self.npe + nodes).flatten(), r.flatten(0, 1))
        return -R.reshape(self.ne, self.npe, self.ncu).transpose(1, 2) / self.dtf

    def _second_nodes(self):
        """The second element's nodes in the order of the face's nodes, [f, a]."""
        e2, l2 = self.f2e[2], self.f2e[3]
        a = self.con[e2, l2] - self.npf * torch.arange(self.nf, device=DEV)[:, None]    # face node of local node b
        return torch.gather(self.perm[l2], 1, torch.argsort(a, 1))


def _gmres(op, b, restart=100, tol=1e-13, most=6000):
    """Restarted GMRES with twice-applied Gram-Schmidt, to the end of 64 bits."""
    x, done, n0 = torch.zeros_like(b), 0, b.norm()
    while done < most:
        r = b - op(x) if done else b.clone()
        beta = r.norm()
        if beta <= tol * n0:
            break
        V = torch.zeros(restart + 1, b.numel(), dtype=b.dtype, device=b.device)
        H = torch.zeros(restart + 1, restart, dtype=b.dtype, device=b.device)
        V[0] = r / beta
        for j in range(restart):
            w = op(V[j])
            for _ in range(2):
                h = V[:j + 1] @ w
                w = w - h @ V[:j + 1]
                H[:j + 1, j] += h
            H[j + 1, j] = w.norm()
            V[j + 1] = w / H[j + 1, j]
            done += 1
        e = torch.zeros(restart + 1, dtype=b.dtype, device=b.device)
        e[0] = beta
        y = torch.linalg.lstsq(H.cpu(), e.cpu()[:, None]).solution[:, 0].to(b.device)
        step = y @ V[:restart]
        x = x + step
        if step.norm() <= tol * x.norm():
            break
    return x


def exact(case, seed):
    with torch.no_grad():
        return _exact(case, seed)


def _exact(case, seed):
    i = _inputs(case, seed)
    d, step = _Dense(case, i), case["step"]
    if case["model"] == "euler3d_ldg":
        R = d.ldg_residual(d.u)
        if step == "residual":
            return [R.flatten(), float(R.norm())]
        eps = 1e-3  # the products are differences of residuals with this step
        J = lambda v: ((d.ldg_residual(d.u + eps * v.reshape(R.shape)) - R) / eps).flatten()  # noqa: E731
        return [_gmres(J, -R.flatten(), tol=1e-11)]
    U = d.getq()
    if step == "residual":
        Ru, Rh = d.residual(U)
        b = d.scatter(Rh)
        return [U.flatten(), Ru.flatten(), Rh.flatten(), b, float(b.norm() + Ru.norm())]
    d.assemble(U)
    col = lambda A: A.transpose(1, 2).flatten()  # noqa: E731
    if step == "assemble":
        if case["form"] == "mixed":
            return [d.Ru.flatten(), d.Rh.flatten(), d.b, col(d.H), col(d.F)]
        return [d.Ru.flatten(), d.Rh.flatten(), d.b, col(d.H), col(d.F), col(d.precond())]
    P = d.precond()
    if step == "krylov":
        w = d.matvec(_vector(case, seed, d.nf * d.npf * d.ncu).to(DEV))
        return [w, d.pre(P, w)]
    x = _gmres(lambda v: d.pre(P, d.matvec(v)), d.pre(P, d.b))
    if step == "gmres":
        return [x]
    d.u = d.u + (d.Ru + (d.F @ d.gather(x)[..., None])[..., 0]).reshape(d.u.shape)
    d.uh = d.uh + x.reshape(-1, d.ncu)
    return [d.getq().flatten().cpu(), d.uh.flatten().cpu()]
