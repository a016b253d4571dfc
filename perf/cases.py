"""The work that programs have this package do, as cases for measurement.

Four kinds of call, each through an entry point that a program can call:

* ``sweep``    one transport sweep of every ordinate on a prepared plan (``obte_bte_sweep``), the layer that
               every solve repeats: triangles and tetrahedra, FP32 and FP64;
* ``solve``    one kappa_eff solve on a prepared plan (``bte.solve_plan``): the served form (FP32 with
               refinement at 1e-5, each plan solved without the periodic-inflow preconditioner), the resident
               form (the preconditioner built on the first solve) and plain FP64;
* ``rta``      the drop-in calls of a script, ``Fourier`` and then ``BTE_RTA`` from host arrays (FP64,
               the default tolerance);
* ``fourier``  the diffusive first guess alone (``Fourier``);
* ``pixels``   kappa_eff and dkappa/drho of a pixel cell for a new density field: ``PixelSolver`` (MFP-resolved)
               and the gray ``get_solver``.

Sizes are those of the package's benchmark (2k-60k triangles, 48 or 96 directions, 30-100 mean free paths, the
110k-tetrahedron cube's ordinates on a smaller mesh, 128 x 128 pixels) and of its tests.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np


def listed():
    return [
        # one sweep of the smallest served request: few short chains, latency counts
        {"name": "sweep32_2k_30x48", "kind": "sweep", "n": 2000, "nm": 30, "nq": 48, "dim": 2, "prec": "fp32"},
        # one sweep of a mid-sized request with odd ordinate counts
        {"name": "sweep32_11k_77x48", "kind": "sweep", "n": 11003, "nm": 77, "nq": 48, "dim": 2, "prec": "fp32"},
        # one sweep of the resident 2D benchmark cell
        {"name": "sweep32_60k_100x96", "kind": "sweep", "n": 60000, "nm": 100, "nq": 96, "dim": 2, "prec": "fp32"},
        # one sweep of a spherical-pore cube with the 3D benchmark's 30 MFPs x 16 x 32 directions
        {"name": "sweep32_tet24k_30x512", "kind": "sweep", "n": 24000, "nm": 30, "nq": 512, "dim": 3, "prec": "fp32"},
        # the output pass and the plain FP64 solve sweep in FP64
        {"name": "sweep64_20k_100x96", "kind": "sweep", "n": 20000, "nm": 100, "nq": 96, "dim": 2, "prec": "fp64"},
        # a served request: FP32 with refinement at 1e-5, no preconditioner (a plan is solved once)
        {"name": "solve_served_8k_60x48", "kind": "solve", "n": 8000, "nm": 60, "nq": 48, "dim": 2,
         "prec": "fp32_refine", "rtol": 1e-5, "precond": -1},
        # the resident benchmark solve: the same plan solved again and again, preconditioner built once
        {"name": "solve_resident_60k_100x96", "kind": "solve", "n": 60000, "nm": 100, "nq": 96, "dim": 2,
         "prec": "fp32_refine", "rtol": 1e-7, "precond": 1},
        # a script's own calls on the golden-sized cell: Fourier, then BTE_RTA in FP64 at the default tolerance
        {"name": "rta_1k_12x24", "kind": "rta", "n": 1000, "nm": 12, "nq": 24, "dim": 2, "rtol": 1e-4},
        # the first guess alone, at the benchmark size
        {"name": "fourier_60k", "kind": "fourier", "n": 60000, "dim": 2},
        # the reference's gray inverse solver
        {"name": "pixels_gray_24x32", "kind": "pixels", "n": 24, "nm": 1, "nq": 32, "kn": 0.5},
        # a design step of an MFP-resolved cell
        {"name": "pixels_64_20x32", "kind": "pixels", "n": 64, "nm": 20, "nq": 32, "kn": 0.0},
        # the design step of the benchmark
        {"name": "pixels_128_50x64", "kind": "pixels", "n": 128, "nm": 50, "nq": 64, "kn": 0.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sweep", "sweep", "sweep", "solve", "solve", "rta", "fourier", "pixels"])
    if kind == "sweep":
        prec = rng.choice(["fp32", "fp32", "fp64"])
        if rng.random() < 0.3:
            nq = rng.choice([4, 8]) * rng.choice([8, 16, 24])
            return {"kind": "sweep", "n": _log_int(rng, 1500, 24000), "nm": rng.randint(5, 30), "nq": nq, "dim": 3,
                    "prec": prec}
        return {"kind": "sweep", "n": _log_int(rng, 600, 40000), "nm": rng.randint(5, 100),
                "nq": rng.choice([24, 48, 60, 96]), "dim": 2, "prec": prec}
    if kind == "solve":
        prec, rtol = rng.choice([("fp32_refine", 1e-5), ("fp32_refine", 1e-5), ("fp64", 1e-8)])
        return {"kind": "solve", "n": _log_int(rng, 1500, 5000 if prec == "fp64" else 20000), "nm": rng.randint(30, 60),
                "nq": rng.choice([48, 96]), "dim": 2, "prec": prec, "rtol": rtol, "precond": -1}
    if kind == "rta":
        return {"kind": "rta", "n": _log_int(rng, 600, 4000), "nm": rng.randint(5, 40), "nq": rng.choice([24, 36, 48]),
                "dim": 2, "rtol": rng.choice([1e-4, 1e-6])}
    if kind == "fourier":
        if rng.random() < 0.3:
            return {"kind": "fourier", "n": _log_int(rng, 1500, 24000), "dim": 3}
        return {"kind": "fourier", "n": _log_int(rng, 600, 60000), "dim": 2}
    if rng.random() < 0.4:
        return {"kind": "pixels", "n": rng.randint(10, 64), "nm": 1, "nq": 2 * rng.randint(6, 24),
                "kn": rng.choice([0.1, 0.5, 1.0])}
    return {"kind": "pixels", "n": rng.randint(16, 64), "nm": rng.randint(4, 30), "nq": rng.choice([16, 32, 48]),
            "kn": 0.0}


# ---- inputs --------------------------------------------------------------------------------------

def _mesh(case):
    """A case's geometry: a cell with a square or circular pore, or a cube with a spherical one."""
    from openbte_gb300.geometry import porous_cell_2d, porous_cube_3d
    from openbte_gb300.mesh import mesh_from_cell
    n = case["n"]
    if case["dim"] == 3:
        cell = porous_cube_3d(n, 0.10, seed=n % 1000 + 1)
    else:
        cell = porous_cell_2d(n, 0.10 + 0.05 * (n % 6), "circle" if n % 2 else "square", seed=n % 1000 + 1)
    return mesh_from_cell(cell), cell.size


def _material(case, seed):
    """The synthetic lognormal material; its bulk conductivity and median mean free path come from the seed."""
    from openbte_gb300.material import synthetic_isotropic_2d, synthetic_isotropic_3d
    rng = np.random.default_rng([seed, 11])
    bulk, median = float(rng.uniform(100.0, 200.0)), float(rng.uniform(200.0, 400.0))
    if case["dim"] == 3:
        n_theta = 4 if case["nq"] < 128 else 8 if case["nq"] < 512 else 16
        return synthetic_isotropic_3d(case["nm"], n_theta, case["nq"] // n_theta, kappa_bulk=bulk, median=median)
    return synthetic_isotropic_2d(case["nm"], case["nq"], kappa_bulk=bulk, median=median)


def _conductivity(case, seed):
    """A diagonal conductivity (W/mK) for the diffusive solve alone."""
    return np.diag(150.0 * np.random.default_rng([seed, 9]).uniform(0.7, 1.3, case["dim"]))


def _conditions(case, size):
    from openbte_gb300 import objects as O
    jumps = {"Periodic_x": 1, "Periodic_y": 0}
    if case["dim"] == 3:
        jumps["Periodic_z"] = 0
    bcs = O.BoundaryConditions(periodic=jumps, diffuse="Boundary")
    norm = -1.0 / size if case["dim"] == 3 else -1
    return bcs, O.EffectiveThermalConductivity(normalization=norm, contact="Periodic_x")


def _temperatures(geo, rng):
    """A lattice temperature as an iteration meets it: the drop across the cell and a rough part."""
    x = np.array([np.asarray(geo.nodes)[np.asarray(e)].mean(axis=0)[0] for e in geo.elems])
    x = (x - x.min()) / max(x.max() - x.min(), 1e-300)
    return (0.5 - x) * rng.uniform(0.6, 1.0) + 0.05 * rng.standard_normal(len(x))


def _density(n, seed):
    """Seeded smoothed random field on an n x n periodic grid in [0.05, 0.95]."""
    rng = np.random.default_rng([seed, 3])
    z = rng.standard_normal((n, n))
    k = np.fft.fftfreq(n)
    z = np.real(np.fft.ifft2(np.fft.fft2(z) * np.exp(-(k[:, None] ** 2 + k[None, :] ** 2) * (n / 8.0) ** 2)))
    z = (z - z.min()) / (z.max() - z.min())
    return 0.05 + 0.9 * z.reshape(-1)


def _sweep_state(geo, mat, bcs, seed):
    """The state vector a sweep reads: (DeltaT, T_B of every diffuse wall, periodic inflow per source and MFP)."""
    rng = np.random.default_rng([seed, 5])
    f = _Faces(geo, bcs)
    dT = _temperatures(geo, rng)
    nm = len(mat.mfps)
    x = []
    for s in np.asarray(mat.vmfp):
        src = f.sources(s)
        x.append((dT[src][:, None] + 0.02 * rng.standard_normal((len(src), nm))).reshape(-1))
    tb = dT[f.wall_elem] + 0.02 * rng.standard_normal(len(f.wall_elem))
    return np.concatenate([dT, tb] + x)


def prepare(case, seed):
    import torch
    seed = int(seed) % (1 << 31)
    if case["kind"] == "pixels":
        n, rho = case["n"], _density(case["n"], seed)
        if case["nm"] == 1:
            from openbte_gb300.inverse import get_solver
            return {"case": case, "func": get_solver(grid=n, Kn=case["kn"], n_phi=case["nq"]), "rho": rho}
        from openbte_gb300.inverse import IsotropicMaterial, PixelSolver
        solver = PixelSolver(n, IsotropicMaterial.lognormal(case["nm"], case["nq"]), size=100.0)
        # a design loop holds its densities on the device
        return {"case": case, "solver": solver, "rho": torch.tensor(rho, dtype=torch.float64, device="cuda")}
    geo, size = _mesh(case)
    bcs, ek = _conditions(case, size)
    if case["kind"] == "fourier":
        return {"case": case, "geo": geo, "bcs": bcs, "ek": ek, "kappa": _conductivity(case, seed)}
    mat = _material(case, seed)
    if case["kind"] == "rta":
        return {"case": case, "geo": geo, "bcs": bcs, "ek": ek, "mat": mat}
    from openbte_gb300.runtime import HostProblem, Plan
    if case["kind"] == "sweep":
        plan = Plan(HostProblem(geo, mat, bcs, ek))
        u = torch.tensor(_sweep_state(geo, mat, bcs, seed), dtype=torch.float64, device="cuda")
        assert u.numel() == plan.nu
        # the sweep's tables are laid out once, as a solve's set-up does
        plan.prepare("fp64" if case["prec"] == "fp64" else "fp32", 2)
        return {"case": case, "plan": plan, "u": u, "out": torch.zeros_like(u)}
    plan = Plan(HostProblem(geo, mat, bcs, ek))
    plan.prepare(case["prec"])
    # the first guess: the drop along x, rough, as a diffusive solve or an earlier result leaves it
    dT0 = torch.tensor(_temperatures(geo, np.random.default_rng([seed, 5])), dtype=torch.float64, device="cuda")
    return {"case": case, "plan": plan, "dT0": dT0}


# ---- one pass ------------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sweep":
        from openbte_gb300 import _lib
        plan, u, out = state["plan"], state["u"], state["out"]
        _lib.check(plan.lib.obte_bte_sweep(plan.handle, _lib.PRECISION[case["prec"]], C.c_void_p(u.data_ptr()),
                                           C.c_void_p(out.data_ptr()), 1), "obte_bte_sweep")
        return out
    if kind == "solve":
        from openbte_gb300.bte import solve_plan
        info, dT, J, K, S = solve_plan(state["plan"], state["dT0"], precision=case["prec"], rtol=case["rtol"],
                                       precond=case["precond"])
        return {"kappa": float(info.kappa_eff), "T": dT, "J": J, "K": K, "S": S}
    if kind == "rta":
        from openbte_gb300 import BTE_RTA, Fourier
        f = Fourier(state["geo"], state["mat"].thermal_conductivity, state["bcs"],
                    effective_thermal_conductivity=state["ek"], verbose=False)
        # the preconditioner is left off, as for a geometry that is solved once
        r = BTE_RTA(state["geo"], state["mat"], state["bcs"], fourier=f, effective_thermal_conductivity=state["ek"],
                    bte_rtol=case["rtol"], precond=-1)
        return {"kappa": r.kappa_eff, "T": r.variables["Temperature_BTE"]["data"], "J": r.variables["Flux_BTE"]["data"],
                "S": r.aux["suppression"], "TF": f.variables["Temperature_Fourier"]["data"],
                "JF": f.variables["Flux_Fourier"]["data"]}
    if kind == "fourier":
        from openbte_gb300 import Fourier
        f = Fourier(state["geo"], state["kappa"], state["bcs"], effective_thermal_conductivity=state["ek"], verbose=False)
        return {"kappa": float(f.aux["kappa_eff"]), "T": f.variables["Temperature_Fourier"]["data"],
                "J": f.variables["Flux_Fourier"]["data"]}
    if case["nm"] == 1:
        (kappa, _), jac = state["func"](state["rho"])
        return {"kappa": kappa, "jac": jac}
    kappa, grad = state["solver"].kappa_and_gradient(state["rho"])
    return {"kappa": float(kappa), "jac": grad}


# ---- the least that a pass reads, writes and computes -----------------------------------------------

def work(case):
    n, dim = case["n"], case.get("dim", 2)
    if case["kind"] == "fourier":
        # mesh arrays in, T and J out; 10 deferred corrections of one linear solve each (~30 products with the
        # operator), ~10 flops a coefficient
        nf = dim + 1
        return {"bytes": n * (nf * (8 * (3 * dim + 4) + 16) / 2 + 8 + 8 * dim), "flops": 10.0 * 30 * n * (nf + 1) * 4}
    if case["kind"] == "pixels":
        ne, nf, b, sweeps = n * n, 4, 4, (120 if n > 96 else 80)
    else:
        ne, nf = n, dim + 1
        b = 8 if case.get("prec", "fp64") == "fp64" else 4
        sweeps = 1 if case["kind"] == "sweep" else 25 if case.get("precond") == 1 else 45
    nm, nq = case["nm"], case["nq"]
    if case["kind"] == "pixels":
        src = 2 * n
    elif dim == 3:
        src = 3.5 * n ** (2.0 / 3.0)
    else:
        src = 2.0 * math.sqrt(n)
    state = ne + (4 * ne if case["kind"] == "pixels" else 2 * math.sqrt(ne)) + src * nq * nm / 2
    # one sweep: the operator of every direction (order, coefficients) and the state in, the state out
    per_sweep_bytes = nq * ne * (4 + b * (nf / 2.0 + 1)) + 2 * 8 * state
    # per unknown: the upwind products, the source, the quotient and the weighted sum
    per_sweep_flops = float(ne) * nm * nq * (2 * (nf / 2.0) + 8)
    return {"bytes": sweeps * per_sweep_bytes, "flops": sweeps * per_sweep_flops}


# ---- the same answers in 64 bits, from the equations ------------------------------------------------

class _Faces:
    """Directed faces of a mesh: per element up to nf internal faces (neighbour, normal area / volume, whether
    they cross the periodic boundary, the temperature jump across them) and the diffuse walls."""

    def __init__(self, geo, bcs):
        dim = int(geo.dim)
        sem = np.asarray(geo.side_elem_map)
        na = np.asarray(geo.normal_areas)[:, :dim]
        vol = np.asarray(geo.elem_volumes)
        inner = np.asarray(geo.internal)
        self.n, self.dim, self.vol, self.na, self.sem = int(geo.n_elems), dim, vol, na, sem
        cut = np.zeros(len(sem), bool)
        jump = np.zeros(len(sem))
        for region, sides in geo.periodic_sides.items():
            cut[np.asarray(sides, dtype=np.int64)] = True
            jump[np.asarray(sides, dtype=np.int64)] = bcs.periodic[region]
        i, j = sem[inner, 0], sem[inner, 1]
        own = np.concatenate([i, j])
        self.own, self.nb = own, np.concatenate([j, i])
        self.k = np.concatenate([na[inner] / vol[i][:, None], -na[inner] / vol[j][:, None]])
        self.cut = np.concatenate([cut[inner]] * 2)
        # T across the face is T_neighbour + jump for the first element, - jump for the second
        self.jump = np.concatenate([jump[inner], -jump[inner]])
        w = geo.side_physical_regions.get(bcs.diffuse, []) if bcs.diffuse else []
        w = np.asarray(w, dtype=np.int64)
        self.wall_elem = sem[w, 0] if len(w) else np.zeros(0, np.int64)
        self.wall_k = na[w] / vol[self.wall_elem][:, None] if len(w) else np.zeros((0, dim))
        self.wall_area = na[w]
        # per element: its directed faces, padded with -1
        order = np.argsort(own, kind="stable")
        count = np.bincount(own, minlength=self.n)
        start = np.concatenate([[0], np.cumsum(count)[:-1]])
        self.of = np.full((self.n, int(count.max())), -1)
        self.of[own[order], np.arange(len(own)) - start[own[order]]] = order

    def sources(self, s):
        return np.unique(self.nb[((self.k @ np.asarray(s)[: self.dim]) < 0) & self.cut])


def _transport(f, s, lam, b, p, tb, x, src):
    """T[n, m] of one direction: (1 + L D) T + L sum_in g T_up = b + L p - L sum_walls min(g, 0) T_B, with the inflow
    across the periodic boundary given by x[len(src), m]; element by element down the upwind order."""
    n, nm = f.n, len(lam)
    s = np.asarray(s)[: f.dim]
    g = f.k @ s
    gw = f.wall_k @ s
    D = np.zeros(n)
    np.add.at(D, f.own, np.maximum(g, 0))
    np.add.at(D, f.wall_elem, np.maximum(gw, 0))
    rhs = np.array(p)
    np.add.at(rhs, f.wall_elem, -np.minimum(gw, 0) * tb)
    T = np.zeros((n + len(src) + 1, nm))                # elements, periodic sources, a zero row
    T[n:n + len(src)] = x
    ge = np.where(f.of >= 0, g[f.of], 0.0)
    up = np.where(f.of >= 0, f.nb[f.of], 0)
    cut = (f.of >= 0) & f.cut[f.of]
    inflow = ge < 0
    row = np.where(inflow & ~cut, up, n + len(src))
    per = inflow & cut
    if len(src):
        row[per] = n + np.searchsorted(src, up[per])
    coef = np.where(inflow, ge, 0.0)
    left = (inflow & ~cut).sum(axis=1)
    front = np.nonzero(left == 0)[0]
    down = np.where((ge > 0) & ~cut, up, n)
    left = np.concatenate([left, [1 << 30]])
    while len(front):
        acc = np.einsum("ek,ekm->em", coef[front], T[row[front]])
        T[front] = (b[front][:, None] + lam * (rhs[front][:, None] - acc)) / (1.0 + lam * D[front][:, None])
        nxt, cnt = np.unique(down[front], return_counts=True)
        left[nxt] -= cnt
        front = nxt[(left[nxt] == 0) & (nxt < n)]
    return T[:n]


class _Map:
    """The source iteration's map on (DeltaT, T_B, periodic inflow) and its outputs."""

    def __init__(self, geo, mat, bcs, ek):
        self.f = f = _Faces(geo, bcs)
        self.lam = np.asarray(mat.mfps, dtype=np.float64)
        self.dirs = np.asarray(mat.vmfp, dtype=np.float64)
        self.tau = np.asarray(mat.t_coeff)
        self.sig = np.asarray(mat.sigma)
        self.src = [f.sources(s) for s in self.dirs]
        gb = np.einsum("mqj,sj->mqs", self.sig[:, :, : f.dim], f.wall_k)
        out = np.minimum(gb, 0).sum(axis=(0, 1))
        self.emit = np.maximum(gb, 0) / np.where(out != 0, -out, np.inf)
        self.P = np.zeros((len(self.dirs), f.n))
        for q, s in enumerate(self.dirs):
            np.add.at(self.P[q], f.own, -np.minimum(f.k @ s[: f.dim], 0) * f.jump)
        sides = np.asarray(geo.periodic_sides[ek.contact], dtype=np.int64)
        self.e1, self.e2 = f.sem[sides, 0], f.sem[sides, 1]
        self.sn = np.einsum("mqi,ci->mqc", self.sig[:, :, : f.dim], f.na[sides])
        self.areas = np.linalg.norm(f.na[sides], axis=1)
        self.nrm, self.alpha = ek.normalization, bcs.periodic[ek.contact]

    def __call__(self, u, with_src=True, outputs=False):
        f, nm = self.f, len(self.lam)
        n, nd = f.n, len(f.wall_elem)
        dT, tb = u[:n], u[n:n + nd]
        new_T, new_B, xs = np.zeros(n), np.zeros(nd), []
        at = n + nd
        J = np.zeros((n, self.sig.shape[2]))
        K, S = np.zeros(self.tau.shape), np.zeros(self.tau.shape)
        for q, s in enumerate(self.dirs):
            k = len(self.src[q])
            x = u[at:at + k * nm].reshape(k, nm)
            at += k * nm
            T = _transport(f, s, self.lam, dT, self.P[q] if with_src else np.zeros(n), tb, x, self.src[q])
            new_T += T @ self.tau[:, q]
            new_B += np.einsum("sm,ms->s", T[f.wall_elem], self.emit[:, q])
            xs.append(T[self.src[q]].reshape(-1))
            if outputs:
                J += (T - dT[:, None]) @ self.sig[:, q]
                pos, neg = np.maximum(self.sn[:, q], 0), np.minimum(self.sn[:, q], 0)
                K[:, q] = self.nrm * (np.einsum("cm,mc->m", T[self.e1], pos)
                                      + np.einsum("cm,mc->m", T[self.e2] + self.alpha, neg))
                S[:, q] = self.nrm * (self.areas @ T[self.e1])
        v = np.concatenate([new_T, new_B] + xs)
        return (v, J, K, S) if outputs else v

    def level(self):
        """The weights of the quantity that the iteration conserves: volumes and, on the walls, outgoing fluxes."""
        f = self.f
        g = np.abs(np.minimum(f.wall_area @ self.dirs[:, : f.dim].T, 0))
        return f.vol, np.einsum("mq,m,sq->s", self.tau, self.lam, g)

    def fixed_point(self, dT0, tol=1e-12, restart=60):
        f = self.f
        n, nd = f.n, len(f.wall_elem)
        zero = np.zeros(n + nd + sum(len(s) for s in self.src) * len(self.lam))
        rhs = self(zero)
        x = zero.copy()
        for _ in range(4):
            r = rhs - x + self(x, False)
            beta = np.linalg.norm(r)
            if beta <= tol * max(np.linalg.norm(x), np.linalg.norm(rhs)):
                break
            V, H = [r / beta], np.zeros((restart + 1, restart))
            for j in range(restart):
                w = V[j] - self(V[j], False)
                for _ in range(2):
                    for i in range(j + 1):
                        h = V[i] @ w
                        H[i, j] += h
                        w = w - h * V[i]
                H[j + 1, j] = np.linalg.norm(w)
                V.append(w / H[j + 1, j])
                e = np.zeros(j + 2)
                e[0] = beta
                y, *_ = np.linalg.lstsq(H[:j + 2, :j + 1], e, rcond=None)
                if np.linalg.norm(e - H[:j + 2, :j + 1] @ y) <= 0.5 * tol * np.linalg.norm(rhs):
                    break
            x = x + sum(a * v for a, v in zip(y, V))
        u, J, K, S = self(x, outputs=True)
        lt, lb = self.level()
        c = (lt @ dT0 + lb @ dT0[f.wall_elem] - lt @ u[:n] - lb @ u[n:n + nd]) / (lt.sum() + lb.sum())
        return u[:n] + c, J, K, S + c * self.nrm * self.areas.sum()


def _fourier(geo, bcs, ek, kappa, max_iter=40, rtol=1e-8):
    """Two-point diffusion with the non-orthogonal part corrected from least-squares gradients (a sparse solve per
    correction); element 10 carries no coupling, temperatures centred between their extremes."""
    import scipy.sparse as sp
    import scipy.sparse.linalg as sla
    dim, n = int(geo.dim), int(geo.n_elems)
    kappa = np.asarray(kappa)[:dim, :dim]
    na, d = np.asarray(geo.normal_areas)[:, :dim], np.asarray(geo.dists)[:, :dim]
    orth = np.einsum("ki,ij,kj->k", na, kappa, na) / np.einsum("ki,ki->k", na, d)
    non = na @ kappa.T - d * orth[:, None]
    sem, inner, vol = np.asarray(geo.side_elem_map), np.asarray(geo.internal), np.asarray(geo.elem_volumes)
    i, j = sem[inner, 0], sem[inner, 1]
    vo = orth[inner]
    F = sp.csr_matrix((np.concatenate([vo / vol[i], -vo / vol[i], vo / vol[j], -vo / vol[j]]),
                       (np.concatenate([i, i, j, j]), np.concatenate([i, j, j, i]))), shape=(n, n)).tolil()
    F[10, :] = 0
    F[10, 10] = 1
    lu = sla.splu(F.tocsc())
    jump = np.zeros(len(sem))
    B = np.zeros(n)
    for region, sides in geo.periodic_sides.items():
        sides = np.asarray(sides, dtype=np.int64)
        jump[sides] = bcs.periodic[region]
        np.add.at(B, sem[sides, 0], jump[sides] * orth[sides] / vol[sem[sides, 0]])
        np.add.at(B, sem[sides, 1], -jump[sides] * orth[sides] / vol[sem[sides, 1]])
    B[10] = 0
    esm = np.array([geo.elem_side_map[e] for e in range(n)])
    own = sem[esm, 0] == np.arange(n)[:, None]
    other = np.where(own, sem[esm, 1], sem[esm, 0])
    is_inner = np.zeros(len(sem), bool)
    is_inner[inner] = True
    live = is_inner[esm]
    sign = np.where(own, 1.0, -1.0)
    gw = np.asarray(geo.gradient_weights)
    w, vn = np.asarray(geo.interp_weights)[inner][:, None], non[inner]
    Cc, old, err, it = np.zeros(n), 0.0, 1.0, 0
    while err > rtol and it < max_iter:
        it += 1
        T = lu.solve(B + Cc)
        T = T - 0.5 * (T.max() + T.min())
        diff = np.where(live, T[other] - T[:, None] + sign * jump[esm], 0.0)
        grad = np.einsum("kjs,ks->kj", gw, diff)
        flux = np.einsum("ki,ki->k", w * grad[i] + (1 - w) * grad[j], vn)
        Cc = np.zeros(n)
        np.add.at(Cc, i, flux / vol[i])
        np.add.at(Cc, j, -flux / vol[j])
        size = np.linalg.norm(Cc)
        err = 0.0 if size == 0 else abs(size - old) / size
        old = size
    sides = np.asarray(geo.periodic_sides[ek.contact], dtype=np.int64)
    k = ek.normalization * np.sum((T[sem[sides, 0]] - T[sem[sides, 1]] - bcs.periodic[ek.contact]) * orth[sides])
    return float(k), T, -grad @ kappa.T * 1e9


def _gray_pixels(n, kn, nq, rho):
    """kappa and dkappa/drho of the gray pixel model: upwind transport on an n x n periodic grid where a side
    transmits t = 2 r r' / (r + r') and re-emits the rest, one sparse solve for X and one for the adjoint."""
    import scipy.sparse as sp
    import scipy.sparse.linalg as sla
    h, ne = 1.0 / n, n * n
    r = 1e-12 + rho * (1.0 - 1e-12)
    phi = 2 * np.pi * np.arange(nq) / nq
    s = np.stack([np.cos(phi), np.sin(phi)], axis=1)
    ii, jj = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    p = (ii * n + jj).reshape(-1)
    e1 = np.concatenate([p, p])
    e2 = np.concatenate([(((ii + 1) % n) * n + jj).reshape(-1), (ii * n + (jj + 1) % n).reshape(-1)])
    nv = np.concatenate([np.tile([h, 0.0], (ne, 1)), np.tile([0.0, -h], (ne, 1))])
    contact = np.concatenate([(ii == n - 1).reshape(-1), np.zeros(ne, bool)])
    t = 2 * r[e1] * r[e2] / (r[e1] + r[e2])
    own, nb, av = np.concatenate([e1, e2]), np.concatenate([e2, e1]), np.concatenate([nv, -nv])
    side = np.concatenate([np.arange(2 * ne)] * 2)
    jump = np.concatenate([contact * 1.0, contact * -1.0])
    g = av @ s.T / h ** 2                                  # [faces, q]
    sig = 2.0 / (nq * kn) * s
    sn = av @ sig.T
    emit = np.maximum(sn, 0) / (-np.minimum(sn, 0).sum(axis=1))[:, None]
    D = np.zeros((ne, nq))
    np.add.at(D, own, np.maximum(g, 0))
    F, Q = np.nonzero(g < 0)
    c = own[F]
    at = c * nq + Q
    lg = kn * g[F, Q]
    rows, cols, vals = [np.arange(ne * nq)], [np.arange(ne * nq)], [(1 + kn * D).reshape(-1)]
    rows.append(at), cols.append(nb[F] * nq + Q), vals.append(lg * t[side[F]])
    for q2 in range(nq):                                   # re-emission and the lattice temperature
        rows.append(at), cols.append(c * nq + q2), vals.append(lg * (1 - t[side[F]]) * emit[F, q2])
        rows.append(np.arange(ne * nq)), cols.append(np.arange(ne * nq) // nq * nq + q2)
        vals.append(np.full(ne * nq, -1.0 / nq))
    A = sp.csr_matrix((np.concatenate(vals), (np.concatenate(rows), np.concatenate(cols))), shape=(ne * nq, ne * nq))
    b = np.zeros(ne * nq)
    np.add.at(b, at, -lg * t[side[F]] * jump[F])
    one = np.ones((ne * nq, 1))                            # constants are in the null space
    lu = sla.splu(sp.bmat([[A, sp.csr_matrix(one)], [sp.csr_matrix(one.T), None]]).tocsc())
    X = lu.solve(np.concatenate([b, [0.0]]))[:-1].reshape(ne, nq)
    cs = np.nonzero(contact)[0]
    sc = nv[cs] @ sig.T
    part = np.maximum(sc, 0) * X[e1[cs]] + np.minimum(sc, 0) * (X[e2[cs]] + 1.0)
    kappa = -np.sum(part * t[cs][:, None])
    dk = np.zeros((ne, nq))
    np.add.at(dk, e1[cs], -np.maximum(sc, 0) * t[cs][:, None])
    np.add.at(dk, e2[cs], -np.minimum(sc, 0) * t[cs][:, None])
    lam = lu.solve(np.concatenate([dk.reshape(-1), [0.0]]), trans="T")[:-1].reshape(ne, nq)
    R = np.einsum("fq,fq->f", emit, X[own])
    dt = np.zeros(2 * ne)
    np.add.at(dt, side[F], -lam[c, Q] * lg * (X[nb[F], Q] + jump[F] - R[F]))
    dt[cs] -= part.sum(axis=1)
    grad = np.zeros(ne)
    np.add.at(grad, e1, dt * 0.5 * (t / r[e1]) ** 2)
    np.add.at(grad, e2, dt * 0.5 * (t / r[e2]) ** 2)
    return np.array([kappa]), grad[None, :]


def exact(case, seed):
    seed = int(seed) % (1 << 31)
    if case["kind"] == "pixels":
        if case["nm"] > 1 or case["n"] ** 2 * case["nq"] > 24 * 24 * 32:
            return None
        kappa, jac = _gray_pixels(case["n"], case["kn"], case["nq"], _density(case["n"], seed))
        return {"kappa": kappa, "jac": jac}
    if case["kind"] == "sweep" and case["n"] * case["nm"] * case["nq"] > 600_000_000:
        return None
    if case["kind"] == "solve" or (case["kind"] == "rta" and case["n"] * case["nq"] > 25_000):
        return None
    geo, size = _mesh(case)
    bcs, ek = _conditions(case, size)
    if case["kind"] == "fourier":
        if case["dim"] == 3 and case["n"] > 12000:
            return None
        k, T, J = _fourier(geo, bcs, ek, _conductivity(case, seed))
        return {"kappa": k, "T": T, "J": J}
    mat = _material(case, seed)
    if case["kind"] == "sweep":
        return _Map(geo, mat, bcs, ek)(_sweep_state(geo, mat, bcs, seed))
    _, TF, JF = _fourier(geo, bcs, ek, mat.thermal_conductivity)
    T, J, K, S = _Map(geo, mat, bcs, ek).fixed_point(TF)
    return {"kappa": float(K.sum()), "T": T, "J": J * 1e9, "S": S, "TF": TF, "JF": JF}
