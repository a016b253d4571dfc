"""Solves take the sweeps that GMRES with an orthogonal basis takes.

A converged solution alone does not show a wrong Arnoldi step: restarts and the output pass recompute the true residual,
so a lost tile of products or a skipped second pass mostly costs sweeps.  Here the same restarted GMRES runs in
numpy, with Gram-Schmidt done twice in 64 bits and the library's sweep as its operator, and counts its sweeps: one for
the first residual, one a step, one a restart, one for the output pass.  Both stop at the same tolerance; rounding may
move the step at which the estimate passes it by one a cycle.

Up to 8 blocks a step is one cluster launch (gray600, a600), above five launches; 4 and 17 steps a cycle end in the first and
the second tile of 16 basis vectors, 40 in the third.  The diffusion correction is checked with two V-cycles an
application, and on 8 x 8 pixels, where its hierarchy is one dense operator.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gmres_sweeps(apply, f, x, restart, rtol):
    """Sweeps of restarted GMRES on x - K x = f from x until the estimate meets rtol max(|x|, |r|)."""
    count = 1
    r = f - x + apply(x)
    while True:
        beta = np.linalg.norm(r)
        tol = rtol * max(np.linalg.norm(x), beta)
        if beta <= tol:
            return count, x
        V, H = [r / beta], np.zeros((restart + 1, restart))
        for j in range(restart):
            w = V[j] - apply(V[j])
            count += 1
            B = np.array(V)
            for _ in range(2):
                h = B @ w
                H[:j + 1, j] += h
                w = w - h @ B
            H[j + 1, j] = np.linalg.norm(w)
            V.append(w / H[j + 1, j])
            e = np.zeros(j + 2)
            e[0] = beta
            y, *_ = np.linalg.lstsq(H[:j + 2, :j + 1], e, rcond=None)
            est = np.linalg.norm(e - H[:j + 2, :j + 1] @ y)
            if est <= tol:
                break
        x = x + y @ np.array(V[:-1])
        if est <= tol:
            return count, x
        r = f - x + apply(x)
        count += 1


@pytest.mark.parametrize("name", ["gray600", "a600", "circ1k", "c0_2k", "cube1k5"])
@pytest.mark.parametrize("precision,rtol", [("fp64", 1e-9), ("fp32", 1e-5)])
@pytest.mark.parametrize("restart", [4, 17, 40])
def test_solves_take_the_sweeps_of_an_orthogonal_basis(case, name, precision, rtol, restart):
    import torch
    import sweep_order
    from openbte_gb300 import _lib
    from openbte_gb300.bte import solve_plan
    from openbte_gb300.runtime import HostProblem, Plan
    geo, mat, bcs, ek, _ = case(name)
    plan = Plan(HostProblem(geo, mat, bcs, ek))
    out = torch.zeros(plan.nu, dtype=torch.float64, device="cuda")

    def apply(v, source=0):
        u = torch.tensor(v, dtype=torch.float64, device="cuda")
        _lib.check(plan.lib.obte_bte_sweep(plan.handle, _lib.PRECISION[precision], C.c_void_p(u.data_ptr()),
                                           C.c_void_p(out.data_ptr()), source), "sweep")
        return out.cpu().numpy().copy()

    dT = 0.3 * np.random.default_rng(3).standard_normal(geo.n_elems)
    row, nb, k, cut = sweep_order.directed_faces(geo)
    walls = np.asarray(geo.side_elem_map)[np.asarray(geo.side_physical_regions["Boundary"]), 0]
    x = [np.repeat(dT[np.unique(nb[((k @ d[: geo.dim]) < 0) & cut])], len(mat.mfps)) for d in np.asarray(mat.vmfp)]
    u0 = np.concatenate([dT, dT[walls]] + x)
    f = apply(np.zeros(plan.nu), 1)
    want, _ = _gmres_sweeps(apply, f, u0, restart, rtol)
    info, *_ = solve_plan(plan, torch.tensor(dT, device="cuda"), precision=precision, rtol=rtol, max_sweeps=2000,
                          restart=restart, precond=-1, dsa=-1)
    cycles = 1 + want // (restart + 1)
    assert abs(info.n_sweeps - (want + 1)) <= cycles, (info.n_sweeps, want + 1)


@pytest.mark.parametrize("n,cycles", [(8, 1), (8, 2), (24, 2), (48, 2)])
@pytest.mark.parametrize("precision", ["fp64", "fp32_refine"])
def test_correction_with_more_cycles_and_one_level(monkeypatch, n, cycles, precision):
    from openbte_gb300.inverse import IsotropicMaterial, PixelSolver
    from test_dsa_gpu import _density
    mat = IsotropicMaterial.lognormal(8, 16)
    rho = 0.05 + 0.9 * _density(n, 3)
    res = {}
    for dsa in (-1, 1):
        monkeypatch.setenv("OBTE_DSA_CYCLES", str(cycles))
        solver = PixelSolver(n, mat, size=100.0, precision=precision, rtol=1e-10, dsa=dsa)
        k, _ = solver.kappa_and_gradient(rho)
        res[dsa] = k, solver.last_info.n_sweeps
    (k0, s0), (k1, s1) = res[-1], res[1]
    assert abs(k1 - k0) <= (1e-8 if precision == "fp64" else 5e-8) * abs(k0)      # as with one cycle
    assert s1 <= s0
