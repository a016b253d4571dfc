"""The barriers inside the one-launch Fourier solve and diffusion correction give up with a status.

A barrier over the blocks of a cooperative launch polls a counter, at most a given number of times.  Here block 0 does
not arrive at one barrier and the waits are short: every block gives up and leaves, the call returns
OBTE_ERR_DEVICE_TIMEOUT (a solve after the step in which it happened), and the same plan then gives what it gave
before.  Nothing faults or hangs.  2,000 elements and more: smaller problems use a cluster's hardware barrier.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2000, 20000])          # a quarter of the SMs, all of them
@pytest.mark.parametrize("barrier", [0, 1, 25])
def test_fourier_barrier_that_runs_out_returns_timeout(n, barrier):
    from openbte_gb300 import _lib, objects as O
    from openbte_gb300.fourier import FourierPlan
    from openbte_gb300.geometry import porous_cell_2d
    from openbte_gb300.mesh import mesh_from_cell
    geo = mesh_from_cell(porous_cell_2d(n, 0.20, "square", seed=3))
    bcs = O.BoundaryConditions(periodic={"Periodic_x": 1, "Periodic_y": 0}, diffuse="Boundary")
    ek = O.EffectiveThermalConductivity(normalization=-1, contact="Periodic_x")
    plan = FourierPlan(geo, np.diag([150.0, 110.0]), bcs, ek, [], 0)
    info, T, _ = plan.solve()
    before = T.cpu().numpy()
    hook = plan.lib.obte_fourier_plan_test_barrier_timeout
    _lib.check(hook(plan.handle, barrier, 2048), "hook")
    with pytest.raises(_lib.OBTEError) as e:
        plan.solve()
    assert e.value.status == _lib.OBTE_ERR_DEVICE_TIMEOUT and "timed out" in str(e.value)
    _lib.check(hook(plan.handle, -1, 0), "hook")
    again, T, _ = plan.solve()
    assert again.n_cg == info.n_cg
    np.testing.assert_array_equal(T.cpu().numpy(), before)          # sums in a fixed order
    assert hook(plan.handle, -2, 0) == hook(plan.handle, 0, -1) == _lib.OBTE_ERR_BAD_ARG


@pytest.mark.parametrize("barrier", [0, 2])
@pytest.mark.parametrize("precision", ["fp64", "fp32_refine"])
def test_correction_barrier_that_runs_out_ends_the_solve(case, barrier, precision):
    import time
    import torch
    from openbte_gb300 import _lib
    from openbte_gb300.bte import solve_plan
    from openbte_gb300.runtime import HostProblem, Plan
    geo, mat, bcs, ek, _ = case("c0_2k")
    assert geo.n_elems > 1536
    plan = Plan(HostProblem(geo, mat, bcs, ek))
    dT0 = torch.zeros(plan.n, dtype=torch.float64, device="cuda")

    def solve():
        return solve_plan(plan, dT0, precision=precision, rtol=1e-8, precond=-1, dsa=1)
    info, before, *_ = solve()
    assert info.converged
    hook = plan.lib.obte_bte_plan_test_barrier_timeout
    for _ in range(2):                                   # both of the alternating counters
        _lib.check(hook(plan.handle, barrier, 2048), "hook")
        launches = plan.lib.obte_launch_count()
        t0 = time.perf_counter()
        with pytest.raises(_lib.OBTEError) as e:
            solve()
        assert e.value.status == _lib.OBTE_ERR_DEVICE_TIMEOUT and "timed out" in str(e.value)
        # the first step's correction gave up and the step ended the solve: two sweeps, not up to max_sweeps
        assert plan.lib.obte_launch_count() - launches < 30
        assert time.perf_counter() - t0 < 2.0
        _lib.check(hook(plan.handle, -1, 0), "hook")
        again, T, *_ = solve()
        assert again.converged and again.n_sweeps == info.n_sweeps
        np.testing.assert_allclose(T.cpu().numpy(), before.cpu().numpy(), rtol=0, atol=1e-7 * float(before.abs().max()))
    assert hook(plan.handle, -2, 0) == hook(plan.handle, 0, -1) == _lib.OBTE_ERR_BAD_ARG
