"""A long one-launch solve leaves room for other streams' kernels.

Two threads repeat Fourier solves of 8,000 triangles (3-4 ms each, one cooperative launch) on streams of their own while
a third sweeps a small plan (two launches and a 4-byte copy, 0.08 ms alone) on four others.  Where a solve holds every SM, a
sweep waits for the ends of several of them: 6 ms.  Where a solve's results wait for it in the copy engine's queue, a
sweep's copy waits behind them: half a solve, 1.5 ms.  Beside solves that do neither it takes 0.08-0.4 ms; 1 ms is
the line between.
"""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_sweeps_run_beside_repeated_fourier_solves(case):
    import ctypes as C
    import torch
    from openbte_gb300 import _lib, objects as O
    from openbte_gb300.fourier import FourierPlan
    from openbte_gb300.geometry import porous_cell_2d
    from openbte_gb300.mesh import mesh_from_cell
    from openbte_gb300.runtime import HostProblem, Plan
    big = mesh_from_cell(porous_cell_2d(8000, 0.20, "square", seed=3))
    bcs_big = O.BoundaryConditions(periodic={"Periodic_x": 1, "Periodic_y": 0}, diffuse="Boundary")
    ek_big = O.EffectiveThermalConductivity(normalization=-1, contact="Periodic_x")
    geo, mat, bcs, ek, _ = case("a600")
    stop, ready, errors = threading.Event(), threading.Barrier(3), []

    def fourier():
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                plan = FourierPlan(big, np.diag([150.0, 120.0]), bcs_big, ek_big, [], 0)
                plan.solve()
                ready.wait()
                while not stop.is_set():
                    plan.solve()
        except Exception as e:                  # reported below
            errors.append(e)
            ready.abort()

    threads = [threading.Thread(target=fourier) for _ in range(2)]
    for t in threads:
        t.start()
    took = []
    try:
        streams = [torch.cuda.Stream() for _ in range(4)]
        for k, stream in enumerate(streams):
            with torch.cuda.stream(stream):
                plan = Plan(HostProblem(geo, mat, bcs, ek))
                u = torch.zeros(plan.nu, dtype=torch.float64, device="cuda")
                out = torch.zeros_like(u)

                def sweep():
                    _lib.check(plan.lib.obte_bte_sweep(plan.handle, _lib.PRECISION["fp32"], C.c_void_p(u.data_ptr()),
                                                       C.c_void_p(out.data_ptr()), 1), "sweep")
                sweep()
                if k == 0:
                    ready.wait()
                for _ in range(40):
                    t0 = time.perf_counter()
                    sweep()
                    took.append(time.perf_counter() - t0)
    finally:
        stop.set()
        for t in threads:
            t.join()
    assert not errors, errors
    assert np.median(took) < 1e-3, f"median {1e3 * np.median(took):.2f} ms beside two Fourier solves"
