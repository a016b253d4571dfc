"""A right-hand side that is not a number gives temperatures, fluxes and a kappa that are not numbers either.

A residual of NaN compares like no number: it must neither pass for a converged one nor keep the iterations going to
their limit.  One multigrid level, a cluster, the grid; the diagonal preconditioner; walls at a temperature.
"""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,jacobi,mixed", [(250, 0, 0), (600, 0, 0), (2000, 0, 0), (2000, 1, 0), (700, 0, 1), (3000, 0, 1)])
def test_nan_in_the_heat_source_reaches_the_outputs(monkeypatch, n, jacobi, mixed):
    from openbte_gb300 import Fourier, objects as O
    from openbte_gb300 import fourier as module
    from openbte_gb300.geometry import porous_cell_2d
    from openbte_gb300.mesh import mesh_from_cell
    geo = mesh_from_cell(porous_cell_2d(n, 0.20, "square", seed=3))
    jumps = {"Periodic_x": 1, "Periodic_y": 0}
    bcs = O.BoundaryConditions(periodic=jumps, diffuse="Boundary")
    if mixed:
        bcs = O.BoundaryConditions(periodic=jumps, mixed={"Boundary": {"value": 0.4, "boundary_conductance": 20.0}})
    ek = O.EffectiveThermalConductivity(normalization=-1, contact="Periodic_x")
    heat = np.zeros(geo.n_elems)
    heat[geo.n_elems // 2] = np.nan
    if jacobi:
        monkeypatch.setenv("OBTE_FOURIER_JACOBI", "1")
    module._PLANS.clear()
    t0 = time.perf_counter()
    f = Fourier(geo, np.diag([150.0, 110.0]), bcs, effective_thermal_conductivity=ek, heat_source=heat, verbose=False)
    took = time.perf_counter() - t0
    module._PLANS.clear()
    T = f.variables["Temperature_Fourier"]["data"]
    assert np.isnan(T).sum() >= geo.n_elems - 1         # all but the pinned element
    assert np.isnan(f.variables["Flux_Fourier"]["data"]).any()
    assert np.isnan(f.aux["kappa_eff"])
    assert took < 5.0
