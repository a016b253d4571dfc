"""The one-launch Fourier solve against the CPU restatement, where its shape changes.

One multigrid level (the dense inverse alone), two and three; the largest meshes of one cluster (1,536 elements)
and the smallest on all SMs; tetrahedra; the diagonal preconditioner on both; walls held at a temperature (no
pinned element).  Bounds as in the comparison with the reference: CG stops at 1e-13 of its right-hand side and the
corrections contract, so temperatures agree to 1e-9 of the largest and fluxes (one gradient more) to 1e-8.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,jacobi,mixed", [
    (250, 2, 0, 0), (600, 2, 0, 0), (1500, 2, 0, 0), (1600, 2, 0, 0), (4500, 2, 0, 0), (1800, 3, 0, 0),
    (600, 2, 1, 0), (2000, 2, 1, 0), (250, 2, 0, 1), (700, 2, 0, 1), (3000, 2, 0, 1)])
def test_fourier_sizes_match_the_oracle(monkeypatch, n, dim, jacobi, mixed):
    from fourier_oracle import fourier
    from openbte_gb300 import Fourier, objects as O
    from openbte_gb300.geometry import porous_cell_2d, porous_cube_3d
    from openbte_gb300.mesh import mesh_from_cell
    cell = porous_cube_3d(n, 0.10, seed=3) if dim == 3 else porous_cell_2d(n, 0.20, "square", seed=3)
    geo = mesh_from_cell(cell)
    jumps = {"Periodic_x": 1, "Periodic_y": 0}
    if dim == 3:
        jumps["Periodic_z"] = 0
    bcs = O.BoundaryConditions(periodic=jumps, diffuse="Boundary")
    if mixed:
        bcs = O.BoundaryConditions(periodic=jumps,
                                   mixed={"Boundary": {"value": 0.4, "boundary_conductance": 20.0}})
    ek = O.EffectiveThermalConductivity(normalization=-1, contact="Periodic_x")
    kappa = np.diag([150.0, 110.0, 130.0][:dim])
    if jacobi:
        monkeypatch.setenv("OBTE_FOURIER_JACOBI", "1")
    from openbte_gb300 import fourier as module
    module._PLANS.clear()
    f = Fourier(geo, kappa, bcs, effective_thermal_conductivity=ek, verbose=False)
    module._PLANS.clear()
    k, T, J, _ = fourier(geo, kappa, bcs, ek)
    here = f.variables
    np.testing.assert_allclose(here["Temperature_Fourier"]["data"], T, rtol=0, atol=1e-9 * max(1.0, np.abs(T).max()))
    np.testing.assert_allclose(here["Flux_Fourier"]["data"], J * 1e9, rtol=0, atol=1e-8 * np.abs(J * 1e9).max())
    assert abs(f.aux["kappa_eff"] - k) <= 1e-8 * abs(k)
