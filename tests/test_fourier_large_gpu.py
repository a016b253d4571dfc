"""The Fourier solve where its blocks become wider (more than 512 rows to an SM: 77,824 elements on 152 SMs).

Meshes on both sides of the line against the CPU restatement, with the bounds of the smaller ones (CG stops at 1e-13 of
its right-hand side: temperatures to 1e-9 of the largest, fluxes to 1e-8); a barrier of the wide form that runs out.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(n):
    from openbte_gb300 import objects as O
    from openbte_gb300.geometry import porous_cell_2d
    from openbte_gb300.mesh import mesh_from_cell
    geo = mesh_from_cell(porous_cell_2d(n, 0.20, "square", seed=3))
    bcs = O.BoundaryConditions(periodic={"Periodic_x": 1, "Periodic_y": 0}, diffuse="Boundary")
    return geo, bcs, O.EffectiveThermalConductivity(normalization=-1, contact="Periodic_x")


@pytest.mark.parametrize("n,wide", [(76000, False), (80000, True)])
def test_wide_blocks_match_the_oracle(n, wide):
    import torch
    from fourier_oracle import fourier
    from openbte_gb300 import _lib
    from openbte_gb300.fourier import FourierPlan
    geo, bcs, ek = _problem(n)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert (geo.n_elems > 512 * sms) == wide
    kappa = np.diag([150.0, 110.0])
    plan = FourierPlan(geo, kappa, bcs, ek, [], 0)
    info, T, J = plan.solve()
    k, T0, J0, _ = fourier(geo, kappa, bcs, ek)
    np.testing.assert_allclose(T.cpu().numpy(), T0, rtol=0, atol=1e-9 * max(1.0, np.abs(T0).max()))
    np.testing.assert_allclose(J.cpu().numpy(), J0, rtol=0, atol=1e-8 * np.abs(J0).max())
    assert abs(info.kappa - k) <= 1e-8 * abs(k)
    hook = plan.lib.obte_fourier_plan_test_barrier_timeout
    _lib.check(hook(plan.handle, 3, 2048), "hook")
    with pytest.raises(_lib.OBTEError) as e:
        plan.solve()
    assert e.value.status == _lib.OBTE_ERR_DEVICE_TIMEOUT
    _lib.check(hook(plan.handle, -1, 0), "hook")
    np.testing.assert_array_equal(plan.solve()[1].cpu().numpy(), T.cpu().numpy())
