"""Solves whose Arnoldi steps reach the edges of their launch shapes, against the reference's golden outputs.

A step runs as one launch: clusters of 2, 4 and 8 blocks for small states, a grid above; tiles of 16 basis vectors
(restart 4 stays in the first, 40 reaches the third); one share of the state per block or several blocks per share.
The meshes' states have different remainders of 4 entries.  The FP64 basis runs in fp64, the FP32 one in
fp32_refine; dsa=1 adds the one-launch diffusion correction (cells not a multiple of its 32-element segments).
Every form converges to the same fixed point: at a residual of 1e-11 the golden comparison's 1e-6 holds.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["gray600", "a600", "circ1k", "cube1k5"])
@pytest.mark.parametrize("precision,restart,dsa", [("fp64", 4, 0), ("fp64", 40, 0), ("fp32_refine", 4, 0),
                                                   ("fp32_refine", 40, 0), ("fp64", 40, 1), ("fp32_refine", 20, 1)])
def test_arnoldi_launch_shapes_converge_to_the_reference(case, name, precision, restart, dsa):
    from openbte_gb300 import BTE_RTA
    geo, mat, bcs, ek, d = case(name)
    r = BTE_RTA(geo, mat, bcs, effective_thermal_conductivity=ek, bte_rtol=1e-11, precision=precision, restart=restart,
                dsa=dsa, precond=-1, max_sweeps=4000, refine_steps=8)
    assert r.aux["converged"]
    assert abs(r.kappa_eff - d["bte_kappa"]) / abs(d["bte_kappa"]) < 1e-6
    T = r.variables["Temperature_BTE"]["data"]
    shift = T.mean() - d["bte_T"].mean()            # the level follows the first guess
    np.testing.assert_allclose(T - shift, d["bte_T"], rtol=0, atol=1e-6 * np.abs(d["bte_T"]).max())
