"""Every launch shape of the sweep against the exact per-ordinate solves.

A plan's threads per CTA, unit size, staged units and MFPs per CTA follow from its shape; the switches that
force them reach the edges on small meshes: units smaller than a level (32 elements), units of several passes
(256 elements on 32 threads), two and eight staged units (as many as the pipeline holds, more than some
directions' units at the ends), both MFP groupings with a ragged last chunk.  Tolerances are those of the
other sweep tests: 1e-11 (FP64) and 2e-5 (FP32) of the largest exact value.
"""
import ctypes as C

import numpy as np
import pytest

from test_bte_gpu import _state_from_exact

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-11, "fp32": 2e-5}


@pytest.fixture(scope="module")
def exact():
    """Exact solves per case, once for all shapes."""
    done = {}

    def get(case, name):
        if name not in done:
            geo, mat, bcs, ek, _ = case(name)
            rng = np.random.default_rng(11)
            dT = 0.3 * rng.standard_normal(geo.n_elems)
            TB = 0.3 * rng.standard_normal(len(geo.side_physical_regions["Boundary"]))
            done[name] = (geo, mat, bcs, ek, dT, TB, _state_from_exact(geo, mat, bcs, dT, TB))
        return done[name]
    return get


@pytest.mark.parametrize("name", ["a600", "cube1k5"])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("threads,unit,nbuf,wide", [(32, 32, 2, 0), (32, 256, 3, 1), (96, 64, 8, 0), (128, 128, 2, 1),
                                                    (64, 1024, 4, 1)])
def test_sweep_shapes_equal_exact_ordinate_solves(case, exact, monkeypatch, name, precision, threads, unit, nbuf, wide):
    import torch
    from openbte_gb300 import _lib
    from openbte_gb300.runtime import HostProblem, Plan
    geo, mat, bcs, ek, dT, TB, (refT, refB, x) = exact(case, name)
    monkeypatch.setenv("OBTE_SWEEP_THREADS", str(threads))
    monkeypatch.setenv("OBTE_SWEEP_UNIT", str(unit))
    monkeypatch.setenv("OBTE_SWEEP_NBUF", str(nbuf))
    monkeypatch.setenv("OBTE_SWEEP_KV", str((8 if wide else 4) // (1 if precision == "fp32" else 2)))
    plan = Plan(HostProblem(geo, mat, bcs, ek))
    u = torch.tensor(np.concatenate([dT, TB, x]), dtype=torch.float64, device="cuda")
    out = torch.full_like(u, float("nan"))
    _lib.check(plan.lib.obte_bte_sweep(plan.handle, _lib.PRECISION[precision], C.c_void_p(u.data_ptr()),
                                       C.c_void_p(out.data_ptr()), 1), "sweep")
    o = out.cpu().numpy()
    atol = TOL[precision] * max(np.abs(refT).max(), 1.0)
    n = geo.n_elems
    np.testing.assert_allclose(o[:n], refT, rtol=0, atol=atol)
    np.testing.assert_allclose(o[n:n + len(TB)], refB, rtol=0, atol=atol)
    np.testing.assert_allclose(o[n + len(TB):], x, rtol=0, atol=atol)
