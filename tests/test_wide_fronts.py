"""Plans whose front of live rows nearly fills shared memory: accepted, and swept right.

A strip 3 cells wide and `ny` cells high, in two triangles a cell: a direction along x holds two rows of every cell of a
column at once, 2 ny live rows (16 bytes each; 32 with twice the mean free paths to a CTA).  7,600 rows fit as
16-byte rows alone; 13,200 with units of 128 elements do not (their stages and output blocks take 26 KB), with units
of 32 they do.
"""
import ctypes as C

import numpy as np
import pytest


def strip(ny, n_mfp, n_phi=8):
    """(geometry, material, boundary conditions, contact) of the strip."""
    from openbte_gb300 import objects as O
    from openbte_gb300.geometry import PeriodicCell2D
    from openbte_gb300.material import synthetic_isotropic_2d
    from openbte_gb300.mesh import mesh_from_cell
    nx = 3
    x, y = np.arange(nx + 1) - nx / 2, np.arange(ny + 1) - ny / 2
    nodes = np.stack(np.meshgrid(x, y, indexing="ij"), -1).reshape(-1, 2)
    i, j = (a.reshape(-1) for a in np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij"))

    def at(i, j):
        return i * (ny + 1) + j
    elems = np.stack([np.stack([at(i, j), at(i + 1, j), at(i + 1, j + 1)], 1),
                      np.stack([at(i, j), at(i + 1, j + 1), at(i, j + 1)], 1)], 1).reshape(-1, 3)
    v, h = np.arange(ny), np.arange(nx)
    segments = {"Boundary": np.zeros((0, 2), np.int64),
                "Periodic_x_a": np.stack([at(0, v), at(0, v + 1)], 1), "Periodic_x_b": np.stack([at(nx, v), at(nx, v + 1)], 1),
                "Periodic_y_a": np.stack([at(h, 0), at(h + 1, 0)], 1), "Periodic_y_b": np.stack([at(h, ny), at(h + 1, ny)], 1)}
    v, h = np.arange(ny + 1), np.arange(nx + 1)
    periodic = {"x": np.stack([at(0, v), at(nx, v)], 1), "y": np.stack([at(h, 0), at(h, ny)], 1)}
    geo = mesh_from_cell(PeriodicCell2D(nodes, elems, segments, periodic, float(nx), 0.0, "none", 0))
    return (geo, synthetic_isotropic_2d(n_mfp, n_phi), O.BoundaryConditions(periodic={"Periodic_x": 1, "Periodic_y": 0}),
            O.EffectiveThermalConductivity(normalization=-1.0, contact="Periodic_x"))


@pytest.mark.parametrize("ny,n_mfp", [(3800, 304), (6600, 304), (6600, 30)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_tables_of_a_wide_front_can_be_laid_out(ny, n_mfp, precision):
    from openbte_gb300 import _lib
    from openbte_gb300.runtime import HostProblem, Plan
    geo, mat, bcs, ek = strip(ny, n_mfp)
    plan = Plan(HostProblem(geo, mat, bcs, ek), host_only=True)
    assert max(plan.schedule(q)[2] for q in range(8)) == 2 * ny
    digest = C.c_uint64()
    _lib.check(plan.lib.obte_bte_tables_digest(plan.handle, _lib.PRECISION[precision], C.byref(digest)), "tables")


def test_a_front_beyond_shared_memory_is_refused():
    from openbte_gb300 import _lib
    from openbte_gb300.runtime import HostProblem, Plan
    geo, mat, bcs, ek = strip(8000, 4)             # 16,000 rows of 16 bytes
    plan = Plan(HostProblem(geo, mat, bcs, ek), host_only=True)
    digest = C.c_uint64()
    for precision in ("fp32", "fp64"):
        with pytest.raises(_lib.OBTEError) as e:
            _lib.check(plan.lib.obte_bte_tables_digest(plan.handle, _lib.PRECISION[precision], C.byref(digest)), "tables")
        assert e.value.status == _lib.OBTE_ERR_UNSUPPORTED
        assert "shared memory" in str(e.value)


@pytest.mark.gpu
@pytest.mark.parametrize("ny,n_mfp", [(3800, 304), (6600, 5)])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("fp32", 2e-5)])
def test_wide_fronts_equal_exact_ordinate_solves(ny, n_mfp, precision, tol):
    """The temperatures of an output pass against sparse solves of single ordinates, the lattice temperature of a plain
    sweep against their weighted sum; tolerances of the other sweep tests."""
    import torch
    import bte_oracle
    import sweep_order
    from openbte_gb300 import _lib
    from openbte_gb300.runtime import HostProblem, Plan
    geo, mat, bcs, ek = strip(ny, n_mfp)
    plan = Plan(HostProblem(geo, mat, bcs, ek))
    rng = np.random.default_rng(6)
    n = geo.n_elems
    dT = 0.3 * rng.standard_normal(n)
    ops = bte_oracle.setup_operators(geo, mat, bcs)
    solver = bte_oracle.OrdinateSolver(geo, np.asarray(mat.mfps, dtype=np.float64), ops)
    row, nb, k, cut = sweep_order.directed_faces(geo)
    ordinates = [(0, 0), (2, 1), (2, n_mfp - 1), (6, n_mfp // 2)]     # 2 and 6 run along x
    exact, x = {}, []
    for q in range(8):
        src = np.unique(nb[((k @ np.asarray(mat.vmfp[q])[:2]) < 0) & cut])
        own = 0.1 * rng.standard_normal((len(src), n_mfp))
        for (qq, m) in ordinates:
            if qq == q:                       # the inflow that the ordinate's own solution implies
                exact[q, m] = solver.solve(q, m, dT + mat.mfps[m] * ops["perturbation"][q])
                own[:, m] = exact[q, m][src]
        x.append(own.reshape(-1))
    u = torch.tensor(np.concatenate([dT] + x), dtype=torch.float64, device="cuda")
    assert u.numel() == plan.nu
    code = _lib.PRECISION[precision]
    T = torch.zeros((8, n, n_mfp), dtype=torch.float32 if precision == "fp32" else torch.float64, device="cuda")
    out = torch.zeros_like(u)
    _lib.check(plan.lib.obte_bte_sweep_fields(plan.handle, code, C.c_void_p(u.data_ptr()), C.c_void_p(out.data_ptr()), 1,
                                              C.c_void_p(T.data_ptr())), "fields")
    scale = max(1.0, max(np.abs(v).max() for v in exact.values()))
    for (q, m), want in exact.items():
        np.testing.assert_allclose(T[q, :, m].cpu().numpy(), want, rtol=0, atol=tol * scale)
    _lib.check(plan.lib.obte_bte_sweep(plan.handle, code, C.c_void_p(u.data_ptr()), C.c_void_p(out.data_ptr()), 1), "sweep")
    total = torch.einsum("qnm,mq->n", T.double(), torch.tensor(np.asarray(mat.t_coeff), device="cuda"))
    np.testing.assert_allclose(out[:n].cpu().numpy(), total.cpu().numpy(), rtol=0, atol=tol * scale)
