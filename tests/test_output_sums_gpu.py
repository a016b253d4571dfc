"""kappa and suppression sums of an output pass: the same bits in every pass, in the order they always had.

An FP32 output pass adds kcoef T and scoef T of a direction's contact elements in FP32, so their order is part of
the result: by units of 128 elements of a level (fewer where more than 48 cut inflow faces or 64 elements with
outputs would come together), in a unit the groups of 32 elements with fewer contact elements first, elements of a
group in order; K and S are the means of the sums with the later and with the earlier of equal groups first.  The sums
are restated here in numpy from the stored
temperatures of the same pass; one FP32 rounding in another place is 6e-8 of a sum, so 1e-12 holds the order.
Repeated passes and other threads, stages and (larger) units give the same bits; units below 128 elements
cut the groups, and agree to FP32 rounding only: n terms of one sign, n 6e-8 at most, 1e-5 for a few hundred.

A solve that may not sweep again (max_sweeps=1) makes its output pass at the state that its first guess implies.
"""
import ctypes as C

import numpy as np
import pytest

import sweep_order

pytestmark = pytest.mark.gpu


def _cell(dim):
    from openbte_gb300 import objects as O
    from openbte_gb300.geometry import porous_cell_2d, porous_cube_3d
    from openbte_gb300.material import synthetic_isotropic_2d, synthetic_isotropic_3d
    from openbte_gb300.mesh import mesh_from_cell
    if dim == 2:
        cell = porous_cell_2d(12000, 0.20, "circle", seed=4)
        mat = synthetic_isotropic_2d(13, 24)
    else:
        cell = porous_cube_3d(4000, 0.10, seed=4)
        mat = synthetic_isotropic_3d(7, 4, 8)
    geo = mesh_from_cell(cell)
    jumps = {"Periodic_x": 1, "Periodic_y": 0}
    if dim == 3:
        jumps["Periodic_z"] = 0
    bcs = O.BoundaryConditions(periodic=jumps, diffuse="Boundary")
    ek = O.EffectiveThermalConductivity(normalization=-1.0, contact="Periodic_x")
    return geo, mat, bcs, ek


def _units(lp, order, n_cut, special):
    """First positions of a direction's base units (and the end), for every pair of caps."""
    def split(cap_pf, cap_sx):
        first, over = [], [0, 0]
        for a, b in zip(lp[:-1], lp[1:]):
            cnt = pf = sx = 0
            for pos in range(a, b):
                e = order[pos]
                if cnt == 0 or cnt == 128 or pf + n_cut[e] > cap_pf or sx + special[e] > cap_sx:
                    if cnt:
                        over[0] += pf > 48
                        over[1] += sx > 64
                    first.append(pos)
                    cnt = pf = sx = 0
                cnt += 1
                pf += n_cut[e]
                sx += special[e]
            over[0] += pf > 48
            over[1] += sx > 64
        return first, over
    return split


def _sums(geo, mat, bcs, ek, plan, T):
    """K and S [n_mfp, n_dir] from FP32 sums as the pass adds them, the constant of K and the shifts of both per offset."""
    row, nb, k, cut = sweep_order.directed_faces(geo)
    dirs = np.asarray(mat.vmfp)
    walls = np.asarray(geo.side_physical_regions["Boundary"])
    we = np.asarray(geo.side_elem_map)[walls, 0]
    sides = np.asarray(geo.periodic_sides[ek.contact])
    e1, e2 = np.asarray(geo.side_elem_map)[sides].T
    na = np.asarray(geo.normal_areas)[sides]
    area = np.linalg.norm(na, axis=1)
    n, n_dir, n_mfp = geo.n_elems, len(dirs), len(mat.mfps)
    sigma = np.asarray(mat.sigma)
    data = []
    for q in range(n_dir):
        d = dirs[q][: geo.dim]
        g = k @ d
        inflow = (g < 0) & cut
        special = np.zeros(n, bool)
        special[nb[inflow]] = True
        special[we[np.asarray(geo.normal_areas)[walls][:, : geo.dim] @ d > 0]] = True
        special[e1] = special[e2] = True
        order, lp, _ = plan.schedule(q)
        data.append((order, lp, _units(lp, order, np.bincount(row[inflow], minlength=n), special)))
    none = 1 << 30
    free = [u(none, none) for _, _, u in data]
    total = sum(len(f) for f, _ in free)
    pf = 48 if 100 * sum(o[0] for _, o in free) <= total else none
    sx = 64 if 100 * sum(o[1] for _, o in free) <= total else none
    K, S = np.zeros((2, n_mfp, n_dir), np.float32), np.zeros((2, n_mfp, n_dir), np.float32)
    const, kshift, sshift = np.zeros((n_mfp, n_dir)), np.zeros((n_mfp, n_dir)), np.zeros(n_dir)
    for q, (order, lp, u) in enumerate(data):
        first = np.array(u(pf, sx)[0])
        sn = np.zeros((n_mfp, len(sides)))
        for a in range(geo.dim):
            sn = sn + sigma[:, q, a][:, None] * na[:, a][None, :]
        kc, sc = np.zeros((n, n_mfp)), np.zeros(n)
        for c in range(len(sides)):
            kc[e1[c]] += np.maximum(sn[:, c], 0)
            kc[e2[c]] += np.minimum(sn[:, c], 0)
            sc[e1[c]] += area[c]
            const[:, q] += np.minimum(sn[:, c], 0)
        contact = np.zeros(n, bool)
        contact[e1] = contact[e2] = True
        pos = np.nonzero(contact[order])[0]
        unit = np.searchsorted(first, pos, side="right") - 1
        group = (pos - first[unit]) // 32
        tag = unit * 8 + group
        count = np.bincount(tag, minlength=tag.max() + 1)[tag]
        for o, ties in enumerate((-group, group)):
            for p in pos[np.lexsort((pos, ties, count, unit))]:
                e = order[p]
                K[o, :, q] = K[o, :, q] + (kc[e] * ek.normalization).astype(np.float32) * T[q, e]
                S[o, :, q] = S[o, :, q] + np.float32(sc[e] * ek.normalization) * T[q, e]
        kshift[:, q] = (kc * ek.normalization).sum(axis=0)
        sshift[q] = sc.sum() * ek.normalization
    K, S = K.astype(np.float64).mean(axis=0), S.astype(np.float64).mean(axis=0)
    return K, S, const * ek.normalization * bcs.periodic[ek.contact], kshift, sshift


def _pass(plan, dT0, precision):
    from openbte_gb300.bte import solve_plan
    info, _, J, K, S = solve_plan(plan, dT0, precision=precision, rtol=1e-5, max_sweeps=1, precond=-1)
    return info, J.cpu().numpy(), K.cpu().numpy(), S.cpu().numpy()


def _state(geo, mat, dT):
    row, nb, k, cut = sweep_order.directed_faces(geo)
    walls = np.asarray(geo.side_elem_map)[np.asarray(geo.side_physical_regions["Boundary"]), 0]
    x = []
    for d in np.asarray(mat.vmfp):
        src = np.unique(nb[((k @ d[: geo.dim]) < 0) & cut])
        x.append(np.repeat(dT[src], len(mat.mfps)))
    return np.concatenate([dT, dT[walls]] + x)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_contact_sums_keep_their_order_in_every_shape(monkeypatch, dim, precision):
    import torch
    from openbte_gb300 import _lib
    from openbte_gb300.runtime import HostProblem, Plan
    geo, mat, bcs, ek = _cell(dim)
    rng = np.random.default_rng(2)
    dT = 0.5 * rng.standard_normal(geo.n_elems)
    dT0 = torch.tensor(dT, dtype=torch.float64, device="cuda")
    u = torch.tensor(_state(geo, mat, dT), dtype=torch.float64, device="cuda")
    first = None
    for threads, unit, nbuf in [(0, 0, 0), (0, 0, 0), (32, 128, 3), (128, 128, 2), (96, 256, 2), (128, 512, 2), (64, 32, 4)]:
        for name, v in (("THREADS", threads), ("UNIT", unit), ("NBUF", nbuf)):
            if v:
                monkeypatch.setenv("OBTE_SWEEP_" + name, str(v))
        plan = Plan(HostProblem(geo, mat, bcs, ek))
        info, J, K, S = _pass(plan, dT0, precision)
        again = _pass(plan, dT0, precision)
        big = np.abs(K).max()
        # the offset c that both carry is a sum of FP64 atomics: equal to rounding
        np.testing.assert_allclose(again[2], K, rtol=0, atol=1e-13 * big)
        np.testing.assert_allclose(again[3], S, rtol=0, atol=1e-13 * np.abs(S).max())
        if first is None:
            first = (K, S, J)
            T = torch.zeros((len(mat.vmfp), geo.n_elems, len(mat.mfps)),
                            dtype=torch.float32 if precision == "fp32" else torch.float64, device="cuda")
            out = torch.zeros_like(u)
            _lib.check(plan.lib.obte_bte_sweep_fields(plan.handle, _lib.PRECISION[precision], C.c_void_p(u.data_ptr()),
                                                      C.c_void_p(out.data_ptr()), 1, C.c_void_p(T.data_ptr())), "fields")
            k, s, const, kshift, sshift = _sums(geo, mat, bcs, ek, plan, T.cpu().numpy())
            c = info.offset
            tol = 1e-12 if precision == "fp32" else 1e-5      # the restatement adds in FP32
            np.testing.assert_allclose(K, k + const + c * kshift, rtol=0, atol=tol * big)
            np.testing.assert_allclose(S, s + c * sshift, rtol=0, atol=tol * np.abs(S).max())
            continue
        tol = 1e-12 if unit != 32 or precision == "fp64" else 1e-5
        np.testing.assert_allclose(K, first[0], rtol=0, atol=tol * big)
        np.testing.assert_allclose(S, first[1], rtol=0, atol=tol * np.abs(S).max())
        np.testing.assert_allclose(J, first[2], rtol=0, atol=1e-12 * np.abs(J).max())
