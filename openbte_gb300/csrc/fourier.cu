// Fourier first guess on the device (openbte/fourier.py:15-185).
//
// The reference assembles the orthogonal part of the finite-volume diffusion
// operator (fourier.py:51-63), factorises it with SuperLU and runs a
// deferred non-orthogonal correction (fourier.py:149-178):
//   T = F^-1 (B + C);  T -= (max T + min T)/2;  grad = LS gradient(T);
//   C = div(w grad_i + (1-w) grad_j) . v_nonorth;  stop when |‖C‖-‖C_old‖|/‖C‖ <= rtol.
// Here F = V^-1 L with L the symmetric volume-weighted Laplacian (plus Robin
// terms of mixed walls), so each T is a conjugate-gradient solve of
// L T = V (B + C) on the device.  Without mixed walls the reference replaces
// row N = 10 by the identity (fourier.py:115-118), i.e. T_N = (B + C)_N; that
// value is moved to the right-hand side and CG runs on the remaining SPD
// system.  The least-squares gradient (openbte/objects.py:322-405), the
// correction gather and the diffusive kappa (openbte/objects.py:139-172) are
// device code too: the whole solve after assembly is one launch.
#include <cuda_runtime.h>

#include <cstdlib>

#include <algorithm>
#include <cmath>
#include <map>
#include <vector>

#include "grid.cuh"

namespace obte {
namespace {

constexpr int FT = 256;

// the root of a sum of squares; NaN stays NaN (fmax would turn it into a converged residual of zero)
__device__ __forceinline__ double root(double s) { return sqrt(s < 0 ? 0.0 : s); }

// Blocks of a solve: as many as its rows fill, 104 to a block: the barrier is cheaper with fewer blocks, and the other SMs
// are left to other streams (8,000 triangles: 77 blocks 3.55 ms, 152 3.7, 39 3.95); at least a quarter of the SMs
// (2,000 triangles: 20 blocks 3.9 ms, 38 3.45).  Above two rows to a thread of every SM's block, half an SM to a block
// instead of a third: 100,000 tetrahedra 58 and 68 ms, 200,000 triangles 11.1 and 13.4 ms, while below the gain is less
// than the room is worth (60,000 triangles 6.8 and 7.3 ms, but beside them 101 and 129 solves of 8,000 x 60 x 48 a second).
PhaseShape fourier_shape(int64_t n, int num_sms) {
  PhaseShape s = phase_shape(n, num_sms);
  if (s.cluster) return s;
  s.blocks = (int)std::min<int64_t>(num_sms, std::max<int64_t>(num_sms / 4, (n + 103) / 104));
  if (n > 2 * (int64_t)GridBarrier::kThreads * num_sms) s.threads = WideGridBarrier::kThreads;
  return s;
}

// Everything of the solve after assembly, for the one launch that runs it.
struct FourierParams {
  int64_t n;
  CsrDev A;                                  // L
  int has_amg;
  AmgDev amg;
  const double *dinv, *vol, *B, *colpin;
  int pin, nv, dim;
  const int32_t* g_nb;                       // gradient stencils
  const double* g_off;
  const unsigned char* g_mixed;
  const double* gw;
  const int32_t *s_i, *s_j;                  // internal sides
  const double *s_w, *s_vnon;
  const int32_t *c_ptr, *c_side;
  double *T, *C, *r[2], *z, *p[2], *Ap, *grad, *part;
  int max_iter, cg_max, check;
  int smem;                                  // bytes of shared memory for the matrices
  double rtol, cg_rtol;
  double* out;                               // deferred corrections, CG iterations
  BarrierParams bar;
};

// The deferred-correction loop (fourier.py:145-178) with its preconditioned CG solves, one launch.  Phases end at
// a barrier over the blocks; scalars are sums of per-block partials that every block adds up itself, in a
// fixed order.  A CG iteration takes one barrier for the product with the direction, one for the residual and
// its restriction (both formed in the gather), and those of the V-cycle; the directions and residuals
// alternate between two buffers so that neighbours read the values of the phase before.
//
// The solve was bound by its launches (60k triangles: 10 corrections, 184 CG iterations, 2,180 launches of 4.6 us
// with their gaps, 11.7 ms; 600 triangles 6.9 ms).  Its matrices stay in shared memory as far as a third of an SM
// has room (60k triangles: 69 of 85 KB an SM), so what is left of a phase is the barrier, one gather through L2 and
// a chain of FP64 operations at 64-76 cycles each: 7.3 and 2.7 ms.
template <typename Bar>
__global__ void __launch_bounds__(Bar::kThreads, Bar::kBlocks) fourier_kernel(const __grid_constant__ FourierParams P) {
  extern __shared__ __align__(16) char smem[];
  __shared__ double red[Bar::kThreads];
  __shared__ Rows sA;
  __shared__ AmgRows sM;
  Bar bar(P.bar);
  const int tid = threadIdx.x, nthr = blockDim.x, nb = gridDim.x;
  Arena ar{smem, P.smem};
  load_rows(P.A, &sA, ar);
  if (P.has_amg) load_amg(P.amg, &sM, ar);
  int r0, r1;
  block_range(P.n, r0, r1);
  // partials: one row of nb per sum
  double *p_pap = P.part, *p_rr = P.part + nb, *p_rz = P.part + 2 * nb, *p_bb = P.part + 3 * nb, *p_mx = P.part + 4 * nb,
         *p_mn = P.part + 5 * nb, *p_cc = P.part + 6 * nb;
  auto put_slot = [&](double v, int slot, int count, double* row) {
    const double s = block_sum(v, slot, count, red);
    if (tid == 0) row[blockIdx.x] = s;
  };
  const int own = min(r1 - r0, nthr);
  auto put = [&](double v, double* row) { put_slot(v, tid < own ? tid : -1, own, row); };      // rows by thread
  auto put_rows = [&](double v, int vec, double* row) {                                      // of block_rows
    put_slot(v, tid % vec == 0 ? tid / vec : -1, min(r1 - r0, nthr / vec), row);
  };
  for (int i = r0 + tid; i < r1; i += nthr) {
    P.T[i] = 0.0;
    P.C[i] = 0.0;
  }
  if (!bar.wait()) return;
  double norm_old = 0, tol = 0, rz = 0;      // thread 0's
  int it = 0, ncg = 0, rb = 0, pb = 0;       // rb, pb: current buffers of r and p
  bool more = P.max_iter > 0;
  while (more) {
    ++it;
    // right-hand side V (B + C), the pinned value moved over; the previous T was re-centred: shifted back onto
    // the pinned value the warm start differs from the new solution only by the change of C
    const double tn = P.pin >= 0 ? P.B[P.pin] + P.C[P.pin] : 0.0;
    const double delta = P.pin >= 0 ? tn - P.T[P.pin] : 0.0;
    {
      double rr = 0, bb = 0;
      double* r = P.r[rb];
      block_rows(sA, [&](int c) { return P.T[c] + delta; }, [&](int i, double Ti) {
        double v = P.vol[i] * (P.B[i] + P.C[i]);
        if (P.pin >= 0) v = i == P.pin ? 0.0 : v - P.colpin[i] * tn;
        const double ri = v - Ti;
        r[i] = ri;
        rr += ri * ri;
        bb += v * v;
      });
      put_rows(rr, sA.vec, p_rr);
      put_rows(bb, sA.vec, p_bb);
    }
    if (!bar.wait()) return;
    if (P.pin >= 0)
      for (int i = r0 + tid; i < r1; i += nthr) P.T[i] += delta;
    grid_sum(p_bb, nb, red, [&](double s) { return tol = P.cg_rtol * fmax(root(s), 1e-300); });
    auto open = [&](double s) { return root(s) <= tol ? 0.0 : 1.0; };
    bool run = grid_sum(p_rr, nb, red, open) != 0;
    // z = M^-1 r and the partials of r . z, after the restriction (or nothing) of the phase before
    auto precondition = [&](const double* r) -> bool {
      double dot = 0;
      auto up = [&](int row, double v) {
        P.z[row] = v;
        dot += r[row] * v;
      };
      int vec = 1;
      if (!P.has_amg) {
        for (int i = r0 + tid; i < r1; i += nthr) up(i, r[i] * P.dinv[i]);
      } else if (P.amg.nl == 1) {
        block_dense(sM, P.amg.nc, r, up);
        vec = 32;
      } else if (!amg_cycle(P.amg, sM, bar, [&](int c) { return r[c]; }, up)) {
        return false;
      } else {
        vec = sM.Q[0].vec;
      }
      put_rows(dot, vec, p_rz);
      return bar.wait();
    };
    auto restrict0 = [&](auto value) {         // b_1 = Q_0^T r
      if (P.has_amg && P.amg.nl > 1) {
        double* b1 = P.amg.b[1];
        block_rows(sM.Qt[0], value, [&](int row, double v) { b1[row] = v; });
      }
    };
    if (run) {
      const double* r = P.r[rb];
      restrict0([&](int c) { return r[c]; });
      if (!bar.wait()) return;
      if (!precondition(r)) return;
      grid_sum(p_rz, nb, red, [&](double s) { return rz = s; });
    }
    double beta = 0;
    bool fresh = true;                         // first direction: p = z
    for (int k = 0; run; ++k) {
      // p = z + beta p, Ap, partials of p . Ap
      {
        const double* po = P.p[pb];
        double* pn = P.p[pb ^ 1];
        double pap = 0;
        auto dir = [&](int c) { return fresh ? P.z[c] : P.z[c] + beta * po[c]; };
        block_rows(sA, dir, [&](int i, double s) {
          const double pi = dir(i);
          pn[i] = pi;
          P.Ap[i] = s;
          pap += s * pi;
        });
        pb ^= 1;
        fresh = false;
        put_rows(pap, sA.vec, p_pap);
      }
      if (!bar.wait()) return;
      const double a = grid_sum(p_pap, nb, red, [&](double pap) { return pap != 0 ? rz / pap : 0.0; });
      {
        const double *ro = P.r[rb], *p = P.p[pb];
        double* rn = P.r[rb ^ 1];
        double s = 0;
        for (int i = r0 + tid; i < r1; i += nthr) {
          P.T[i] += a * p[i];
          const double ri = ro[i] - a * P.Ap[i];
          rn[i] = ri;
          s += ri * ri;
        }
        restrict0([&](int c) { return ro[c] - a * P.Ap[c]; });
        rb ^= 1;
        if ((k + 1) % P.check == 0) put(s, p_rr);        // the residual is tested every `check` iterations
      }
      if (!bar.wait()) return;
      if (!precondition(P.r[rb])) return;
      beta = grid_sum(p_rz, nb, red, [&](double s) {
        const double b = rz != 0 ? s / rz : 0.0;
        rz = s;
        return b;
      });
      if ((k + 1) % P.check == 0) {
        ncg += P.check;
        // (a residual that is not a number has reached T and stays one)
        run = grid_sum(p_rr, nb, red, [&](double s) { return s == s ? open(s) : 0.0; }) != 0 && k + 1 < P.cg_max;
      }
    }
    // T_pin, then T -= (max + min) / 2 (fourier.py:155-156)
    double shift = 0;
    if (P.pin >= 0) {
      double mx = -INFINITY, mn = INFINITY;
      for (int i = r0 + tid; i < r1; i += nthr) {
        if (i == P.pin) P.T[i] = tn;
        mx = fmax(mx, P.T[i]);
        mn = fmin(mn, P.T[i]);
      }
      mx = block_max(mx, red);
      mn = -block_max(-mn, red);
      if (tid == 0) {
        p_mx[blockIdx.x] = mx;
        p_mn[blockIdx.x] = mn;
      }
      if (!bar.wait()) return;
      mx = -INFINITY;
      mn = INFINITY;
      if (tid < nb) {                        // more threads than blocks
        mx = p_mx[tid];
        mn = p_mn[tid];
      }
      mx = block_max(mx, red);
      mn = -block_max(-mn, red);
      __syncthreads();
      if (tid == 0) red[0] = (mx + mn) * 0.5;
      __syncthreads();
      shift = red[0];
    } else if (!bar.wait()) {
      return;
    }
    // least-squares gradient of the shifted T: grad[c] = sum_k gw[c][:, k] diff[c][k],
    //   diff = T[nb] - T[c] + off (nb >= 0), off (nb < 0, no mixed), value - T[c] (mixed)
    const int nv = P.nv, dim = P.dim;
    for (int64_t c = r0 + tid; c < r1; c += nthr) {
      const double tc = P.T[c] - shift;
      double g[3] = {0, 0, 0};
      for (int k = 0; k < nv; ++k) {
        const int j = P.g_nb[c * nv + k];
        double d;
        if (P.g_mixed[c * nv + k]) d = P.g_off[c * nv + k] - tc;
        else d = (j >= 0 ? (P.T[j] - shift) - tc : 0.0) + P.g_off[c * nv + k];
#pragma unroll
        for (int a = 0; a < 3; ++a)
          if (a < dim) g[a] += P.gw[(c * dim + a) * nv + k] * d;
      }
#pragma unroll
      for (int a = 0; a < 3; ++a)
        if (a < dim) P.grad[c * dim + a] = g[a];
    }
    if (!bar.wait()) return;
    // C[c] = sum over its internal sides of +-(w grad_i + (1 - w) grad_j) . v_nonorth / V_c; partial |C|^2
    double cc = 0;
    for (int64_t c = r0 + tid; c < r1; c += nthr) {
      if (P.pin >= 0) P.T[c] -= shift;
      double v = 0;
      for (int k = P.c_ptr[c]; k < P.c_ptr[c + 1]; ++k) {
        const int e = P.c_side[k], sd = e >= 0 ? e : -e - 1;
        const int64_t i = P.s_i[sd], j = P.s_j[sd];
        const double w = P.s_w[sd];
        double f = 0;
        for (int a = 0; a < dim; ++a)
          f += (w * P.grad[i * dim + a] + (1.0 - w) * P.grad[j * dim + a]) * P.s_vnon[(int64_t)sd * dim + a];
        v += e >= 0 ? f : -f;
      }
      v /= P.vol[c];
      P.C[c] = v;
      cc += v * v;
    }
    put(cc, p_cc);
    if (!bar.wait()) return;
    more = grid_sum(p_cc, nb, red, [&](double s) {
             const double norm = root(s);
             const double err = norm == 0 ? 0 : fabs(norm - norm_old) / norm;   // fourier.py:168-171
             norm_old = norm;
             return err > P.rtol && it < P.max_iter ? 1.0 : 0.0;
           }) != 0;
  }
  if (blockIdx.x == 0 && tid == 0) {
    P.out[0] = (double)it;
    P.out[1] = (double)ncg;
  }
}

// After the solve: diffusive kappa terms per contact side (objects.py:152-170), the solve's counts and error word, all
// into page-locked host memory, and J = -kappa . grad.  (Copied from the device they waited in the copy engine's queue
// for the solve, and other streams' copies behind them: a sweep beside two streams of Fourier solves, 0.08 ms alone, took
// half a solve.)
struct OutputParams {
  int64_t n, nc;
  int dim;
  const int32_t *e1, *e2;
  const double *coef, *T, *kap, *grad, *sc;
  double t2const;
  double *J, *words, *terms;
};
__global__ void __launch_bounds__(FT) fourier_outputs_kernel(const __grid_constant__ OutputParams P) {
  const int64_t t0 = (int64_t)blockIdx.x * FT + threadIdx.x, stride = (int64_t)gridDim.x * FT;
  if (t0 < 4) P.words[t0] = P.sc[t0];
  for (int64_t k = t0; k < P.nc; k += stride) {
    const double t2 = P.e2[k] >= 0 ? P.T[P.e2[k]] + P.t2const : P.t2const;
    P.terms[k] = (P.T[P.e1[k]] - t2) * P.coef[k];
  }
  if (P.J)
    for (int64_t c = t0; c < P.n; c += stride)
      for (int a = 0; a < P.dim; ++a) {
        double s = 0;
        for (int b = 0; b < P.dim; ++b) s += P.kap[a * P.dim + b] * P.grad[c * P.dim + b];
        P.J[c * P.dim + a] = -s;
      }
}

}  // namespace
}  // namespace obte

struct obte_fourier_plan_s {
  obte_context ctx = nullptr;
  int64_t n = 0, ns_int = 0, nc = 0;
  int dim = 2, nv = 3, pin = -1;
  int nb = 1;
  double normalization = 0, contact_t2 = 0;
  std::vector<double> kappa;
  obte::DevBuf rp, ci, val, dinv, vol, B, colpin, g_nb, g_off, g_mixed, gw, s_i, s_j, s_w, s_vnon, c_ptr, c_side,
      k_e1, k_e2, k_coef, kap;
  // work
  obte::DevBuf C, r, z, p, Ap, part, sc, grad;
  obte::HostBuf hout;               // the two counts of a solve, its error word and kappa terms, written by the device
  int test_skip = -1, test_polls = 0;   // obte_fourier_plan_test_barrier_timeout
  // smoothed-aggregation AMG V-cycle as the CG preconditioner (null: Jacobi)
  obte::AmgPtr amg;
};

using namespace obte;

extern "C" obte_status obte_fourier_plan_create(obte_context ctx, const obte_fourier_problem* pb,
                                                obte_fourier_plan* out) {
  if (!ctx || !pb || !out) { set_error("null argument"); return OBTE_ERR_BAD_ARG; }
  const int dim = pb->dim;
  const int64_t n = pb->n_elems, ns = pb->n_sides;
  const int nv = pb->elem_nv;
  if ((dim != 2 && dim != 3) || n <= 0 || ns <= 0 || nv < dim + 1 || nv > 8 || !pb->side_elem_map ||
      !pb->normal_areas || !pb->dists || !pb->elem_volumes || !pb->interp_weights || !pb->gradient_weights ||
      !pb->elem_side_map || !pb->kappa) {
    set_error("bad Fourier problem");
    return OBTE_ERR_BAD_ARG;
  }
  OBTE_CUDA(cudaSetDevice(ctx->device));
  const int64_t* sem = pb->side_elem_map;
  const double* na = pb->normal_areas;
  const double* vol = pb->elem_volumes;
  auto inr = [&](int64_t v, int64_t m) { return v >= 0 && v < m; };
  // v_orth, v_nonorth (objects.py:312-319)
  std::vector<double> vo(ns), vn(ns * dim);
  const double* K = pb->kappa;
  for (int64_t s = 0; s < ns; ++s) {
    double num = 0, den = 0;
    double kn[3] = {0, 0, 0};
    for (int a = 0; a < dim; ++a)
      for (int b = 0; b < dim; ++b) kn[a] += K[a * dim + b] * na[s * dim + b];
    for (int a = 0; a < dim; ++a) { num += na[s * dim + a] * kn[a]; den += na[s * dim + a] * pb->dists[s * dim + a]; }
    vo[s] = num / den;
    for (int a = 0; a < dim; ++a) vn[s * dim + a] = kn[a] - pb->dists[s * dim + a] * vo[s];
  }
  // L (symmetric, volume-weighted) as a map per row; B (fourier.py:51-107)
  std::vector<std::map<int64_t, double>> L(n);
  std::vector<double> B(n, 0.0);
  for (int64_t t = 0; t < pb->n_internal; ++t) {
    const int64_t s = pb->internal[t];
    if (!inr(s, ns)) { set_error("internal side out of range"); return OBTE_ERR_BAD_ARG; }
    const int64_t i = sem[2 * s], j = sem[2 * s + 1];
    if (!inr(i, n) || !inr(j, n)) { set_error("side_elem_map out of range"); return OBTE_ERR_BAD_ARG; }
    L[i][i] += vo[s]; L[i][j] -= vo[s];
    L[j][j] += vo[s]; L[j][i] -= vo[s];
  }
  for (int64_t k = 0; k < pb->n_mixed; ++k) {
    const int64_t s = pb->mixed_sides[k];
    if (!inr(s, ns)) { set_error("mixed side out of range"); return OBTE_ERR_BAD_ARG; }
    const int64_t i = sem[2 * s];
    const double h = pb->mixed_conductance[k];
    const double tmp = vo[s] * h / (h + vo[s] / pb->side_areas[s]);
    L[i][i] += tmp;
    B[i] = pb->mixed_value[k] * tmp / vol[i];
  }
  for (int64_t k = 0; k < pb->n_periodic; ++k) {
    const int64_t s = pb->periodic_sides[k];
    if (!inr(s, ns)) { set_error("periodic side out of range"); return OBTE_ERR_BAD_ARG; }
    const int64_t i = sem[2 * s], j = sem[2 * s + 1];
    B[i] += pb->periodic_jump[k] * vo[s] / vol[i];
    B[j] -= pb->periodic_jump[k] * vo[s] / vol[j];
  }
  if (pb->heat_source)
    for (int64_t i = 0; i < n; ++i) B[i] += pb->heat_source[i] * 1e-18;
  int pin = -1;
  if (pb->n_mixed == 0) {
    pin = pb->pin_elem;
    if (!inr(pin, n)) { set_error("pin element out of range"); return OBTE_ERR_BAD_ARG; }
    B[pin] = 0;
  }
  // masked CSR (row and column of the pinned element removed; its column kept aside)
  std::vector<int32_t> rp(n + 1, 0), ci;
  std::vector<double> val, dinv(n, 0.0), colpin(n, 0.0);
  for (int64_t i = 0; i < n; ++i) {
    if ((int)i != pin)
      for (auto& kv : L[i]) {
        if (kv.first == pin) { colpin[i] = kv.second; continue; }
        ci.push_back((int32_t)kv.first);
        val.push_back(kv.second);
        if (kv.first == i) dinv[i] = kv.second != 0 ? 1.0 / kv.second : 0.0;
      }
    rp[i + 1] = (int32_t)ci.size();
  }
  // gradient stencil (objects.py:330-403)
  std::vector<int32_t> gnb(n * nv, -1);
  std::vector<double> goff(n * nv, 0.0);
  std::vector<unsigned char> gmix(n * nv, 0);
  std::vector<int64_t> esm(pb->elem_side_map, pb->elem_side_map + n * nv);
  auto slot_of = [&](int64_t e, int64_t s) -> int {
    for (int k = 0; k < nv; ++k)
      if (esm[e * nv + k] == s) return k;
    return -1;
  };
  for (int64_t t = 0; t < pb->n_internal; ++t) {
    const int64_t s = pb->internal[t];
    const int64_t i = sem[2 * s], j = sem[2 * s + 1];
    const int a = slot_of(i, s), b = slot_of(j, s);
    if (a < 0 || b < 0) { set_error("elem_side_map does not list an internal side"); return OBTE_ERR_BAD_ARG; }
    gnb[i * nv + a] = (int32_t)j;
    gnb[j * nv + b] = (int32_t)i;
  }
  for (int64_t k = 0; k < pb->n_periodic; ++k) {
    const int64_t s = pb->periodic_sides[k];
    const int64_t i = sem[2 * s], j = sem[2 * s + 1];
    const int a = slot_of(i, s), b = slot_of(j, s);
    if (a < 0 || b < 0) { set_error("elem_side_map does not list a periodic side"); return OBTE_ERR_BAD_ARG; }
    goff[i * nv + a] += pb->periodic_jump[k];
    goff[j * nv + b] -= pb->periodic_jump[k];
  }
  for (int64_t k = 0; k < pb->n_mixed; ++k) {
    const int64_t s = pb->mixed_sides[k];
    const int64_t i = sem[2 * s];
    const int a = slot_of(i, s);
    if (a < 0) { set_error("elem_side_map does not list a mixed side"); return OBTE_ERR_BAD_ARG; }
    gmix[i * nv + a] = 1;
    goff[i * nv + a] = pb->mixed_value[k];
  }
  // correction: internal sides and per-element gather lists (+ side+1 / -(side+1))
  const int64_t ni = pb->n_internal;
  std::vector<int32_t> s_i(ni), s_j(ni);
  std::vector<double> s_w(ni), s_vn(ni * dim);
  std::vector<std::vector<int32_t>> gl(n);
  for (int64_t t = 0; t < ni; ++t) {
    const int64_t s = pb->internal[t];
    s_i[t] = (int32_t)sem[2 * s];
    s_j[t] = (int32_t)sem[2 * s + 1];
    s_w[t] = pb->interp_weights[s];
    for (int a = 0; a < dim; ++a) s_vn[t * dim + a] = vn[s * dim + a];
    gl[s_i[t]].push_back((int32_t)t);
    gl[s_j[t]].push_back((int32_t)(-t - 1));
  }
  std::vector<int32_t> cptr(n + 1, 0), cside;
  for (int64_t c = 0; c < n; ++c) {
    cside.insert(cside.end(), gl[c].begin(), gl[c].end());
    cptr[c + 1] = (int32_t)cside.size();
  }
  // contact (objects.py:139-172)
  std::vector<int32_t> ke1, ke2;
  std::vector<double> kco;
  double t2const = 0;
  if (pb->contact_kind == OBTE_CONTACT_PERIODIC || pb->contact_kind == OBTE_CONTACT_MIXED) {
    for (int64_t k = 0; k < pb->n_contact; ++k) {
      const int64_t s = pb->contact_sides[k];
      if (!inr(s, ns)) { set_error("contact side out of range"); return OBTE_ERR_BAD_ARG; }
      ke1.push_back((int32_t)sem[2 * s]);
      if (pb->contact_kind == OBTE_CONTACT_PERIODIC) {
        ke2.push_back((int32_t)sem[2 * s + 1]);
        kco.push_back(vo[s] * pb->normalization);
      } else {
        ke2.push_back(-1);
        const double h = pb->contact_conductance;
        kco.push_back(vo[s] * h / (h + vo[s] / pb->side_areas[s]) * pb->normalization);
      }
    }
    t2const = pb->contact_alpha;
  }
  auto* P = new obte_fourier_plan_s();
  P->ctx = ctx;
  P->n = n; P->dim = dim; P->nv = nv; P->pin = pin; P->ns_int = ni; P->nc = (int64_t)ke1.size();
  P->contact_t2 = t2const;
  P->kappa.assign(pb->kappa, pb->kappa + dim * dim);
  P->nb = (int)std::max<int64_t>(1, std::min<int64_t>((n + FT - 1) / FT, (int64_t)ctx->num_sms * 2));
  cudaStream_t st = ctx->stream;
  std::vector<double> volv(vol, vol + n);
  std::vector<double> gwv(pb->gradient_weights, pb->gradient_weights + n * dim * nv);
  std::vector<int32_t> gmix32(gmix.begin(), gmix.end());
  obte_status s0 = OBTE_OK;
  auto up = [&](obte_status s) { if (s0 == OBTE_OK) s0 = s; };
  up(upload(P->rp, rp, st)); up(upload(P->ci, ci, st)); up(upload(P->val, val, st)); up(upload(P->dinv, dinv, st));
  up(upload(P->vol, volv, st)); up(upload(P->B, B, st)); up(upload(P->colpin, colpin, st));
  up(upload(P->g_nb, gnb, st)); up(upload(P->g_off, goff, st));
  {
    std::vector<int32_t> tmpm(gmix.size());
    // stored as bytes on the device
    up(P->g_mixed.alloc(gmix.size()));
    if (s0 == OBTE_OK && !gmix.empty()) {
      cudaError_t e = cudaMemcpyAsync(P->g_mixed.p, gmix.data(), gmix.size(), cudaMemcpyHostToDevice, st);
      if (e != cudaSuccess) up(cuda_fail(e, "cudaMemcpyAsync", __FILE__, __LINE__));
    }
  }
  up(upload(P->gw, gwv, st));
  up(upload(P->s_i, s_i, st)); up(upload(P->s_j, s_j, st)); up(upload(P->s_w, s_w, st)); up(upload(P->s_vnon, s_vn, st));
  up(upload(P->c_ptr, cptr, st)); up(upload(P->c_side, cside, st));
  up(upload(P->k_e1, ke1, st)); up(upload(P->k_e2, ke2, st)); up(upload(P->k_coef, kco, st));
  up(upload(P->kap, P->kappa, st));
  const size_t vb = (size_t)n * sizeof(double);
  // r and p alternate between two buffers; partials: seven sums of one value per block
  up(P->C.alloc(vb)); up(P->r.alloc(2 * vb)); up(P->z.alloc(vb)); up(P->p.alloc(2 * vb));
  up(P->Ap.alloc(vb)); up(P->part.alloc(7 * sizeof(double) * (size_t)fourier_shape(n, ctx->num_sms).blocks));
  up(P->sc.alloc(4 * sizeof(double))); up(P->grad.alloc(vb * dim));
  // OBTE_FOURIER_JACOBI=1 keeps the diagonal preconditioner (same solution, ~40x more CG iterations)
  const char* jac = std::getenv("OBTE_FOURIER_JACOBI");
  if (s0 == OBTE_OK && !(jac && std::atoi(jac) != 0))
    up(amg_build(n, rp, ci, val, pin, st, P->amg));
  if (s0 == OBTE_OK) {
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) s0 = cuda_fail(e, "cudaStreamSynchronize", __FILE__, __LINE__);
  }
  if (s0 != OBTE_OK) { delete P; return s0; }
  *out = P;
  return OBTE_OK;
}

extern "C" obte_status obte_fourier_plan_destroy(obte_fourier_plan plan) {
  if (plan && plan->ctx) cudaStreamSynchronize(plan->ctx->stream);
  delete plan;
  return OBTE_OK;
}

extern "C" obte_status obte_fourier_plan_test_barrier_timeout(obte_fourier_plan plan, int32_t skip_barrier,
                                                              int32_t wait_limit) {
  if (!plan) { set_error("null plan"); return OBTE_ERR_BAD_ARG; }
  if (skip_barrier < -1 || wait_limit < 0) { set_error("skip_barrier must be >= -1 and wait_limit >= 0"); return OBTE_ERR_BAD_ARG; }
  plan->test_skip = skip_barrier;
  plan->test_polls = wait_limit;
  return OBTE_OK;
}

extern "C" obte_status obte_fourier_solve(obte_fourier_plan P, const obte_fourier_opts* opts, double* T, double* J,
                                          obte_fourier_info* info) {
  if (!P || !opts || !T) { set_error("null argument"); return OBTE_ERR_BAD_ARG; }
  cudaStream_t st = P->ctx->stream;
  const int64_t n = P->n;
  const int nb = P->nb;
  const int max_iter = opts->max_iter > 0 ? opts->max_iter : 40;
  const double rtol = opts->rtol > 0 ? opts->rtol : 1e-8;
  const double cg_rtol = opts->cg_rtol > 0 ? opts->cg_rtol : 1e-13;
  const int cg_max = opts->cg_max_iter > 0 ? opts->cg_max_iter : 20000;
  if (!P->hout.p) OBTE_TRY(P->hout.alloc((size_t)(4 + P->nc) * sizeof(double)));
  FourierParams f = {};
  f.n = n;
  f.A = CsrDev{n, P->rp.as<int32_t>(), P->ci.as<int32_t>(), P->val.as<double>()};
  f.has_amg = P->amg ? 1 : 0;
  if (P->amg) amg_device(*P->amg, f.amg, false);
  f.dinv = P->dinv.as<double>(); f.vol = P->vol.as<double>(); f.B = P->B.as<double>(); f.colpin = P->colpin.as<double>();
  f.pin = P->pin; f.nv = P->nv; f.dim = P->dim;
  f.g_nb = P->g_nb.as<int32_t>(); f.g_off = P->g_off.as<double>(); f.g_mixed = P->g_mixed.as<unsigned char>();
  f.gw = P->gw.as<double>();
  f.s_i = P->s_i.as<int32_t>(); f.s_j = P->s_j.as<int32_t>(); f.s_w = P->s_w.as<double>(); f.s_vnon = P->s_vnon.as<double>();
  f.c_ptr = P->c_ptr.as<int32_t>(); f.c_side = P->c_side.as<int32_t>();
  f.T = T; f.C = P->C.as<double>();
  f.r[0] = P->r.as<double>(); f.r[1] = f.r[0] + n;
  f.p[0] = P->p.as<double>(); f.p[1] = f.p[0] + n;
  f.z = P->z.as<double>(); f.Ap = P->Ap.as<double>(); f.grad = P->grad.as<double>(); f.part = P->part.as<double>();
  f.max_iter = max_iter; f.cg_max = cg_max;
  f.check = P->amg ? 4 : 8;          // iterations between two convergence tests
  f.rtol = rtol; f.cg_rtol = cg_rtol;
  f.out = P->sc.as<double>();
  f.bar = {reinterpret_cast<unsigned*>(f.out + 2), reinterpret_cast<int*>(f.out + 3),
           P->test_polls > 0 ? P->test_polls : kBarrierPolls, P->test_skip};
  OBTE_CUDA(cudaMemsetAsync(P->sc.p, 0, 4 * sizeof(double), st));
  const PhaseShape shape = fourier_shape(n, P->ctx->num_sms);
  // shared memory for a block's part of the matrices (an eighth more, as rows differ), as far as it may have
  const int64_t bytes = (int64_t)(P->val.bytes + P->ci.bytes + P->rp.bytes) + (P->amg ? amg_bytes(*P->amg) : 0);
  const bool wide = shape.threads == WideGridBarrier::kThreads;
  const int most = shape.cluster ? ClusterBarrier::kSmem : wide ? WideGridBarrier::kSmem : GridBarrier::kSmem;
  f.smem = (int)std::min<int64_t>(most, (bytes / shape.blocks * 9 / 8 + 2048 + 127) & ~(int64_t)127);
  OBTE_CUDA(phase_launch(shape, shape.cluster ? fourier_kernel<ClusterBarrier>
                                : wide        ? fourier_kernel<WideGridBarrier>
                                              : fourier_kernel<GridBarrier>,
                         f, f.smem, most, st));
  count_launch();
  double* h = P->hout.as<double>();
  OutputParams o = {};
  o.n = n; o.nc = P->nc; o.dim = P->dim;
  o.e1 = P->k_e1.as<int32_t>(); o.e2 = P->k_e2.as<int32_t>(); o.coef = P->k_coef.as<double>();
  o.T = T; o.kap = P->kap.as<double>(); o.grad = P->grad.as<double>(); o.sc = P->sc.as<double>();
  o.t2const = P->contact_t2;
  o.J = J; o.words = h; o.terms = h + 4;
  fourier_outputs_kernel<<<nb, FT, 0, st>>>(o);
  count_launch();
  OBTE_CUDA(cudaGetLastError());
  OBTE_CUDA(cudaStreamSynchronize(st));
  if (reinterpret_cast<int*>(h + 3)[0] != 0) {
    set_error("a device-side wait timed out in the Fourier kernel");
    return OBTE_ERR_DEVICE_TIMEOUT;
  }
  double kappa = 0;
  for (int64_t k = 0; k < P->nc; ++k) kappa += h[4 + k];
  if (info) {
    info->kappa = kappa;
    info->n_iter = (int32_t)h[0];
    info->n_cg = (int32_t)h[1];
  }
  return OBTE_OK;
}
