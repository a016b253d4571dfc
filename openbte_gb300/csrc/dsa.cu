// Diffusion-synthetic acceleration (DSA) of the GMRES on the sweep fixed point.
//
// The reference iterates the source step dT <- sum_mq t_coeff T_mq(dT) plainly (openbte/bte.py:193-249);
// where the transport is diffusive at the scale of the slow error — temperatures relaxing across a
// network of partially transmitting interfaces (openbte/inverse/bte.py:145-163), or through many mean
// free paths — each step removes only a small part of a smooth error and the iteration count grows
// with the size of the cell.  For a smooth temperature error e the transport operator acts as a
// diffusion operator: with T_mq = (1 + F_mq . grad)^-1 e ~ e - F . grad e + (F . grad)^2 e and
// sum_mq t_mq = 1, sum_mq t_mq F_mq = 0,
//     (I - K) e = div(sum_mq t_mq F_mq T_mq) ~ -div(D grad e),   D = sum_mq t_mq F_mq F_mq^T,
// F_mq = mfp_m v_q.  The right preconditioner M^-1 = I + E L^-1 R adds to a GMRES direction v the
// solution of the diffusion problem whose source is v's temperature part: R takes the temperature
// entries weighted by the element volumes, L is the finite-volume diffusion operator on the elements,
// E adds the cell correction to the temperatures, to the wall temperatures of each wall's element and to
// the periodic inflow of each source slot's element (a smooth correction shifts them alike).
//
// L (symmetric, volume-weighted): per internal side k between elements i, j, with area A and centre
// distance d, the conductance
//     A sum_m 1 / (d / D_m + (1 - t_k) / (G_m t_k))
// in series per MFP m: the bulk D_m = sum_q t_mq mfp_m^2 |v_q|^2 / dim and, on a side that transmits the
// fraction t < 1 of the phonons, the interface conductance G_m t / (1 - t), G_m = sum_q t_mq
// max(F_mq . n, 0) (the half-range flux; two-stream balance of the transmitted and reflected streams at
// the interface).  Periodic sides couple their elements like internal ones (the correction carries no
// jump); diffuse walls are insulating; isothermal walls hold the correction at zero through
// A sum_m 1 / (d / D_m + 1 / (2 G_m)).  No diagonal is below 5 % of the (upper) median (per volume): an element
// whose sides barely transmit keeps its slow mode to GMRES.  Without isothermal walls L has the constant
// null vector, as I - K has the uniform shift: the source is projected onto zero mean and the
// correction's volume-weighted mean removed, and a diagonal of 1e-6 of the largest keeps the hierarchy's
// coarsest operator invertible.
//
// The solve is `cycles` (OBTE_DSA_CYCLES, default 1) steps of d <- d + B (b - L d) from d = 0 with B one
// V-cycle of the smoothed-aggregation hierarchy of amg.cu: a fixed linear map, as the non-flexible GMRES
// requires of its preconditioner (on the 128^2-pixel design problem, 50 MFPs x 64 directions: 210 sweeps per
// gradient evaluation without it, 89 / 88 / 88 with 1 / 2 / 3 cycles).  The operator is built on the plan's
// first accelerated solve and rebuilt after new side transmissions.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "grid.cuh"

namespace obte {

namespace {

struct DsaParams {
  int64_t n, nd, nu;
  int n_mfp, project, cycles;
  double inv_vol_sum;
  CsrDev A;                                  // L
  AmgDev amg;
  const double* vol;
  const int32_t *wcell, *xcell;
  const double *in, *base;
  double *out, *b, *d, *r, *e, *part;
  BarrierParams bar;
  unsigned* count_next;                      // the next application's barrier counter, cleared here
};

// out = base + E L^-1 R in, one launch.  Phases end at a barrier (grid.cuh): the weighted sum of `in`; the
// right-hand side b = V (in - mean) formed in the gather of its restriction; the V-cycle; the weighted sum of
// d; the extension out[i] = base[i] + d[cell(i)] - mean over the state: temperatures, wall temperatures (element
// of the wall), periodic inflow (element of the source slot, every MFP).
//
// As 12 launches of 3.9 us each with its gap an application took 47 us (64^2 and 128^2 pixels); with the Arnoldi
// step in one launch as well, 64^2 pixels x 20 x 32 went from 33.1 to 26.5 ms a gradient evaluation.
template <typename Bar>
__global__ void __launch_bounds__(Bar::kThreads, Bar::kBlocks == 1 ? 1 : 4) dsa_kernel(const __grid_constant__ DsaParams P) {
  __shared__ double red[Bar::kThreads];
  __shared__ Rows sA;
  __shared__ AmgRows sM;
  Bar bar(P.bar);
  const int tid = threadIdx.x, nthr = blockDim.x, nb = gridDim.x;
  if (blockIdx.x == 0 && tid == 0) *P.count_next = 0;
  Arena ar{nullptr, 0};                      // read once: not worth copying
  load_amg(P.amg, &sM, ar, 32);
  if (P.cycles > 1) load_rows(P.A, &sA, ar, 32);
  int r0, r1;
  block_range(P.n, r0, r1, 32);
  // V x over each 32 consecutive elements of the block (x complete in the block)
  const int segments = (int)((P.n + 31) / 32);
  auto weigh = [&](const double* x, double* seg) {
    for (int i0 = r0 + (tid & ~31); i0 < r1; i0 += nthr) {       // whole warps
      const int i = i0 + (tid & 31);
      double v = i < r1 ? P.vol[i] * x[i] : 0.0;
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if ((tid & 31) == 0) seg[i0 >> 5] = v;
    }
  };
  // The mean from the segments' sums (after a barrier), in one order for every number of blocks: the correction
  // of a nearly singular operator is sensitive to the rounding of the means, and an FP32 basis turns that
  // into another, equally good, iterate.
  auto mean = [&](const double* seg) {
    double v = 0;
    if (tid < 256)
      for (int i = tid * 8; i < segments; i += 8 * 256) {
        double a[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = i + j < segments ? seg[i + j] : 0.0;
        v += ((a[0] + a[4]) + (a[2] + a[6])) + ((a[1] + a[5]) + (a[3] + a[7]));
      }
    if (tid < 256)
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (tid < 256 && (tid & 31) == 0) red[1 + (tid >> 5)] = v;
    __syncthreads();
    if (tid == 0) {
      const double* a = red + 1;
      red[0] = (((a[0] + a[4]) + (a[2] + a[6])) + ((a[1] + a[5]) + (a[3] + a[7]))) * P.inv_vol_sum;
    }
    __syncthreads();
    return red[0];
  };
  __syncthreads();
  double mu = 0;
  if (P.project) {
    weigh(P.in, P.part);
    if (!bar.wait()) return;
    mu = mean(P.part);
  }
  const int nl = P.amg.nl;
  for (int i = r0 + tid; i < r1; i += nthr) P.b[i] = P.vol[i] * (P.in[i] - mu);
  auto restrict0 = [&](auto value) {         // b_1 = Q_0^T b
    double* b1 = P.amg.b[1];
    block_rows(sM.Qt[0], value, [&](int row, double v) { b1[row] = v; });
  };
  if (nl > 1) restrict0([&](int c) { return P.vol[c] * (P.in[c] - mu); });
  if (!bar.wait()) return;
  // x = B rhs with one V-cycle, after the restriction
  auto cycle = [&](const double* rhs, double* x) -> bool {
    auto up = [&](int row, double v) { x[row] = v; };
    if (nl == 1) {
      block_dense(sM, P.amg.nc, rhs, up);
      return true;
    }
    return amg_cycle(P.amg, sM, bar, [&](int c) { return rhs[c]; }, up);
  };
  if (!cycle(P.b, P.d)) return;
  for (int c = 1; c < P.cycles; ++c) {       // d += B (b - L d)
    if (!bar.wait()) return;
    block_rows(sA, [&](int j) { return P.d[j]; }, [&](int i, double s) { P.r[i] = P.b[i] - s; });
    if (!bar.wait()) return;
    if (nl > 1) {
      restrict0([&](int j) { return P.r[j]; });
      if (!bar.wait()) return;
    }
    if (!cycle(P.r, P.e)) return;
    if (!bar.wait()) return;
    for (int i = r0 + tid; i < r1; i += nthr) P.d[i] += P.e[i];
  }
  __syncthreads();                           // the block's rows of d, by other threads than those that add them up
  mu = 0;
  if (P.project) weigh(P.d, P.part + segments);
  if (!bar.wait()) return;
  if (P.project) mu = mean(P.part + segments);
  const int64_t n = P.n, xoff = P.n + P.nd, t = (int64_t)blockIdx.x * nthr + tid, stride = (int64_t)nb * nthr;
  // four entries of a thread at a time, their loads (element, correction) before any store: the state is larger than
  // the elements by the walls and the inflow, and a block has few threads
  for (int64_t i0 = t; i0 < P.nu; i0 += 4 * stride) {
    double v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int64_t i = i0 + k * stride, x = i - xoff;
      if (i >= P.nu) continue;
      int64_t c = i;
      if (x >= 0) c = P.xcell[P.nu < ((int64_t)1 << 31) ? (int64_t)((unsigned)x / (unsigned)P.n_mfp) : x / P.n_mfp];
      else if (i >= n) c = P.wcell[i - n];
      v[k] = P.base[i] + (P.d[c] - mu);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i0 + k * stride < P.nu) P.out[i0 + k * stride] = v[k];
  }
}

}  // namespace

bool dsa_default(const Schedule& s) {
  // on where a side transmits only part of the phonons (the transmission-interface model): the slow
  // modes there are interface-network diffusion modes
  for (double t : s.dsa.t)
    if (t < 1.0) return true;
  return false;
}

// L as CSR (columns sorted, duplicates merged); `project`: L has the constant null vector
void dsa_matrix(const Schedule& s, std::vector<int32_t>& rp, std::vector<int32_t>& ci, std::vector<double>& val,
                bool& project) {
  const Schedule::DsaData& D = s.dsa;
  const int64_t n = s.n;
  const int n_mfp = s.n_mfp;
  double Dsum = 0;
  for (double v : D.Dm) Dsum += v;
  // conductances of the sides
  const int64_t nfc = (int64_t)D.e1.size();
  std::vector<double> coef(nfc, 0.0);
  parallel_for(nfc, [&](int64_t k) {
    const double t = D.t[k];
    double c = 0;
    if (t >= 1.0) {
      c = Dsum / D.dist[k];
    } else {
      for (int m = 0; m < n_mfp; ++m) {
        const double r = D.dist[k] / D.Dm[m] + (1.0 - t) / (D.Gm[m] * t);
        if (r > 0 && std::isfinite(r)) c += 1.0 / r;
      }
    }
    coef[k] = D.area[k] * c;
  }, std::max<int64_t>(64, 20000 / std::max(n_mfp, 1)));
  std::vector<double> diag(n, 0.0);
  std::vector<int32_t> deg(n + 1, 0);
  for (int64_t k = 0; k < nfc; ++k) {
    if (D.e1[k] == D.e2[k]) continue;
    diag[D.e1[k]] += coef[k];
    diag[D.e2[k]] += coef[k];
    ++deg[D.e1[k] + 1];
    ++deg[D.e2[k] + 1];
  }
  for (size_t k = 0; k < D.iso_cell.size(); ++k) {
    double c = 0;
    for (int m = 0; m < n_mfp; ++m) c += 1.0 / (D.iso_dist[k] / D.Dm[m] + 0.5 / D.Gm[m]);
    diag[D.iso_cell[k]] += D.iso_area[k] * c;
  }
  project = D.iso_cell.empty();
  double dmax = 0;
  for (double v : diag) dmax = std::max(dmax, v);
  const double reg = 1e-6 * (dmax > 0 ? dmax : 1.0);
  // an element whose sides barely transmit (a pore pixel, t ~ 1e-12) has a temperature mode that I - K
  // relaxes at a rate ~t: the diffusion operator models that rate, but inverting it would multiply the
  // rounding noise of the FP32 sweeps in that element by ~1 / t.  Its diagonal is raised to 5 % of the
  // median, so the correction leaves such modes to GMRES as if there were no acceleration.
  {
    std::vector<double> dd;
    dd.reserve(n);
    for (int64_t i = 0; i < n; ++i) dd.push_back(diag[i] / D.vol[i]);
    std::nth_element(dd.begin(), dd.begin() + n / 2, dd.end());
    const double floor_per_vol = 0.05 * dd[n / 2];
    for (int64_t i = 0; i < n; ++i) diag[i] = std::max(diag[i], floor_per_vol * D.vol[i]);
  }
  // CSR: diagonal first, then the neighbours in side order; two sides joining the same pair (periodic
  // images) stay separate entries
  rp.assign(n + 1, 0);
  for (int64_t i = 0; i < n; ++i) rp[i + 1] = rp[i] + 1 + deg[i + 1];
  ci.assign(rp[n], 0);
  val.assign(rp[n], 0.0);
  std::vector<int32_t> pos(rp.begin(), rp.end() - 1);
  for (int64_t i = 0; i < n; ++i) {
    ci[pos[i]] = (int32_t)i;
    val[pos[i]++] = diag[i] + reg;
  }
  for (int64_t k = 0; k < nfc; ++k) {
    const int32_t i = D.e1[k], j = D.e2[k];
    if (i == j) continue;
    ci[pos[i]] = j; val[pos[i]++] = -coef[k];
    ci[pos[j]] = i; val[pos[j]++] = -coef[k];
  }
  // the hierarchy wants sorted columns with duplicates merged
  {
    std::vector<int32_t> rp2(n + 1, 0), ci2;
    std::vector<double> val2;
    ci2.reserve(ci.size());
    val2.reserve(val.size());
    std::vector<std::pair<int32_t, double>> row;
    for (int64_t i = 0; i < n; ++i) {
      row.clear();
      for (int32_t k = rp[i]; k < rp[i + 1]; ++k) row.emplace_back(ci[k], val[k]);
      std::sort(row.begin(), row.end(), [](const std::pair<int32_t, double>& a, const std::pair<int32_t, double>& b) {
        return a.first < b.first;
      });
      for (size_t k = 0; k < row.size(); ++k) {
        if (!ci2.empty() && (int64_t)ci2.size() > rp2[i] && ci2.back() == row[k].first) {
          val2.back() += row[k].second;
        } else {
          ci2.push_back(row[k].first);
          val2.push_back(row[k].second);
        }
      }
      rp2[i + 1] = (int32_t)ci2.size();
    }
    rp.swap(rp2);
    ci.swap(ci2);
    val.swap(val2);
  }
}

obte_status ensure_dsa(obte_plan plan) {
  if (plan->dsa) return OBTE_OK;
  PhaseTimer timer("dsa setup");
  const auto t0 = std::chrono::steady_clock::now();
  const Schedule& s = plan->sched;
  const Schedule::DsaData& D = s.dsa;
  const int64_t n = s.n;
  const int64_t nfc = (int64_t)D.e1.size();
  std::vector<int32_t> rp, ci;
  std::vector<double> val;
  bool project = true;
  dsa_matrix(s, rp, ci, val, project);
  std::unique_ptr<DsaOp> op(new DsaOp());
  cudaStream_t st = plan->stream;
  // rebuilt for every density field of a design loop: coarsen down to 64 rows, whose dense inverse costs
  // little (on 128^2 pixels the hierarchy's set-up took 16.5 ms with the default 400-row coarsest
  // operator, 6.8 ms with 64 rows, for one more sweep per solve)
  OBTE_TRY(amg_build(n, rp, ci, val, -1, st, op->amg, 64));
  OBTE_TRY(upload(op->rp, rp, st));
  OBTE_TRY(upload(op->ci, ci, st));
  OBTE_TRY(upload(op->val, val, st));
  OBTE_TRY(upload(op->vol, D.vol, st));
  for (DevBuf* b : {&op->b, &op->d, &op->r, &op->e}) OBTE_TRY(b->alloc((size_t)n * sizeof(double)));
  // partial sums of the two weighted means, and the two barrier counters that launches use in turn
  const int64_t segments = (n + 31) / 32;
  OBTE_TRY(op->mean.alloc((size_t)(2 * segments + 1) * sizeof(double)));
  OBTE_CUDA(cudaMemsetAsync(op->mean.as<double>() + 2 * segments, 0, sizeof(double), st));
  double vs = 0;
  for (double v : D.vol) vs += v;
  op->inv_vol_sum = vs > 0 ? 1.0 / vs : 0.0;
  op->project = project;
  if (const char* e = std::getenv("OBTE_DSA_CYCLES")) op->cycles = std::max(1, std::min(16, std::atoi(e)));
  op->levels = amg_levels(*op->amg);
  op->bytes = (int64_t)(op->rp.bytes + op->ci.bytes + op->val.bytes + op->vol.bytes + 4 * n * sizeof(double));
  OBTE_CUDA(wait_stream(st));
  op->setup_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  if (timer.on)
    std::fprintf(stderr, "[obte trace] dsa: %lld elements, %lld sides, %d levels, %d cycles per apply\n",
                 (long long)n, (long long)nfc, op->levels, op->cycles);
  plan->dsa = std::move(op);
  return OBTE_OK;
}

void dsa_start_async(obte_plan plan) {
  dsa_join(plan);
  if (!plan->ctx || !dsa_default(plan->sched)) return;
  plan->dsa.reset();
  plan->dsa_build_status = OBTE_OK;
  const int device = plan->ctx->device;
  plan->dsa_build = std::thread([plan, device] {
    if (cudaSetDevice(device) != cudaSuccess) {
      plan->dsa_build_status = OBTE_ERR_CUDA;
      return;
    }
    plan->dsa_build_status = ensure_dsa(plan);
  });
}

obte_status dsa_join(obte_plan plan) {
  if (plan->dsa_build.joinable()) plan->dsa_build.join();
  const obte_status st = plan->dsa_build_status;
  plan->dsa_build_status = OBTE_OK;
  if (st != OBTE_OK) plan->dsa.reset();      // a failed build is redone (with its message) by the solve
  return st;
}

obte_status dsa_add(obte_plan plan, const double* in, const double* base, double* out) {
  DsaOp& op = *plan->dsa;
  const Schedule& s = plan->sched;
  const PhaseShape ps = phase_shape(s.n, plan->ctx->num_sms);
  DsaParams f = {};
  f.n = s.n; f.nd = s.nd; f.nu = plan->nu; f.n_mfp = s.n_mfp;
  f.project = op.project ? 1 : 0;
  f.cycles = op.cycles;
  f.inv_vol_sum = op.inv_vol_sum;
  f.A = CsrDev{s.n, op.rp.as<int32_t>(), op.ci.as<int32_t>(), op.val.as<double>()};
  amg_device(*op.amg, f.amg, true);
  f.vol = op.vol.as<double>();
  f.wcell = plan->diffuse_cell.as<int32_t>();
  f.xcell = plan->x_cell.as<int32_t>();
  f.in = in; f.base = base; f.out = out;
  f.b = op.b.as<double>(); f.d = op.d.as<double>(); f.r = op.r.as<double>(); f.e = op.e.as<double>();
  f.part = op.mean.as<double>();
  unsigned* count = reinterpret_cast<unsigned*>(f.part + 2 * ((s.n + 31) / 32));
  f.bar = {count + op.turn, plan->err.as<int>(),
           plan->test_barrier_polls > 0 ? plan->test_barrier_polls : kBarrierPolls, plan->test_barrier_skip};
  f.count_next = count + (op.turn ^ 1);
  OBTE_CUDA(phase_launch(ps, ps.cluster ? dsa_kernel<ClusterBarrier> : dsa_kernel<GridBarrier>, f, 0, 0, plan->stream));
  op.turn ^= 1;                   // a launch that failed has cleared nothing: its counter is still the next one
  count_launch();
  return OBTE_OK;
}

}  // namespace obte

using namespace obte;

extern "C" obte_status obte_bte_dsa_operator(obte_plan plan, int64_t* nnz, int32_t* row_ptr, int32_t* col,
                                             double* val, int32_t* project) {
  if (!plan || !nnz) { set_error("null argument"); return OBTE_ERR_BAD_ARG; }
  std::vector<int32_t> rp, ci;
  std::vector<double> v;
  bool proj = true;
  dsa_matrix(plan->sched, rp, ci, v, proj);
  const int64_t cap = *nnz;
  *nnz = (int64_t)ci.size();
  if (project) *project = proj ? 1 : 0;
  if (!row_ptr && !col && !val) return OBTE_OK;          // size query
  if (cap < (int64_t)ci.size()) { set_error("dsa operator: arrays too small"); return OBTE_ERR_BAD_ARG; }
  if (row_ptr) std::copy(rp.begin(), rp.end(), row_ptr);
  if (col) std::copy(ci.begin(), ci.end(), col);
  if (val) std::copy(v.begin(), v.end(), val);
  return OBTE_OK;
}
