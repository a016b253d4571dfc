// Device code shared by the kernels that run many small phases in one launch: a barrier over all blocks, sums
// over all blocks, sparse row products and the multigrid V-cycle.
//
// The phases of a multigrid-preconditioned iteration on a few thousand to a hundred thousand elements take
// 1-2 us each, less than the launch between two of them (3.9-4.6 us with its gap); here a phase ends at a
// barrier instead.  Small problems run as one cluster of 8 CTAs (hardware barrier, 0.4-0.8 us), larger ones on
// a part of every SM as a cooperative launch (all blocks resident) with an arrive counter in global memory (1.3 us).
// Vectors that change between phases are read with plain loads (never through the read-only path).
#pragma once

#include <cuda_runtime.h>

#include "internal.h"

namespace obte {

// float -> double, exactly, on the integer pipe for normal numbers (GB300's FP64 pipe converts two lanes a
// clock per SM; zeros, denormals, infinities and NaN take the conversion instruction)
__device__ __forceinline__ double widen(float f) {
  const unsigned b = __float_as_uint(f), e = b & 0x7f800000u;
  if (e == 0u || e == 0x7f800000u) return (double)f;
  return __hiloint2double((int)(((b & 0x7fffffffu) >> 3) + (896u << 20) | (b & 0x80000000u)), (int)(b << 29));
}

// What the barrier of a cooperative launch needs: its counter (zero at launch) and error word, the polls after which
// a wait gives up (a wait of 1-2 s by default), and for the test of that the barrier at which block 0 does not arrive
// (-1: none).
struct BarrierParams {
  unsigned* count;
  int* err;
  int polls, skip;
};
constexpr int kBarrierPolls = 1 << 21;

// Barrier over the blocks of a cluster.
struct ClusterBarrier {
  static constexpr int kThreads = 512, kBlocks = 1;      // threads per block, blocks an SM has registers for
  static constexpr int kSmem = 200 * 1024;               // shared memory for a solve's matrices at most
  __device__ ClusterBarrier(const BarrierParams&) {}
  __device__ bool wait() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    return true;
  }
};

// Barrier over the blocks of a cooperative launch: the counter grows by the number of blocks per
// barrier.  The wait is bounded; when it gives up (on any block) the error word is set and wait() is false in
// every thread of that block, whose caller returns; the other blocks run into their own bounds.
template <int THREADS, int BLOCKS, int SMEM>
struct GridBarrierOf {
  static constexpr int kThreads = THREADS, kBlocks = BLOCKS, kSmem = SMEM;
  unsigned* count;
  int* err;
  int polls;
  unsigned target = 0, skip;                 // skip: the target at which this block does not arrive, 0: none
  __device__ GridBarrierOf(const BarrierParams& p)
      : count(p.count), err(p.err), polls(p.polls), skip(blockIdx.x == 0 ? (unsigned)(p.skip + 1) * gridDim.x : 0) {}
  __device__ bool wait() {
    __shared__ int ok;
    __syncthreads();
    target += gridDim.x;
    if (threadIdx.x == 0) {
      if (target != skip) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
      int done = 0;
      for (int i = 0; i < polls && !done; ++i) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
        done = (int)(v - target) >= 0;
      }
      if (!done) atomicOr(err, 1);
      ok = done;
    }
    __syncthreads();
    return ok != 0;
  }
};

using GridBarrier = GridBarrierOf<256, 3, 69 * 1024>;          // a third of an SM to a block
using WideGridBarrier = GridBarrierOf<512, 2, 104 * 1024>;     // half

// Sum over the block's first `count` slots in a fixed order, valid in thread 0: the thread of slot s passes its
// value with slot = s, the others a negative slot; red: one double per thread.  A warp's FP64 operation holds its quarter
// of the SM for 64-76 cycles however many warps share it, so the sum is a chain of additions to be kept
// short: only the slots in use, four quarters at work on the first two levels, then one warp's shuffle tree.
__device__ __forceinline__ double block_sum(double v, int slot, int count, double* red) {
  __syncthreads();
  if (slot >= 0) red[slot] = v;
  __syncthreads();
  const int tid = threadIdx.x;
  auto four = [&](int n) {                     // red[tid], red[tid + n], ... of 4 n slots
    double a[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) a[j] = tid + j * n < count ? red[tid + j * n] : 0.0;
    return count > 2 * n ? (a[0] + a[1]) + (a[2] + a[3]) : a[0] + a[1];
  };
  if (count > 128) {                           // blockDim <= 512
    double s = 0;
    if (tid < 128) s = four(128);
    __syncthreads();
    if (tid < 128) red[tid] = s;
    __syncthreads();
    count = 128;
  }
  double s = 0;
  if (tid < 32) {
    s = four(32);
    for (int o = count > 16 ? 16 : count > 8 ? 8 : 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  return s;
}
// The largest value of the block, valid in warp 0.
__device__ __forceinline__ double block_max(double v, double* red) {
  __syncthreads();
  red[threadIdx.x] = v;
  __syncthreads();
  double s = -INFINITY;
  if (threadIdx.x < 32) {
    for (int k = threadIdx.x; k < (int)blockDim.x; k += 32) s = fmax(s, red[k]);
    for (int o = 16; o > 0; o >>= 1) s = fmax(s, __shfl_xor_sync(0xffffffffu, s, o));
  }
  return s;
}
// f(sum of nb block partials), f called by one thread and its value returned to all (part: written before the
// last barrier; fixed order).  Scalars are formed once: a division in every warp would hold the FP64 pipe for
// longer than the rest of the phase.
template <typename F>
__device__ __forceinline__ double grid_sum(const double* part, int nb, double* red, F f) {
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = 0;
    for (int b0 = threadIdx.x; b0 < nb; b0 += 256) {
      double a[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] = b0 + 32 * j < nb ? part[b0 + 32 * j] : 0.0;
      double w = a[0];
      if (nb > 32) w = (a[0] + a[1]) + (a[2] + a[3]);
      if (nb > 128) w += (a[4] + a[5]) + (a[6] + a[7]);
      v = b0 < 32 ? w : v + w;
    }
    for (int o = nb > 16 ? 16 : nb > 8 ? 8 : 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) red[0] = f(v);
  }
  __syncthreads();
  return red[0];
}

// Sparse matrix on the device.
struct CsrDev {
  int64_t n;
  const int32_t* rp;
  const int32_t* ci;
  const double* val;
  int vec = 0;              // lanes per row, 0: by the block's rows (load_rows)
};
constexpr int kAmgMaxLevels = 12;
struct AmgDev {
  int nl;                   // levels
  int nc;                   // coarsest rows
  const double* inv;        // dense inverse of the coarsest operator
  CsrDev G[kAmgMaxLevels], Q[kAmgMaxLevels], Qt[kAmgMaxLevels];
  double* b[kAmgMaxLevels];
  double* x[kAmgMaxLevels];
};
void amg_device(const AmgHierarchy& H, AmgDev& d, bool fixed_order);
int64_t amg_bytes(const AmgHierarchy& H);      // of the matrices that a V-cycle reads

// A block's rows [r0, r1) of a matrix; rp, ci and val are its own part, in shared memory where they fit.
struct Rows {
  int r0, r1;
  int base;                 // rp's value for the first of ci and val
  int vec;                  // lanes per row
  const int32_t* rp;
  const int32_t* ci;
  const double* val;
};
struct AmgRows {
  Rows G[kAmgMaxLevels], Q[kAmgMaxLevels], Qt[kAmgMaxLevels];
  int c0, c1;               // rows of the dense inverse
  const double* inv;
};
// Shared memory handed out in order to the parts a launch reads again in every iteration.
struct Arena {
  char* p;
  int left;
  __device__ void* take(int bytes) {
    bytes = (bytes + 15) & ~15;
    if (bytes > left) return nullptr;
    void* r = p;
    p += bytes;
    left -= bytes;
    return r;
  }
};
__device__ __forceinline__ void block_range(int64_t n, int& r0, int& r1, int align = 1) {
  int per = (int)((n + gridDim.x - 1) / gridDim.x);
  per = (per + align - 1) / align * align;
  r0 = (int)min((int64_t)per * blockIdx.x, n);
  r1 = (int)min((int64_t)per * (blockIdx.x + 1), n);
}
// This block's part of a matrix (called by all threads; thread 0 fills `d` in shared memory; a __syncthreads
// must follow).  A solve reads its matrices some hundred times over: from shared memory the gather of
// the vector is the only trip to L2 between two barriers.  (An empty arena leaves them where they are.)
__device__ __forceinline__ void load_rows(const CsrDev& m, Rows* d, Arena& ar, int align = 1) {
  int r0, r1;
  block_range(m.n, r0, r1, align);
  const int nr = r1 - r0, k0 = nr ? m.rp[r0] : 0, k1 = nr ? m.rp[r1] : 0;
  const int32_t *rp = m.rp + r0, *ci = m.ci + k0;
  const double* val = m.val + k0;
  if (double* sv = static_cast<double*>(ar.take((k1 - k0) * 8))) {
    for (int k = threadIdx.x; k < k1 - k0; k += blockDim.x) sv[k] = val[k];
    val = sv;
  }
  if (int32_t* sc = static_cast<int32_t*>(ar.take((k1 - k0) * 4))) {
    for (int k = threadIdx.x; k < k1 - k0; k += blockDim.x) sc[k] = ci[k];
    ci = sc;
  }
  if (int32_t* sr = static_cast<int32_t*>(ar.take((nr + 1) * 4))) {
    if (nr)
      for (int k = threadIdx.x; k <= nr; k += blockDim.x) sr[k] = rp[k];
    rp = sr;
  }
  if (threadIdx.x == 0) {
    // as many lanes as keep the block's threads on one pass over its rows, at most half a row's entries
    int vec = 1;
    while (vec < 32 && 2 * vec * nr <= (int)blockDim.x && 4 * vec * nr <= k1 - k0) vec *= 2;
    if (m.vec) vec = m.vec;
    *d = Rows{r0, r1, k0, vec, rp, ci, val};
  }
}
// align: the blocks' rows of level 0 start at multiples of it
__device__ __forceinline__ void load_amg(const AmgDev& A, AmgRows* d, Arena& ar, int align = 1) {
  for (int l = 0; l < A.nl - 1; ++l) {
    load_rows(A.Qt[l], &d->Qt[l], ar);
    load_rows(A.G[l], &d->G[l], ar, l == 0 ? align : 1);
    load_rows(A.Q[l], &d->Q[l], ar, l == 0 ? align : 1);
  }
  int c0, c1;
  block_range(A.nc, c0, c1, A.nl == 1 ? align : 1);
  const double* inv = A.inv + (size_t)c0 * A.nc;
  const int nv = (c1 - c0) * A.nc;
  if (nv > 0 && nv < (1 << 24))
    if (double* sv = static_cast<double*>(ar.take(nv * 8))) {
      for (int k = threadIdx.x; k < nv; k += blockDim.x) sv[k] = inv[k];
      inv = sv;
    }
  if (threadIdx.x == 0) {
    d->c0 = c0;
    d->c1 = c1;
    d->inv = inv;
  }
}

// out(row, G gx + Q qx) for the block's rows: lane-strided products, then an xor tree, so the order of every
// sum is fixed.
template <int VEC, typename FG, typename FQ, typename FO>
__device__ __forceinline__ void block_rows_vec(const Rows* G, FG gx, const Rows& Q, FQ qx, FO out) {
  const int lane = (int)threadIdx.x % VEC, nr = Q.r1 - Q.r0, r0 = Q.r0;
  for (int b = (int)(threadIdx.x & ~31u) / VEC; b < nr; b += (int)blockDim.x / VEC) {
    const int i = b + (int)(threadIdx.x & 31) / VEC;
    double acc = 0;
    if (i < nr) {
      if (G) {
        const int k1 = G->rp[i + 1] - G->base;
#pragma unroll 4
        for (int k = G->rp[i] - G->base + lane; k < k1; k += VEC) acc += G->val[k] * gx(G->ci[k]);
      }
      const int k1 = Q.rp[i + 1] - Q.base;
#pragma unroll 4
      for (int k = Q.rp[i] - Q.base + lane; k < k1; k += VEC) acc += Q.val[k] * qx(Q.ci[k]);
    }
#pragma unroll
    for (int o = VEC / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (i < nr && lane == 0) out(r0 + i, acc);
  }
}
template <typename FG, typename FQ, typename FO>
__device__ __forceinline__ void block_rows(const Rows* G, FG gx, const Rows& Qs, FQ qx, FO out) {
  const Rows Q = Qs;
  switch (Q.vec) {
    case 1: block_rows_vec<1>(G, gx, Q, qx, out); break;
    case 2: block_rows_vec<2>(G, gx, Q, qx, out); break;
    case 4: block_rows_vec<4>(G, gx, Q, qx, out); break;
    case 8: block_rows_vec<8>(G, gx, Q, qx, out); break;
    case 16: block_rows_vec<16>(G, gx, Q, qx, out); break;
    default: block_rows_vec<32>(G, gx, Q, qx, out);
  }
}
template <typename FQ, typename FO>
__device__ __forceinline__ void block_rows(const Rows& Q, FQ qx, FO out) {
  block_rows(static_cast<const Rows*>(nullptr), [](int) { return 0.0; }, Q, qx, out);
}
// out(row, (inv b)_row) for the block's rows of the dense inverse, a warp per row
template <typename FO>
__device__ __forceinline__ void block_dense(const AmgRows& R, int n, const double* b, FO out) {
  const int lane = threadIdx.x & 31;
  for (int i = threadIdx.x >> 5; i < R.c1 - R.c0; i += blockDim.x >> 5) {
    double s = 0;
#pragma unroll 4
    for (int k = lane; k < n; k += 32) s += R.inv[(size_t)i * n + k] * b[k];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out(R.c0 + i, s);
  }
}

// The V-cycle below level 0 and its way up (two levels or more): b[1] = Q_0^T r is complete at a barrier;
// out(row, z) receives the rows of z = G_0 r + Q_0 x_1 (not followed by a barrier).  False when a barrier gave
// up.
template <typename Bar, typename FR, typename FO>
__device__ __forceinline__ bool amg_cycle(const AmgDev& A, const AmgRows& R, Bar& bar, FR r, FO out) {
  for (int l = 1; l < A.nl - 1; ++l) {
    const double* bl = A.b[l];
    double* bn = A.b[l + 1];
    block_rows(R.Qt[l], [&](int c) { return bl[c]; }, [&](int row, double v) { bn[row] = v; });
    if (!bar.wait()) return false;
  }
  double* xc = A.x[A.nl - 1];
  block_dense(R, A.nc, A.b[A.nl - 1], [&](int row, double v) { xc[row] = v; });
  if (!bar.wait()) return false;
  for (int l = A.nl - 2; l >= 1; --l) {
    const double *bl = A.b[l], *xn = A.x[l + 1];
    double* xl = A.x[l];
    block_rows(&R.G[l], [&](int c) { return bl[c]; }, R.Q[l], [&](int c) { return xn[c]; },
               [&](int row, double v) { xl[row] = v; });
    if (!bar.wait()) return false;
  }
  const double* x1 = A.x[1];
  block_rows(&R.G[0], r, R.Q[0], [&](int c) { return x1[c]; }, out);
  return true;
}

// Blocks and threads of such a launch for n elements; cluster: one cluster of `blocks`.
struct PhaseShape {
  int blocks, threads;
  bool cluster;
};
// A cluster's barrier is the cheaper one, but its 8 SMs have a twentieth of the FP64 rate.  Fourier solves of 2D
// cells, cluster against grid: 600 elements 2.73 and 3.35 ms, 1,100 3.31 and 3.59, 1,500 3.97 and 3.95, 2,000 4.09 and
// 3.46, 8,000 4.88 and 3.61; of a 3D one with 2,000, 16.8 and 15.5.
//
// A cooperative launch waits until all its blocks fit and then holds their room for the whole solve, while other
// streams' kernels wait for theirs.  So a block takes no more than a third of an SM: 256 threads of 80 registers
// and 69 KB.  With 512 threads of 128 registers and 200 KB a solve held every SM: four streams of solves of 8,000 triangles
// x 60 x 48 beside one that repeats Fourier solves of 60,000 went from 189 to 6 a second (129 now; with
// Fourier solves of 4-5 us launches 138, beside a fifth of the Fourier solves), four streams of Fourier solves of 8,000
// from 492 a second to 274 (1,075 now), of 60,000 from 234 to 162 (357 now).  Alone, Fourier solves of
// 60,000 triangles take 7.3 ms for the 6.2 of a whole-SM block (half an SM 6.8, a quarter 8.2), of 8,000 3.55 for 3.7.
constexpr int64_t kClusterElems = 1536;
inline PhaseShape phase_shape(int64_t n, int num_sms) {
  if (n <= kClusterElems) return {8, ClusterBarrier::kThreads, true};
  return {num_sms, GridBarrier::kThreads, false};
}
// Launch a kernel over the shape's blocks, `smem` of `max_smem` bytes of shared memory to each.
template <typename Params>
cudaError_t phase_launch(const PhaseShape& ps, void (*kern)(Params), const Params& p, int smem, int max_smem,
                         cudaStream_t st) {
  if (max_smem > 0) {
    // the limit is the kernel's, shared by every plan and thread: always the largest, so that no launch lowers it
    // under another's
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.dynamicSmemBytes = smem;
  cfg.gridDim = dim3(ps.blocks);
  cfg.blockDim = dim3(ps.threads);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  if (ps.cluster) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ps.blocks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  } else {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, p);
}

}  // namespace obte
