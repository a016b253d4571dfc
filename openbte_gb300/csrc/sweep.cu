// Batched upwind transport sweep for sm_103a.
//
// One CTA = one direction q x one chunk of KV mean free paths.  The CTA walks the direction's elements level
// by level (longest-path layers of the upwind DAG with periodic inflow cut, split into units); within a
// unit every thread takes elements tid, tid + threads, ... and computes the chunk's MFPs of each:
//
//   T_mq[c] = (b[c] + L_m (p[c] - sum_in g_f T_up,m)) / (1 + L_m D_q[c])
//
// the row of A_mq T = B of openbte/bte.py:183-218 for an element whose upwind neighbours are known;
// b = DeltaT + heat source, p = perturbation minus the wall inflow g_w T_B (openbte/bte.py:200,211-214).
//
// T_up lives in a ring of shared-memory rows, one per live upstream element and one column per MFP.  Extra
// rows: a zero row for absent faces, a trash row for elements nobody reads, and one bank of rows per staged
// unit for the inflow across cut periodic faces, so inflow across a cut face is an ordinary row read and
// the ring does not grow with the number of periodic sources (3D meshes have thousands per direction).
// The MFP loop is branch-free; per-MFP outputs (periodic source, wall re-emission, contact) are read back from
// the ring while the next unit runs.
//
// Data movement: everything a unit reads arrives in its stage of shared memory by TMA bulk copies
// (cp.async.bulk + mbarrier), `nbuf` units ahead: the unit's records, its list of outputs, its (b, p) values, its
// periodic inflow rows (gathered per sweep by
// sweep_prep_kernel, already in the table's precision and row layout) and, in FP64, its rows of the gain
// table.  The header carries the source addresses of the unit nbuf further, so the loop reads no global
// metadata.  T never goes to HBM.  Reductions of openbte/bte.py:222-243 are register accumulations over the
// MFPs followed by one FP64 atomic per element (DeltaT', T_B', J); K and S are sums of one thread per MFP.
// Every mbarrier wait is bounded; on timeout the thread raises the device error word and skips the unit,
// and the CTA waits (bounded) for its copies in flight and leaves after the next block-wide barrier.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <numeric>

#include "grid.cuh"

namespace obte {

static constexpr int kMaxThreads = 128;   // threads per CTA at most
static constexpr int kBaseUnit = 128;     // elements per unit of the base layout
static constexpr int kMaxUnit = 1023;     // of any layout (counts of a header have ten bits)

// ---- packed element records -------------------------------------------------------
// 32-bit words, ring rows as 16-bit halves in units of 16 bytes (ring_field):
//   w0 cell | w1 so, s0 | w2 s1, s2 | w3 s3 | the reals c0 .. c(NF-1), D | padding to 16 B
// so = output row, s* = inflow rows.  NF = the most cell and periodic inflow
// faces of an element (Schedule::n_up): a convex cell has at least one outflow face, so triangles and squares
// need two rows, tetrahedra three, not one per side.  32 B (FP32) / 48 B (FP64), tetrahedra 32 B / 64 B.  Leaving
// out the rows that every element read as zero, with the rows' bank classes (schedule.cpp), took the 60k-triangle
// sweep (100 x 96, FP32) from 1,430 to 1,167 us and 5 of 7 spilled words from its element loop.
// A unit's static data: its record block (header, records), followed by its output block:
//   header 0: elements | (values start one pair into their window) << 16, first position, periodic outputs |
//             wall and contact outputs << 10 | contact outputs << 20, then of unit u + nbuf: bank rows | size of its
//             output block << 16
//   header 1: of unit u + nbuf: record block (kBlkUnit bytes) and value (16 bytes) sources, their sizes (16-byte units,
//             block | values << 16), its first bank row among all units' rows
//   outputs:  periodic sources (int2: source slot, row; padded to 16 B), wall / contact entries (int4: row | entry
//             in the second order of the contact sums << 20, count | first of the unit's wall entries << 3 | wall entries of the unit << 16, contact entry, first
//             wall entry overall; those with a contact entry first, in the order of their sums), wall entries (4 reals: area vector / volume, 1 / (-sum_mq min(sigma . w, 0))),
//             their wall indices
__host__ __device__ constexpr int rec_words(int real_bytes, int nf) {
  return ((4 + (nf + 1) * (real_bytes / 4)) + 3) & ~3;
}
template <typename Real, int NF> struct Rec {
  static constexpr int CSTEP = sizeof(Real) / 4, COEF = 4, D = COEF + NF * CSTEP;
  static constexpr int W = rec_words(sizeof(Real), NF);
};
static constexpr int kHeader = 32;   // bytes

// 16-bit row reference: byte offset of the row's first 16 bytes in the ring, over 16.  A lane reads a 32-byte
// row as two 16-byte halves; eight lanes (128 bytes) are served per pass, and with the halves in plain
// order all first halves would share 4 of the 8 16-byte bank groups.  Rows whose index has bit 2 set keep
// their halves swapped, so eight consecutive rows' first halves cover all the banks (60k-triangle cell,
// random row order: 9.0 -> 7.0 passes per 32-lane load); with rows chosen by their class mod 8 (schedule.cpp) 4.7;
// 3.6 would be conflict-free.
__host__ __device__ constexpr int ring_field(int row, int row_bytes) {
  return row_bytes == 32 ? 2 * row + ((row >> 2) & 1) : row;
}

// special-element table
//   si: xk wout contact nwall w0 w1 w2 pad     (8 ints)
//   sr: wc0 wc1 wc2 pad                          (4 reals)
static constexpr int SI = 8, SR = 4;

// Level units: each level of direction q split into runs of at most `cap` elements, and cut so that no unit
// holds more than kUnitPf cut periodic inflow faces or kUnitSx output entries.  The stages and the periodic
// banks of the ring are sized by the largest unit; without the caps the few units on the periodic
// boundaries (up to ~110 cut faces and outputs each on the 60k-triangle cell) set them, and the extra ~5 KB
// cost a CTA per SM.  A cap only applies when at most 1 % of the uncapped units exceed it: where most units
// are over it (the pixel model, where every element has reflecting-wall outputs) it would split every unit
// in two and lengthen every chain instead.
constexpr int kUnitPf = 48;
constexpr int kUnitSx = 64;
struct Units {
  std::vector<int32_t> ptr;   // per direction: n[q] + 1 positions (relative to the direction)
  std::vector<int64_t> off;   // [n_dir] first entry of direction q in ptr
  std::vector<int32_t> n;     // [n_dir] units of direction q
};

static void build_units_capped(const Schedule& s, int cap, int cap_pf, int cap_sx, Units& un, int64_t* over_pf,
                               int64_t* over_sx) {
  // directions in parallel into their own lists, concatenated in direction order
  std::vector<std::vector<int32_t>> per(s.n_dir);
  std::vector<int64_t> opf(s.n_dir, 0), osx(s.n_dir, 0);
  parallel_tasks(s.n_dir, [&](int64_t qq) {
    const int q = (int)qq;
    std::vector<int32_t>& ptr = per[q];
    const int32_t* lp = s.lev_ptr.data() + s.lev_off[q];
    ptr.push_back(0);
    for (int Lv = 0; Lv < s.nlev[q]; ++Lv) {
      int cnt = 0, npf = 0, nsx = 0;
      auto close = [&](int32_t end) {
        ptr.push_back(end);
        if (npf > kUnitPf) ++opf[q];
        if (nsx > kUnitSx) ++osx[q];
        cnt = npf = nsx = 0;
      };
      for (int32_t pos = lp[Lv]; pos < lp[Lv + 1]; ++pos) {
        const int info = s.info[(size_t)q * s.n + pos], pf = info & 7, sx = info & 24 ? 1 : 0;
        if (cnt > 0 && (cnt == cap || npf + pf > cap_pf || nsx + sx > cap_sx)) close(pos);
        ++cnt;
        npf += pf;
        nsx += sx;
      }
      if (cnt > 0) close(lp[Lv + 1]);
    }
  });
  un.ptr.clear();
  un.off.assign(s.n_dir, 0);
  un.n.assign(s.n_dir, 0);
  size_t total = 0;
  for (int q = 0; q < s.n_dir; ++q) total += per[q].size();
  un.ptr.reserve(total);
  for (int q = 0; q < s.n_dir; ++q) {
    un.off[q] = (int64_t)un.ptr.size();
    un.n[q] = (int32_t)per[q].size() - 1;
    un.ptr.insert(un.ptr.end(), per[q].begin(), per[q].end());
  }
  if (over_pf) *over_pf = std::accumulate(opf.begin(), opf.end(), (int64_t)0);
  if (over_sx) *over_sx = std::accumulate(osx.begin(), osx.end(), (int64_t)0);
}

static void build_units(const Schedule& s, int cap, Units& un) {
  constexpr int kNone = 1 << 30;
  int64_t over_pf = 0, over_sx = 0;
  build_units_capped(s, cap, kNone, kNone, un, &over_pf, &over_sx);
  const int64_t units = (int64_t)un.ptr.size() - s.n_dir;
  const int cap_pf = over_pf * 100 <= units ? kUnitPf : kNone;
  const int cap_sx = over_sx * 100 <= units ? kUnitSx : kNone;
  if (cap_pf != kNone || cap_sx != kNone) build_units_capped(s, cap, cap_pf, cap_sx, un, nullptr, nullptr);
}
// What the layout of the staged units has to hold.
struct UnitStats {
  int emax = 0;       // most cut inflow faces in one unit
  int unit_wo = 0;    // most wall entries
  int unit_sx = 0;    // most elements with outputs
  int unit_el = 0;    // most elements
  int unit_out = 0;   // largest output block
  int units = 0;      // most units of one direction
  bool bad_wo = false;
};

static inline bool has_outputs(const Schedule& s, size_t it) {
  return s.xk[it] >= 0 || s.wout[it] != 0 || s.contact[it] >= 0;
}

// Output block of a unit: nx periodic sources, nw wall / contact entries, nwo wall entries.
static inline int out_bytes(int nx, int nw, int nwo, int real_bytes) {
  return ((nx * 8 + 15) & ~15) + nw * 16 + nwo * 4 * real_bytes + ((nwo * 4 + 15) & ~15);
}

// Counts of every unit (cut faces, wall entries, periodic outputs, wall / contact outputs), in parallel over
// directions: cnt[4 u + k] for unit u of all directions in order (unit_base[q] + unit of the direction).
static UnitStats count_units(const Schedule& s, const Units& un, int real_bytes, std::vector<int64_t>& unit_base,
                             std::vector<int32_t>& cnt) {
  unit_base.assign(s.n_dir + 1, 0);
  for (int q = 0; q < s.n_dir; ++q) unit_base[q + 1] = unit_base[q] + un.n[q];
  cnt.assign((size_t)unit_base[s.n_dir] * 4, 0);
  std::vector<UnitStats> per(s.n_dir);
  parallel_tasks(s.n_dir, [&](int64_t q) {
    const int32_t* up = un.ptr.data() + un.off[q];
    UnitStats& st = per[q];
    st.units = un.n[q];
    int64_t wo = 0;
    for (int u = 0; u < un.n[q]; ++u) {
      int npf = 0, nwo = 0, nsx = 0, nx = 0, nw = 0;
      for (int32_t pos = up[u]; pos < up[u + 1]; ++pos) {
        const int info = s.info[(size_t)q * s.n + pos];
        if (info == 0) continue;
        npf += info & 7;
        nwo += info >> 5;
        nsx += info & 24 ? 1 : 0;
        nx += (info >> 3) & 1;
        nw += (info >> 4) & 1;
      }
      int32_t* c = cnt.data() + 4 * (size_t)(unit_base[q] + u);
      c[0] = npf; c[1] = nwo; c[2] = nx; c[3] = nw;
      st.unit_out = std::max(st.unit_out, out_bytes(nx, nw, nwo, real_bytes));
      wo += nwo;
      st.emax = std::max(st.emax, npf);
      st.unit_wo = std::max(st.unit_wo, nwo);
      st.unit_sx = std::max(st.unit_sx, nsx);
      st.unit_el = std::max(st.unit_el, (int)(up[u + 1] - up[u]));
    }
    st.bad_wo = wo != s.wo_off[q + 1] - s.wo_off[q];
  });
  UnitStats t;
  for (const UnitStats& p : per) {
    t.emax = std::max(t.emax, p.emax);
    t.unit_wo = std::max(t.unit_wo, p.unit_wo);
    t.unit_sx = std::max(t.unit_sx, p.unit_sx);
    t.unit_el = std::max(t.unit_el, p.unit_el);
    t.unit_out = std::max(t.unit_out, p.unit_out);
    t.units = std::max(t.units, p.units);
    t.bad_wo = t.bad_wo || p.bad_wo;
  }
  return t;
}

// ---- shared memory of a CTA (bytes) --------------------------------------------------
//   [0, 64) mbarriers | [64, 68) first unit that timed out | [96, ...) sigma [3][KV]
//   | [kRingOff, ...) ring | nbuf stages of (record block | values | gain rows) | nbuf + 1 output blocks
// (a unit's outputs are written while the next unit runs, so its output block outlives its stage)
static constexpr int kMaxBuf = 8;
static constexpr int kFailOff = 64, kSigOff = 96, kRingOff = 384;
static_assert(kSigOff + 3 * 32 <= kRingOff, "sigma of 32-byte rows");
static constexpr size_t kSmemPerSM = 233472, kSmemPerCta = 1024;   // capacity, reserved per CTA

struct Layout {
  int KV = 0;         // MFPs per thread and per CTA
  int threads = 0;    // of a plain sweep
  int final_threads = kMaxThreads;   // of an output pass
  int nbuf = 2;
  int emax = 0;       // rows of one periodic bank
  int prow0 = 0;      // first bank row
  int rows = 0;       // ring rows
  int blk = 0, val = 0, gain = 0;   // bytes of a stage's parts
  int out = 0;                      // bytes of an output block
  size_t smem = 0;
  int stage() const { return blk + val + gain; }
};

template <typename Real>
static Layout make_layout(const Schedule& s, const UnitStats& st, const Layout& shape, int nbuf) {
  Layout l = shape;
  const int row_bytes = l.KV * (int)sizeof(Real), al = row_bytes == 32 ? 7 : 0;   // swapped halves: runs of 8 rows
  const int over = std::max(st.unit_el, l.final_threads);   // every thread reads a record, its own or a stale one
  l.nbuf = nbuf;
  l.emax = (st.emax + al) & ~al;
  l.prow0 = (s.max_slots + 2 + al) & ~al;
  l.rows = l.prow0 + nbuf * l.emax;
  l.blk = kHeader + over * rec_words(sizeof(Real), s.n_up) * 4;
  l.val = ((over + 2) * 2 * (int)sizeof(Real) + 15) & ~15;
  l.gain = sizeof(Real) == 8 ? over * row_bytes : 0;
  l.out = st.unit_out;
  l.smem = (size_t)kRingOff + (size_t)l.rows * row_bytes + (size_t)nbuf * l.stage() + (size_t)(nbuf + 1) * l.out;
  return l;
}

// CTAs that share an SM: by shared memory (handed out in 128-byte pieces: 45,600 B a CTA leave room for four, not five,
// and took the 60k-triangle benchmark cell's sweep from 1.43 to 1.73 ms) and by registers (launch bounds of the kernel).
template <typename Real>
static int resident(const Layout& l) {
  const int by_regs = (sizeof(Real) == 4 && l.KV == 8 ? 5 : 4) * kMaxThreads / l.threads;
  return (int)std::min<size_t>((size_t)std::min(by_regs, 32), kSmemPerSM / (((l.smem + 127) & ~(size_t)127) + kSmemPerCta));
}

// Alignment and unit of a static block's offset: 32 bits reach 256 GB of blocks.  (Of the values, 16 bytes an item in
// FP64, 32 bits of 16-byte units reach more items than their blocks leave room for.)
constexpr int kBlkUnit = 64;

struct Packed {
  Layout lay;
  RawVec<int32_t> blk;                  // static blocks of all units, direction by direction
  RawVec<int32_t> cellmap, spec;        // one entry per item
  RawVec<double> P;
  std::vector<int32_t> si;
  std::vector<double> sr;
  // 8 ints per unit: elements | odd << 16, first position, first bank row, bank rows | output block's size << 16;
  // record block (kBlkUnit bytes) and value offsets (16-byte units), their sizes (16-byte units, block | values << 16),
  // periodic outputs | wall and contact outputs << 16
  std::vector<int32_t> desc;
  std::vector<int32_t> pfe;             // 4 ints per bank row: source slot, its unit's first row among all units'
                                        // rows, rows of its unit, its row in the unit | swapped halves << 31
  int64_t n_pf = 0;
};

// The places of each contact entry of direction q in the sums K and S of an output pass, by entry (relative to the
// direction's first).  The sums are in the sweep's precision, so their order is part of the result: unit by unit
// of the base layout, in a unit the 32-element groups with fewer contact elements first, elements of a group in order;
// of groups with equally many the later one first (`first`) or the earlier one first (`second`): K and S of an FP32
// pass are the means of the two sums.  That is how one FP32 shared-memory atomic per element and MFP arrives from a CTA with one
// element of a base unit to a thread: a group with fewer of them is through first, and which of two equal ones is, is
// left to chance.  On 8,000 triangles x 60 x 48 at least 2,876 of 2,880 sums of such atomics have these bits in one of the
// orders (2,858 in position order); their mean is 0.6e-9 to 1.1e-9 off K of a run of the atomics, two runs
// 0.5e-9 to 1.5e-9 off each other, and sums in FP64 1e-7.  The atomics also cost time: the resident solve of 60,000
// triangles x 100 x 96 went from 46.1 to 45.0 ms without them, 8,000 x 60 x 48 from 11.95 to 11.83 ms.
static void contact_order(const Schedule& s, const Units& base, int q, std::vector<int32_t>& first,
                          std::vector<int32_t>& second) {
  struct Entry { int32_t unit, count, group, pos; };
  std::vector<Entry> e;
  const int32_t* up = base.ptr.data() + base.off[q];
  for (int32_t u = 0, pos = 0; u < base.n[q]; ++u)
    for (; pos < up[u + 1]; ++pos)
      if (s.contact[(size_t)q * s.n + pos] >= 0) e.push_back({u, 0, (pos - up[u]) >> 5, pos});
  for (size_t a = 0, b = 0; a < e.size(); a = b) {
    while (b < e.size() && e[b].unit == e[a].unit && e[b].group == e[a].group) ++b;
    for (size_t k = a; k < b; ++k) e[k].count = (int32_t)(b - a);
  }
  std::vector<int32_t> ord(e.size());
  auto places = [&](bool late, std::vector<int32_t>& place) {
    std::iota(ord.begin(), ord.end(), 0);
    std::sort(ord.begin(), ord.end(), [&](int32_t i, int32_t j) {
      const Entry &x = e[i], &y = e[j];
      if (x.unit != y.unit) return x.unit < y.unit;
      if (x.count != y.count) return x.count < y.count;
      return x.group != y.group ? (x.group > y.group) == late : x.pos < y.pos;
    });
    place.resize(e.size());
    for (size_t k = 0; k < ord.size(); ++k) place[ord[k]] = (int32_t)k;
  };
  places(true, first);
  places(false, second);
}

// base: the units of the base layout
template <typename Real>
static obte_status pack(const Schedule& s, const Units& un, const Units& base, const std::vector<int64_t>& unit_base,
                        const std::vector<int32_t>& cnt, const Layout& lay, Packed& pk) {
  const int W = rec_words(sizeof(Real), s.n_up);
  constexpr int CSTEP = sizeof(Real) / 4, COEF = 4, VB = 2 * sizeof(Real);
  const int row_bytes = lay.KV * (int)sizeof(Real);
  auto field = [&](int row) { return ring_field(row, row_bytes); };
  const int zero_row = s.max_slots, trash_row = s.max_slots + 1;
  pk.lay = lay;
  if (field(lay.rows) >= 65535 || s.x_base[s.n_dir] >= ((int64_t)1 << 32)) {
    set_error("sweep ring rows do not fit 16-bit indices");
    return OBTE_ERR_UNSUPPORTED;
  }
  const int64_t n_units = unit_base[s.n_dir];
  // offsets of every unit: block, bank rows
  std::vector<int64_t> boff(n_units + 1, 0), poff(n_units + 1, 0);
  {
    int64_t u = 0;
    for (int q = 0; q < s.n_dir; ++q) {
      const int32_t* up = un.ptr.data() + un.off[q];
      for (int k = 0; k < un.n[q]; ++k, ++u) {
        const int32_t* c = cnt.data() + 4 * (size_t)u;
        const int64_t bytes = kHeader + (int64_t)(up[k + 1] - up[k]) * W * 4 + out_bytes(c[2], c[3], c[1], sizeof(Real));
        boff[u + 1] = boff[u] + (bytes + kBlkUnit - 1) / kBlkUnit;
        poff[u + 1] = poff[u] + c[0];
      }
    }
  }
  pk.n_pf = poff[n_units];
  const int64_t total = (int64_t)s.n_dir * s.n;
  if (boff[n_units] >= ((int64_t)1 << 32) || pk.n_pf >= ((int64_t)1 << 31) ||
      total / (16 / VB) >= ((int64_t)1 << 32)) {
    set_error("sweep tables too large");
    return OBTE_ERR_UNSUPPORTED;
  }
  pk.blk.resize((size_t)boff[n_units] * (kBlkUnit / 4));   // uninitialised: every word is written below
  pk.desc.assign((size_t)std::max<int64_t>(n_units, 1) * 8, 0);
  pk.pfe.assign((size_t)std::max<int64_t>(pk.n_pf, 1) * 4, 0);
  pk.cellmap.resize(total);
  pk.spec.resize(total);
  pk.P.resize(total);
  // descriptors
  parallel_tasks(s.n_dir, [&](int64_t q) {
    const int32_t* up = un.ptr.data() + un.off[q];
    for (int k = 0; k < un.n[q]; ++k) {
      const int64_t u = unit_base[q] + k;
      const int64_t v0 = ((int64_t)q * s.n + up[k]) * VB, v1 = ((int64_t)q * s.n + up[k + 1]) * VB;
      const int odd = (int)((v0 & 15) / VB);
      int32_t* d = pk.desc.data() + 8 * (size_t)u;
      d[0] = (up[k + 1] - up[k]) | (odd << 16);
      d[1] = up[k];
      d[2] = (int32_t)poff[u];
      const int32_t* c = cnt.data() + 4 * (size_t)u;
      const int out16 = out_bytes(c[2], c[3], c[1], sizeof(Real)) / 16;
      const int rec16 = (kHeader + (up[k + 1] - up[k]) * W * 4) / 16;
      d[3] = (int32_t)(poff[u + 1] - poff[u]) | (out16 << 16);
      d[4] = (int32_t)(uint32_t)boff[u];
      d[5] = (int32_t)(uint32_t)(v0 >> 4);
      d[6] = (int32_t)((uint32_t)rec16 | ((uint32_t)(((v1 + 15) >> 4) - (v0 >> 4)) << 16));
      d[7] = c[2] | (c[3] << 16);
    }
  });
  // special entries (elements with outputs or wall inflow): counted per direction, then every direction fills
  // its own range
  auto is_special = [&](size_t it) {
    if (has_outputs(s, it)) return true;
    for (int f = 0; f < s.nf; ++f)
      if ((int)((uint32_t)s.in_idx[it * s.nf + f] >> ITEM_SHIFT) == ITEM_WALL) return true;
    return false;
  };
  std::vector<int64_t> spec_base(s.n_dir + 1, 0);
  parallel_tasks(s.n_dir, [&](int64_t q) {
    int64_t c = 0;
    for (int64_t pos = 0; pos < s.n; ++pos) c += is_special((size_t)q * s.n + pos) ? 1 : 0;
    spec_base[q + 1] = c;
  });
  for (int q = 0; q < s.n_dir; ++q) spec_base[q + 1] += spec_base[q];
  pk.si.assign((size_t)spec_base[s.n_dir] * SI, 0);
  pk.sr.assign((size_t)spec_base[s.n_dir] * SR, 0.0);
  std::vector<int> dir_err(s.n_dir, 0);   // 1: outputs without a ring slot, 2: more than three wall inflows
  parallel_tasks(s.n_dir, [&](int64_t qq) {
    const int q = (int)qq;
    int64_t nsp = spec_base[q];
    const int32_t* up = un.ptr.data() + un.off[q];
    int32_t wo_run = s.wo_off[q];          // first wall entry of the unit
    std::vector<int32_t> place, place2;    // of the direction's contact entries in their sums
    contact_order(s, base, q, place, place2);
    size_t ce = 0;                         // contact entries before the element
    struct Out { int32_t first, second, w[4]; };
    std::vector<Out> entries;              // the unit's wall / contact entries
    std::vector<int32_t> ranked;
    for (int u = 0; u < un.n[q]; ++u) {
      const int64_t gu = unit_base[q] + u;
      const int n_el = up[u + 1] - up[u], npf = cnt[4 * gu], nwo = cnt[4 * gu + 1], nx = cnt[4 * gu + 2],
                nw = cnt[4 * gu + 3];
      int32_t* head = pk.blk.data() + (size_t)boff[gu] * (kBlkUnit / 4);
      int32_t* recs = head + kHeader / 4;
      int32_t* xo = recs + (size_t)n_el * W;
      int32_t* wo = xo + (((size_t)nx * 2 + 3) & ~(size_t)3);
      int32_t* wg = wo + (size_t)nw * 4;
      entries.clear();
      int n_contact = 0;
      if (nx & 1) xo[2 * nx] = xo[2 * nx + 1] = 0;
      // header: this unit, and the source addresses of the unit nbuf further
      const int32_t* own = pk.desc.data() + 8 * (size_t)gu;
      head[0] = own[0];
      head[1] = own[1];
      head[2] = nx | (nw << 10);             // at most kMaxUnit each
      std::fill(head + 3, head + 8, 0);
      if (u + lay.nbuf < un.n[q]) {
        const int32_t* f = pk.desc.data() + 8 * (size_t)(gu + lay.nbuf);
        head[3] = f[3];
        head[4] = f[4];
        head[5] = f[5];
        head[6] = f[6];
        head[7] = f[2];
      }
      for (int e = 0; e < nwo; ++e) {      // wall geometry
        const int32_t w = s.wo_wall[wo_run + e];
        Real g[4] = {0, 0, 0, 0};
        for (int k = 0; k < s.dim; ++k) g[k] = (Real)s.w_db[(size_t)w * s.dim + k];
        g[3] = s.gbm_sum[w] != 0 ? (Real)(1.0 / (-s.gbm_sum[w])) : Real(0);
        std::memcpy(wg + (size_t)e * 4 * CSTEP, g, sizeof(g));
        wg[(size_t)nwo * 4 * CSTEP + e] = w;
      }
      for (int e = nwo; e & 3; ++e) wg[(size_t)nwo * 4 * CSTEP + e] = 0;
      std::fill(wg + (size_t)nwo * 4 * CSTEP + ((nwo + 3) & ~3), pk.blk.data() + (size_t)boff[gu + 1] * (kBlkUnit / 4), 0);
      int ent = 0;
      const int bank = lay.prow0 + (u % lay.nbuf) * lay.emax;
      for (int32_t pos = up[u]; pos < up[u + 1]; ++pos) {
        const size_t it = (size_t)q * s.n + pos;
        int32_t* r = recs + (size_t)(pos - up[u]) * W;
        const int so = s.slot[it] >= 0 ? s.slot[it] : trash_row;
        r[0] = s.cell[it];
        pk.cellmap[it] = s.cell[it];
        pk.P[it] = s.P[it];
        int32_t si[SI] = {s.xk[it], s.wout[it], s.contact[it], 0, 0, 0, 0, 0};
        double sr[SR] = {0, 0, 0, 0};
        const bool outputs = has_outputs(s, it);
        if (outputs && s.slot[it] < 0) { dir_err[q] = 1; return; }
        bool special = outputs;
        double coef[4] = {0, 0, 0, 0};
        int row_in[4] = {zero_row, zero_row, zero_row, zero_row};
        int k = 0;
        for (int f = 0; f < s.nf; ++f) {
          const int32_t code = s.in_idx[it * s.nf + f];
          const int kind = (int)((uint32_t)code >> ITEM_SHIFT);
          const int32_t idx = code & ITEM_MASK;
          const double g = s.in_coef[it * s.nf + f];
          if (kind == ITEM_CELL || kind == ITEM_PERIODIC) {
            if (kind == ITEM_CELL) {
              row_in[k] = idx;
            } else {
              row_in[k] = bank + ent;
              int32_t* pe = pk.pfe.data() + 4 * (size_t)(poff[gu] + ent);
              pe[0] = (int32_t)(uint32_t)(s.x_base[q] + idx);
              pe[1] = (int32_t)poff[gu];
              pe[2] = npf;
              pe[3] = (int32_t)((uint32_t)ent | (uint32_t)(row_bytes == 32 ? ((bank + ent) >> 2) & 1 : 0) << 31);
              ++ent;
            }
            coef[k] = g;
            ++k;
          } else if (kind == ITEM_WALL) {
            if (si[3] >= 3) { dir_err[q] = 2; return; }
            si[4 + si[3]] = idx;
            sr[si[3]] = g;
            si[3]++;
            special = true;
          }
        }
        if (s.xk[it] >= 0) {
          xo[0] = (int32_t)(uint32_t)(s.x_base[q] + s.xk[it]);
          xo[1] = field(so) << 4;
          xo += 2;
        }
        r[3] = field(row_in[3]);
        if (s.wout[it] != 0 || s.contact[it] >= 0) {
          const bool contact = s.contact[it] >= 0;
          entries.push_back({contact ? place[ce] : INT_MAX, contact ? place2[ce] : INT_MAX,
                             {field(so) << 4,
                              (s.wout[it] ? (((s.wout[it] >> 3) - wo_run) << 3) | (s.wout[it] & 7) : 0) | (nwo << 16),
                              s.contact[it], s.wout[it] >> 3}});
          if (contact) {
            ++ce;
            ++n_contact;
          }
        }
        r[1] = field(so) | (field(row_in[0]) << 16);
        r[2] = field(row_in[1]) | (field(row_in[2]) << 16);
        if (special) {
          pk.spec[it] = (int32_t)nsp;
          std::copy(si, si + SI, pk.si.begin() + (size_t)nsp * SI);
          std::copy(sr, sr + SR, pk.sr.begin() + (size_t)nsp * SR);
          ++nsp;
        } else {
          pk.spec[it] = -1;
        }
        for (int f = 0; f < s.n_up; ++f) {
          const Real v = (Real)coef[f];
          std::memcpy(&r[COEF + f * CSTEP], &v, sizeof(Real));
        }
        const Real dv = (Real)s.D[it];
        std::memcpy(&r[COEF + s.n_up * CSTEP], &dv, sizeof(Real));
        for (int wd = COEF + (s.n_up + 1) * CSTEP; wd < W; ++wd) r[wd] = 0;   // padding to 16 bytes
      }
      // contact entries in the first order of their sums, then the others; with the i-th, the one that is i-th in the
      // second order
      std::stable_sort(entries.begin(), entries.end(), [](const Out& a, const Out& b) { return a.first < b.first; });
      ranked.resize(n_contact);
      std::iota(ranked.begin(), ranked.end(), 0);
      std::sort(ranked.begin(), ranked.end(),
                [&](int32_t a, int32_t b) { return entries[a].second < entries[b].second; });
      for (int i = 0; i < n_contact; ++i) entries[i].w[0] |= ranked[i] << 20;
      for (const Out& e : entries) wo = std::copy(e.w, e.w + 4, wo);
      head[2] |= n_contact << 20;
      wo_run += nwo;
    }
  });
  for (int q = 0; q < s.n_dir; ++q) {
    if (dir_err[q] == 1) { set_error("element with per-MFP outputs has no ring slot"); return OBTE_ERR_BAD_ARG; }
    if (dir_err[q] == 2) {
      set_error("more than three wall inflow faces on one element");
      return OBTE_ERR_UNSUPPORTED;
    }
  }
  if (pk.si.empty()) {
    pk.si.assign(SI, 0);
    pk.sr.assign(SR, 0.0);
  }
  return OBTE_OK;
}

// ---- PTX helpers (TMA bulk copy + mbarrier) -----------------------------------------
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void tma_load_1d(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Default cap on the polls of one mbarrier wait (each poll may suspend the thread for a while before it
// returns), far above any copy's latency; a wait that reaches it gives up and reports a timeout.
constexpr int kWaitPolls = 1 << 22;
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, unsigned parity, int limit = kWaitPolls) {
  for (int i = 0; i < limit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
// ---- double-float arithmetic (the output pass of the FP32+refine solve) ----------------------------
// A value is an unevaluated pair hi + lo of FP32 numbers (~44 significant bits), computed on the FP32 pipe
// with error-free transformations: Knuth's two-sum, the FMA two-product (Dekker 1971; Ogita, Rump and
// Oishi 2005), here on two MFPs at once with Blackwell's packed FP32x2 instructions.  The intrinsics round
// every operation and are never contracted, which these transformations rely on.  In the ring and the
// per-thread registers a pair lives in the 8 bytes of a double: low word hi, high word lo.
struct df2 {
  float2 h, l;   // hi and lo parts of two MFPs' values
};
__device__ __forceinline__ float2 f2neg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 f2sub(float2 a, float2 b) { return __fadd2_rn(a, f2neg(b)); }
__device__ __forceinline__ df2 two_sum2(float2 a, float2 b) {
  const float2 s = __fadd2_rn(a, b);
  const float2 bb = f2sub(s, a);
  return {s, __fadd2_rn(f2sub(a, f2sub(s, bb)), f2sub(b, bb))};
}
__device__ __forceinline__ df2 fast_two_sum2(float2 a, float2 b) {   // |a| >= |b| (or a exact)
  const float2 s = __fadd2_rn(a, b);
  return {s, f2sub(b, f2sub(s, a))};
}
__device__ __forceinline__ df2 dadd2(df2 a, df2 b) {
  const df2 s = two_sum2(a.h, b.h);
  return fast_two_sum2(s.h, __fadd2_rn(s.l, __fadd2_rn(a.l, b.l)));
}
__device__ __forceinline__ df2 dneg2(df2 a) { return {f2neg(a.h), f2neg(a.l)}; }
__device__ __forceinline__ df2 dmul2(df2 a, df2 b) {
  const float2 p = __fmul2_rn(a.h, b.h);
  float2 e = __ffma2_rn(a.h, b.h, f2neg(p));
  e = __ffma2_rn(a.h, b.l, e);
  e = __ffma2_rn(a.l, b.h, e);
  return fast_two_sum2(p, e);
}
// a / b: an FP32 reciprocal seed y, the quotient q = a y and one correction by the residual a - q b
__device__ __forceinline__ df2 ddiv2(df2 a, df2 b) {
  const float2 y = make_float2(__fdividef(1.0f, b.h.x), __fdividef(1.0f, b.h.y));
  const float2 q = __fmul2_rn(a.h, y);
  float2 r = __ffma2_rn(f2neg(q), b.h, a.h);
  r = __fadd2_rn(r, a.l);
  r = __ffma2_rn(f2neg(q), b.l, r);
  return fast_two_sum2(q, __fmul2_rn(r, y));
}
// split a double into hi + lo (FP64 pipe: two conversions and a subtraction)
__device__ __forceinline__ float2 dsplit(double d) {
  const float h = __double2float_rn(d);
  return make_float2(h, __double2float_rn(d - (double)h));
}
__device__ __forceinline__ df2 dbcast(double d) {   // the same value in both lanes
  const float2 s = dsplit(d);
  return {make_float2(s.x, s.x), make_float2(s.y, s.y)};
}
__device__ __forceinline__ double dpack(float h, float l) { return __hiloint2double(__float_as_int(l), __float_as_int(h)); }
__device__ __forceinline__ double dpack_split(double d) { const float2 s = dsplit(d); return dpack(s.x, s.y); }
__device__ __forceinline__ float dpack_hi(double x) { return __int_as_float(__double2loint(x)); }
__device__ __forceinline__ float dpack_lo(double x) { return __int_as_float(__double2hiint(x)); }
__device__ __forceinline__ double dpack_value(double x) { return (double)dpack_hi(x) + (double)dpack_lo(x); }
__device__ __forceinline__ df2 dunpack2(double a, double b) {   // two packed pairs -> lanes x, y
  return {make_float2(dpack_hi(a), dpack_hi(b)), make_float2(dpack_lo(a), dpack_lo(b))};
}
__device__ __forceinline__ double widen(double f) { return f; }

// ---- per-sweep inputs -------------------------------------------------------------------
// One launch: the (b, p) values of every item, b = DeltaT + h, p = P - sum_walls g_w T_B; the periodic inflow
// rows of every unit (one warp per row and state: coalesced reads of the source's MFPs, written chunk by
// chunk in the table's precision and row layout, so that a unit's rows are one bulk copy); and zeros for the
// sums the sweep adds to.
template <typename Real>
struct PrepParams {
  const int32_t* __restrict__ cellmap;
  const double* __restrict__ Pq;
  const int32_t* __restrict__ spec;
  const int32_t* __restrict__ si;
  const Real* __restrict__ sr;
  const double* __restrict__ hs;      // heat source, or null
  const double* __restrict__ u_in;
  int64_t n, nd, total;
  int with_src;
  Real* __restrict__ vals;
  const int32_t* __restrict__ pfe;
  int64_t n_pf;
  int n_mfp, m_row;                    // MFPs, MFPs rounded up to whole chunks
  int batch;
  int64_t batch_stride;                // states of a batched sweep (rows only: they agree on DeltaT and T_B)
  int64_t row_stride;                  // reals between two states' rows
  Real* __restrict__ xrow;
  double *zero0, *zero1;               // sums to clear
  int64_t nz0, nz1;
  int row_blocks;                      // blocks that gather rows (the others: values and zeros)
};

template <typename Real, int MC, bool DF>
__global__ void __launch_bounds__(256, 8) sweep_prep_kernel(const __grid_constant__ PrepParams<Real> p) {
  if ((int)blockIdx.x < p.row_blocks) {
    constexpr bool kWide = MC * sizeof(Real) == 32;
    constexpr int U = 4;                 // loads in flight per lane, over the pieces of 32 MFPs of consecutive rows
    const double* __restrict__ X = p.u_in + p.n + p.nd;
    const int lane = threadIdx.x & 31;
    const int np = (p.m_row + 31) >> 5;  // pieces of a row
    const int64_t nw = (int64_t)p.row_blocks * (blockDim.x >> 5), total = p.n_pf * p.batch * np;
    const int4* __restrict__ pfe = reinterpret_cast<const int4*>(p.pfe);
    // the entries of a row are read again for its stores (an L1 hit): kept, they would cost a third of the warps
    for (int64_t f = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * U; f < total; f += nw * U) {
      const int64_t w0 = f / np;
      const int piece0 = (int)(f - w0 * np), left = (int)min((int64_t)U, total - f);
      double v[U];
      int64_t w = w0;
      int piece = piece0;
#pragma unroll
      for (int k = 0; k < U; ++k) {
        v[k] = 0.0;
        const int m = lane + 32 * piece;
        if (k < left && m < p.n_mfp) {
          const int64_t t = p.batch > 1 ? w / p.n_pf : 0;
          v[k] = X[t * p.batch_stride + (int64_t)(unsigned)pfe[w - t * p.n_pf].x * p.n_mfp + m];
        }
        if (++piece == np) { piece = 0; ++w; }
      }
      w = w0;
      piece = piece0;
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const int m = lane + 32 * piece;
        if (k < left && m < p.m_row) {
          const int64_t t = p.batch > 1 ? w / p.n_pf : 0;
          const int4 e = pfe[w - t * p.n_pf];
          const int flip = kWide && e.w < 0 ? MC / 2 : 0;
          Real r = (Real)v[k];
          if constexpr (DF) r = dpack_split((double)r);
          const int64_t row = (int64_t)e.y * (p.m_row / MC) + (e.w & 0x7fffffff) + (int64_t)(m / MC) * e.z;
          p.xrow[t * p.row_stride + row * MC + ((m % MC) ^ flip)] = r;
        }
        if (++piece == np) { piece = 0; ++w; }
      }
    }
    return;
  }
  const int64_t t0 = (int64_t)(blockIdx.x - p.row_blocks) * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)(gridDim.x - p.row_blocks) * blockDim.x;
  const double* __restrict__ TB = p.u_in + p.n;
  for (int64_t it = t0; it < p.total; it += stride) {
    const int c = p.cellmap[it];
    double b = p.u_in[c];
    double pp = 0;
    if (p.with_src) {
      if (p.hs) b += p.hs[c];
      pp = p.Pq[it];
    }
    const int sp = p.spec[it];
    if (sp >= 0) {
      const int32_t* s = p.si + (int64_t)sp * SI;
      const Real* r = p.sr + (int64_t)sp * SR;
      for (int k = 0; k < s[3]; ++k) pp -= (double)r[k] * TB[s[4 + k]];
    }
    p.vals[2 * it] = (Real)b;
    p.vals[2 * it + 1] = (Real)pp;
  }
  for (int64_t i = t0; i < p.nz0; i += stride) p.zero0[i] = 0.0;
  for (int64_t i = t0; i < p.nz1; i += stride) p.zero1[i] = 0.0;
}

template <typename Real>
struct SweepParams {
  int64_t n;
  int64_t nd;
  int n_mfp, n_dir, ds, m_pad;
  int n_chunks;            // chunks of KV MFPs per direction
  int zero_row, prow0;     // ring rows: zero row, first periodic bank row
  int emax;                // rows per periodic bank
  int nbuf;                // units staged at once
  int stage0, stage, val_off, gain_off;   // first stage, bytes of a stage, its values and gain rows
  int out0, out;           // first output block, bytes of one
  const int32_t* __restrict__ blk;        // static blocks
  const int32_t* __restrict__ desc;       // unit descriptors (8 ints), directions in order
  const int64_t* __restrict__ unit_base;  // [n_dir + 1]
  const Real* __restrict__ vals;
  const Real* __restrict__ xrow;          // periodic inflow rows: [unit][chunk][row][KV]
  const Real* __restrict__ mfp;    // [m_pad]
  const Real* __restrict__ tco;    // [n_dir * m_pad]
  const Real* __restrict__ sig;    // [n_dir * m_pad * ds]
  const Real* __restrict__ kcoef;  // [n_ce * m_pad]
  const Real* __restrict__ scoef;  // [n_ce]
  double* __restrict__ u_out;
  double* __restrict__ Jraw;
  double* __restrict__ K;
  double* __restrict__ S_out;
  int* __restrict__ err;
  const double* __restrict__ gain;   // FP64: mfp / (1 + mfp D) [n_dir][n_chunks][n][KV], or null: divide
  float* __restrict__ Xs;   // final pass only: per-ordinate temperatures [n_dir][n][n_mfp], or null
  int xs_add;               // 1: add this pass's temperatures to Xs (the pass at a correction d)
  double* __restrict__ Xd;  // the same in FP64 (FP64 sweeps of obte_bte_sweep_fields), or null
  const int32_t* __restrict__ cta_map;   // CTA -> direction * n_chunks + chunk (a subset or launch order), or null
  // batched subset sweeps (n_cta_batch > 0): CTA b runs entry b % n_cta_batch of cta_map on the state vector
  // u_out + (b / n_cta_batch) batch_stride and the inflow rows xrow + (b / n_cta_batch) row_stride.  The batch
  // shares one set of values (from the first state), so its states must agree on DeltaT and T_B.
  int n_cta_batch;
  int64_t batch_stride, row_stride;
  // bounded-wait test (obte_bte_plan_test_wait_timeout): unit whose bulk copies are not issued (-1: none) and
  // the poll cap of the wait for a unit's copies (kWaitPolls normally)
  int skip_unit;
  int wait_limit;
  // deterministic reductions (det != 0, full sweeps only): each (direction, chunk) CTA stores its partial sums
  // instead of adding them atomically; fixed-order reduction kernels sum them afterwards
  int det;
  Real* __restrict__ dpart;   // [n_dir n_chunks][n] lattice-temperature partial of each sweep position
  Real* __restrict__ jpart;   // [n_dir n_chunks][n][ds] flux partials (final pass)
  Real* __restrict__ wpart;   // [n_chunks][n_wo] wall-output partials (wall-output entries of all directions)
  Real* __restrict__ kpart;   // [n_ce][m_pad] kcoef T of each contact entry (final pass)
  Real* __restrict__ spart;   // [n_ce][m_pad] scoef T
  int64_t n_wo;
};

template <typename Real>
__device__ __forceinline__ Real word_real(const int32_t* r, int word);
template <>
__device__ __forceinline__ float word_real<float>(const int32_t* r, int word) {
  return __int_as_float(r[word]);
}
template <>
__device__ __forceinline__ double word_real<double>(const int32_t* r, int word) {
  return __hiloint2double(r[word + 1], r[word]);
}

// num / den by an FP32 reciprocal seed r (relative error e <= 2^-21)
// and one residual correction of the quotient (Markstein's method), t = num r, q = t + (num - den t) r,
// with relative error e^2 <= 2^-42 (~2e-13): three FP64 operations instead of the five of a fully
// refined reciprocal, on GB300's narrow FP64 pipe, which bounds the FP64 sweep.
__device__ __forceinline__ double quot(double num, double den) {
  const double r = (double)__fdividef(1.0f, (float)den);
  const double t = num * r;
  return fma(fma(-den, t, num), r, t);
}

// 16-byte vectors: 4 floats or 2 doubles.
template <int K>
__device__ __forceinline__ void vload(const float* p, float (&x)[K]) {
  static_assert(K % 4 == 0, "whole vectors");
#pragma unroll
  for (int i = 0; i < K; i += 4) {
    const float4 v = *reinterpret_cast<const float4*>(p + i);
    x[i] = v.x; x[i + 1] = v.y; x[i + 2] = v.z; x[i + 3] = v.w;
  }
}
template <int K>
__device__ __forceinline__ void vload(const double* p, double (&x)[K]) {
#pragma unroll
  for (int i = 0; i < K; i += 2) {
    const double2 v = *reinterpret_cast<const double2*>(p + i);
    x[i] = v.x; x[i + 1] = v.y;
  }
}
template <int K>
__device__ __forceinline__ void vstore(float* p, const float (&x)[K]) {
  static_assert(K % 4 == 0, "whole vectors");
#pragma unroll
  for (int i = 0; i < K; i += 4) *reinterpret_cast<float4*>(p + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
}
template <int K>
__device__ __forceinline__ void vstore(double* p, const double (&x)[K]) {
#pragma unroll
  for (int i = 0; i < K; i += 2) *reinterpret_cast<double2*>(p + i) = make_double2(x[i], x[i + 1]);
}

// A ring row's KV MFPs by the row's byte offset: 16 bytes, or 32 of which bit 4 of the offset says which half comes
// first.
template <int KV, typename Real>
__device__ __forceinline__ void row_load(const unsigned char* ring, unsigned off, Real (&x)[KV]) {
  constexpr int H = 16 / (int)sizeof(Real);
  static_assert(KV == H || KV == 2 * H, "one or two 16-byte vectors per row");
  if constexpr (KV == H) {
    vload(reinterpret_cast<const Real*>(ring + off), x);
  } else {
    Real a[H];
    vload(reinterpret_cast<const Real*>(ring + off), a);
#pragma unroll
    for (int i = 0; i < H; ++i) x[i] = a[i];
    vload(reinterpret_cast<const Real*>(ring + (off ^ 16u)), a);
#pragma unroll
    for (int i = 0; i < H; ++i) x[H + i] = a[i];
  }
}
template <int KV, typename Real>
__device__ __forceinline__ void row_store(unsigned char* ring, unsigned off, const Real (&x)[KV]) {
  constexpr int H = 16 / (int)sizeof(Real);
  if constexpr (KV == H) {
    vstore(reinterpret_cast<Real*>(ring + off), x);
  } else {
    Real a[H];
#pragma unroll
    for (int i = 0; i < H; ++i) a[i] = x[i];
    vstore(reinterpret_cast<Real*>(ring + off), a);
#pragma unroll
    for (int i = 0; i < H; ++i) a[i] = x[H + i];
    vstore(reinterpret_cast<Real*>(ring + (off ^ 16u)), a);
  }
}

// a b, rounded (never contracted into an addition)
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// 1 / x for a normal x (the sweep's denominators are 1 + L D >= 1)
__device__ __forceinline__ float rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Wall re-emission of entry i of a unit's nw (wb: the entries, the wall geometry after them).
// Re-emission weight max(sigma . w, 0) / (-sum min(sigma . w, 0)) from the staged wall geometry (bte.py:73-78),
// wall by wall; the sum runs over the MFPs in order.
template <typename Real, int MC, bool DF>
__device__ __forceinline__ void wall_outputs(const SweepParams<Real>& p, const unsigned char* wb, int nw, int i,
                                             const unsigned char* ring, const Real* s_sig, double* dT_out, int chunk) {
  const int4 ent = reinterpret_cast<const int4*>(wb)[i];
  Real T[MC];
  row_load(ring, (unsigned)ent.x & 0xFFFF0u, T);
  if constexpr (DF) {
#pragma unroll
    for (int j = 0; j < MC; ++j) T[j] = dpack_value(T[j]);
  }
  auto sigv = [&](Real x) -> Real {
    if constexpr (DF) return dpack_value(x);
    else return x;
  };
  const int wn = ent.y & 7;
  const int first = (ent.y >> 3) & 0x1FFF;
  const Real* gw = reinterpret_cast<const Real*>(wb + nw * 16);
  const int* wall = reinterpret_cast<const int*>(gw + 4 * (int)((unsigned)ent.y >> 16)) + first;
  gw += 4 * first;
  for (int k = 0; k < wn; ++k, gw += 4) {
    const Real g0 = gw[0], g1 = gw[1], g2 = gw[2], g3 = gw[3];
    Real w = 0;
#pragma unroll
    for (int j = 0; j < MC; ++j) {
      const Real a = sigv(s_sig[j]) * g0 + sigv(s_sig[MC + j]) * g1 + sigv(s_sig[2 * MC + j]) * g2;
      w += (a > Real(0) ? a * g3 : Real(0)) * T[j];
    }
    if (p.det) p.wpart[(int64_t)chunk * p.n_wo + ent.w + k] = w;
    else atomicAdd(&dT_out[p.n + wall[k]], widen(w));
  }
}

// Resident CTAs per SM the register allocation is bounded for.
template <typename Real, int KV>
struct SweepMinBlocks { static constexpr int v = (sizeof(Real) == 4 && KV == 8) ? 5 : 4; };

// DF (Real = double, FINAL only): the FP64 tables swept in double-float arithmetic (see df2).
template <typename Real, int NF, int KV, bool FINAL, bool DF = false>
__global__ void __launch_bounds__(kMaxThreads, SweepMinBlocks<Real, KV>::v)
    bte_sweep_kernel(const __grid_constant__ SweepParams<Real> p) {
  static_assert(!DF || (sizeof(Real) == 8 && FINAL && KV % 2 == 0), "double-float sweeps: FP64 tables, output pass");
  constexpr int MC = KV;
  using RR = Rec<Real, NF>;
  constexpr int RW = RR::W;                        // record words
  constexpr int RB = RW * 4, ROWB = MC * (int)sizeof(Real), VB = 2 * (int)sizeof(Real);
  constexpr bool kGain = sizeof(Real) == 8 && !DF;
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
  int* s_fail = reinterpret_cast<int*>(smem + kFailOff);
  Real* s_sig = reinterpret_cast<Real*>(smem + kSigOff);    // [3][MC]
  unsigned char* ring = smem + kRingOff;

  int bid = (int)blockIdx.x;
  int bt = 0;
  if (p.n_cta_batch > 0) {
    bt = bid / p.n_cta_batch;
    bid -= bt * p.n_cta_batch;
  }
  const int cta = p.cta_map ? p.cta_map[bid] : bid;
  const int q = cta / p.n_chunks;
  const int chunk = cta - q * p.n_chunks;
  const int m0 = chunk * MC;
  const int mc = min(MC, p.n_mfp - m0);
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int nbuf = p.nbuf;
  const int64_t ub = p.unit_base[q];
  const int nlev = (int)(p.unit_base[q + 1] - ub);
  double* __restrict__ dT_out = p.u_out + bt * p.batch_stride;
  const double* __restrict__ gain_qc =
      kGain && p.gain ? p.gain + ((int64_t)q * p.n_chunks + chunk) * p.n * MC : nullptr;

  // this chunk's ordinate data in registers; padded MFPs get L = t = sigma = 0 (harmless T = b).
  // sigma (wall re-emission and the final pass only) is read from shared memory
  Real lam[KV], tt[KV];
#pragma unroll
  for (int j = 0; j < KV; ++j) {
    const bool ok = j < mc;
    lam[j] = ok ? p.mfp[m0 + j] : Real(0);
    tt[j] = ok ? p.tco[(int64_t)q * p.m_pad + m0 + j] : Real(0);
  }
  for (int i = tid; i < MC * 3; i += nthr) {
    const int d = i / MC, j = i - d * MC;
    const Real sv = (j < mc && d < p.ds) ? p.sig[((int64_t)q * p.m_pad + m0 + j) * p.ds + d] : Real(0);
    if constexpr (DF) s_sig[i] = dpack_split(sv);   // packed hi / lo pairs
    else s_sig[i] = sv;
  }
  // DF: the MFPs and weights as pairs (lanes x, y = MFPs j, j + 1)
  df2 lam2[DF ? KV / 2 : 1], tt2[DF ? KV / 2 : 1];
  if constexpr (DF) {
#pragma unroll
    for (int j = 0; j < KV; j += 2) {
      const float2 l0 = dsplit(lam[j]), l1 = dsplit(lam[j + 1]), t0 = dsplit(tt[j]), t1 = dsplit(tt[j + 1]);
      lam2[j / 2] = {make_float2(l0.x, l1.x), make_float2(l0.y, l1.y)};
      tt2[j / 2] = {make_float2(t0.x, t1.x), make_float2(t0.y, t1.y)};
    }
  }
  for (int j = tid; j < MC; j += nthr) reinterpret_cast<Real*>(ring + (size_t)p.zero_row * ROWB)[j] = Real(0);
  if (tid == 0) {
    for (int i = 0; i < nbuf; ++i) mbar_init(&bars[i], 1);
    *s_fail = INT_MAX;
    fence_mbar_init();
  }
  __syncthreads();

  // Bulk copies of a unit into stage bi and output block oi: records, values, outputs, periodic inflow rows, gain
  // rows.  blk64, val16 = record and value sources, size = their sizes in 16-byte units, prow = first bank row,
  // np = bank rows | size of the output block << 16
  auto issue = [&](int u, int bi, int oi, unsigned blk64, unsigned val16, unsigned size, int prow, unsigned np) {
    if (u == p.skip_unit) return;   // test of the bounded wait: this unit's copies never arrive
    const unsigned bb = (size & 0xFFFFu) << 4, vb = (size >> 16) << 4, ob = (np >> 16) << 4, npf = np & 0xFFFFu;
    unsigned char* st = smem + p.stage0 + bi * p.stage;
    const unsigned char* src = reinterpret_cast<const unsigned char*>(p.blk) + (uint64_t)blk64 * kBlkUnit;
    uint64_t* bar = &bars[bi];
    unsigned gb = 0;
    if constexpr (kGain) gb = gain_qc ? (vb / VB) * ROWB : 0u;     // FP64 values are 16 bytes: vb / 16 elements
    fence_proxy_async();
    mbar_expect_tx(bar, bb + vb + ob + gb + npf * ROWB);
    tma_load_1d(st, src, bb, bar);
    tma_load_1d(st + p.val_off, reinterpret_cast<const unsigned char*>(p.vals) + ((uint64_t)val16 << 4), vb, bar);
    if (ob) tma_load_1d(smem + p.out0 + oi * p.out, src + bb, ob, bar);
    if (npf)
      tma_load_1d(ring + (size_t)(p.prow0 + bi * p.emax) * ROWB,
                  p.xrow + bt * p.row_stride + ((int64_t)prow * p.n_chunks + (int64_t)chunk * npf) * MC, npf * ROWB, bar);
    if constexpr (kGain)
      if (gb) tma_load_1d(st + p.gain_off, gain_qc + ((int64_t)val16 - (int64_t)q * p.n) * MC, gb, bar);
  };
  // the issuing thread: lane 0 of the last warp, whose elements are the last of a unit
  const int issuer = nthr - 32;
  if (tid == issuer)
    for (int u = 0; u < nbuf && u < nlev; ++u) {
      const int4* d = reinterpret_cast<const int4*>(p.desc) + 2 * (ub + u);
      const int4 a = __ldg(d), b = __ldg(d + 1);
      issue(u, u, u, (unsigned)b.x, (unsigned)b.y, (unsigned)b.z, a.z, (unsigned)a.w);
    }

  // record, value pair and gains of one element of a staged unit
  int32_t r[RW];
  Real bv, pw;
  Real gn[kGain ? KV : 1];
  auto fetch = [&](const unsigned char* st, int odd, int el) {
    const int4* r4 = reinterpret_cast<const int4*>(st + kHeader + el * RB);
#pragma unroll
    for (int i = 0; i < RW / 4; ++i) {
      const int4 x = r4[i];
      r[4 * i] = x.x; r[4 * i + 1] = x.y; r[4 * i + 2] = x.z; r[4 * i + 3] = x.w;
    }
    const Real* v = reinterpret_cast<const Real*>(st + p.val_off) + 2 * (odd + el);
    if constexpr (sizeof(Real) == 4) {
      const float2 x = *reinterpret_cast<const float2*>(v);
      bv = x.x; pw = x.y;
    } else {
      const double2 x = *reinterpret_cast<const double2*>(v);
      bv = x.x; pw = x.y;
    }
    if constexpr (kGain)
      if (gain_qc) vload(reinterpret_cast<const double*>(st + p.gain_off) + el * KV, gn);
  };

  int bi = 0;            // stage of unit u (u mod nbuf)
  int oi = 0;            // output block of unit u - 1 (mod nbuf + 1)
  unsigned phase = 0;    // parity of its mbarrier phase ((u / nbuf) & 1)
  const unsigned char* st = smem + p.stage0;
  int4 hd = make_int4(0, 0, 0, 0);
  // final pass: kappa and suppression sums of the direction, MFP `cj` in this thread (a warp before the issuer's)
  const int cj = nthr >= 64 ? tid - (nthr - 64) : tid;
  constexpr bool kTwoOrders = sizeof(Real) == 4;   // in FP64 the order is below any tolerance
  Real ksum = 0, ssum = 0, ksum2 = 0, ssum2 = 0;
  // MFP j of the row at byte offset `off`
  auto row_value = [&](unsigned off, int j) -> Real {
    constexpr int H = 16 / (int)sizeof(Real);
    const Real v = reinterpret_cast<const Real*>(ring + (off ^ (j >= H ? 16u : 0u)))[j % H];
    if constexpr (DF) return dpack_value(v);
    else return v;
  };
  // The unit's part of the contact sums in one of the two orders of its entries (contact_order): products rounded, then
  // added one by one, loads four entries ahead.  One thread per MFP: the sums are the same in every pass and
  // whatever the threads and stages.
  auto contacts = [&](const int4* ent, int count, bool second, Real& ks, Real& ss) {
    for (int i0 = 0; i0 < count; i0 += 4) {
      Real kv[4], sv[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        kv[k] = sv[k] = Real(0);
        if (i0 + k < count) {
          const int4 e = ent[second ? (int)((unsigned)ent[i0 + k].x >> 20) : i0 + k];
          const Real T = row_value((unsigned)e.x & 0xFFFF0u, cj);
          kv[k] = mul_rn(p.kcoef[(int64_t)e.z * p.m_pad + m0 + cj], T);
          sv[k] = mul_rn(p.scoef[e.z], T);
          if (p.det && !second) {
            p.kpart[(int64_t)e.z * p.m_pad + m0 + cj] = kv[k];
            p.spart[(int64_t)e.z * p.m_pad + m0 + cj] = sv[k];
          }
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        ks += kv[k];
        ss += sv[k];
      }
    }
  };
  // Per-MFP outputs of a finished unit, from its rows in the ring: one lane per (periodic source, MFP) from the
  // last thread down, one lane per wall element from the warp before (the high threads have no
  // element in most units), one lane per MFP for the contact sums.  Done while the next unit runs, off the chain
  // from level to level; inside the element loop they would take ~150 instructions of every warp with one such
  // element.
  auto outputs = [&](const unsigned char* ob, int counts) {
    const int nx = counts & 0x3FF, nw = (counts >> 10) & 0x3FF;
    for (int i = nthr - 1 - tid; i < nx * MC; i += nthr) {
      const int k = i / MC, j = MC - 1 - (i - k * MC);      // consecutive lanes, consecutive MFPs
      const int2 e = reinterpret_cast<const int2*>(ob)[k];
      const Real v = row_value((unsigned)e.y, j);
      if (j < mc) dT_out[p.n + p.nd + (int64_t)(unsigned)e.x * p.n_mfp + m0 + j] = widen(v);
    }
    if (nw) {
      const unsigned char* wb = ob + ((nx * 8 + 15) & ~15);
      int i = nthr - 33 - tid;
      if (i < 0) i += nthr;
      for (; i < nw; i += nthr) {
        wall_outputs<Real, MC, DF>(p, wb, nw, i, ring, s_sig, dT_out, chunk);
      }
      if constexpr (FINAL) {
        if (cj >= 0 && cj < mc) {
          contacts(reinterpret_cast<const int4*>(wb), counts >> 20, false, ksum, ssum);
          if constexpr (kTwoOrders)
            if (!p.det) contacts(reinterpret_cast<const int4*>(wb), counts >> 20, true, ksum2, ssum2);
        }
      }
    }
  };
  // wait for a unit's stage and read its header and this thread's first element; a thread whose wait gives up
  // skips the unit and says so
  auto arrive = [&](int u) {
    if (mbar_wait_bounded(&bars[bi], phase, p.wait_limit)) {
      hd = *reinterpret_cast<const int4*>(st);
      fetch(st, hd.x >> 16, tid);
    } else {
      hd = make_int4(0, 0, 0, 0);
      atomicOr(p.err, 1);
      atomicMin(s_fail, u);
    }
  };
  arrive(0);
  __syncthreads();
  int counts = 0;        // outputs of unit u - 1
  for (int u = 0; u < nlev; ++u) {
    // the first failed unit, written before the barrier above; later ones carry a larger number
    const int fail = *(volatile int*)s_fail;
    const int n_el = hd.x & 0xFFFF;
    int el = tid;
    // read together: while the row loads are in flight the issuer refills the stage of unit u - 1
    Real v0[KV], v1[KV], v2[NF > 2 ? KV : 1], v3[NF > 3 ? KV : 1];
    auto rows = [&]() {
      row_load(ring, ((unsigned)r[1] >> 12) & 0xFFFF0u, v0);
      row_load(ring, ((unsigned)r[2] << 4) & 0xFFFF0u, v1);
      if constexpr (NF > 2) row_load(ring, ((unsigned)r[2] >> 12) & 0xFFFF0u, v2);
      if constexpr (NF > 3) row_load(ring, ((unsigned)r[3] << 4) & 0xFFFF0u, v3);
    };
    if (el < n_el) rows();
    if (fail <= u) {
      // let the copies this CTA still has in flight land before leaving (bounded)
      if (tid == issuer)
        for (int w = u; w < nlev && w < (u ? u - 1 + nbuf : nbuf); ++w)
          mbar_wait_bounded(&bars[w % nbuf], (unsigned)(w / nbuf) & 1u, p.wait_limit);
      __syncthreads();
      return;
    }
    if (tid == issuer && u > 0 && u - 1 + nbuf < nlev) {
      const int pb = bi == 0 ? nbuf - 1 : bi - 1;
      const int4* h = reinterpret_cast<const int4*>(smem + p.stage0 + pb * p.stage);
      const int np = h[0].w;
      const int4 d = h[1];
      // unit u - 1 + nbuf takes the stage of unit u - 1, and the output block of unit u - 2
      issue(u - 1 + nbuf, pb, oi == 0 ? nbuf : oi - 1, (unsigned)d.x, (unsigned)d.y, (unsigned)d.z, d.w, (unsigned)np);
    }
    while (el < n_el) {
      const int c = r[0];
      const unsigned so = ((unsigned)r[1] << 4) & 0xFFFF0u;
      const Real b = bv;
      const Real c0 = word_real<Real>(r, RR::COEF);
      const Real c1 = word_real<Real>(r, RR::COEF + RR::CSTEP);
      const Real c2 = NF > 2 ? word_real<Real>(r, RR::COEF + 2 * RR::CSTEP) : Real(0);
      const Real c3 = NF > 3 ? word_real<Real>(r, RR::COEF + 3 * RR::CSTEP) : Real(0);
      const Real D = word_real<Real>(r, RR::D);
      Real T[KV];
      Real dacc = 0, j0 = 0, j1 = 0, j2 = 0;
      const Real* sg0 = s_sig;
      const Real* sg1 = sg0 + MC;
      const Real* sg2 = sg1 + MC;
      if constexpr (DF) {
        // output pass in double-float: the ring holds packed pairs, every product and sum is a pair
        const df2 C0 = dbcast(c0), C1 = dbcast(c1), C2 = dbcast(c2), C3 = dbcast(c3), DD = dbcast(D);
        const df2 BB = dbcast(b), PW = dbcast(pw);
        const df2 ONE = {make_float2(1.0f, 1.0f), make_float2(0.0f, 0.0f)};
        df2 da = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)}, ja = da, jb = da, jc = da;
        Real Tp[KV];
#pragma unroll
        for (int j = 0; j < KV; j += 2) {
          df2 sm = dmul2(C0, dunpack2(v0[j], v0[j + 1]));
          sm = dadd2(sm, dmul2(C1, dunpack2(v1[j], v1[j + 1])));
          if constexpr (NF > 2) sm = dadd2(sm, dmul2(C2, dunpack2(v2[j], v2[j + 1])));
          if constexpr (NF > 3) sm = dadd2(sm, dmul2(C3, dunpack2(v3[j], v3[j + 1])));
          const df2 LM = lam2[j / 2];
          const df2 num = dadd2(BB, dmul2(LM, dadd2(PW, dneg2(sm))));   // b + L (pw - sm)
          const df2 den = dadd2(ONE, dmul2(LM, DD));                    // 1 + L D
          const df2 t2 = ddiv2(num, den);
          Tp[j] = dpack(t2.h.x, t2.l.x);
          Tp[j + 1] = dpack(t2.h.y, t2.l.y);
          da = dadd2(da, dmul2(tt2[j / 2], t2));
          ja = dadd2(ja, dmul2(dunpack2(sg0[j], sg0[j + 1]), t2));
          jb = dadd2(jb, dmul2(dunpack2(sg1[j], sg1[j + 1]), t2));
          if (p.ds > 2) jc = dadd2(jc, dmul2(dunpack2(sg2[j], sg2[j + 1]), t2));
        }
        dacc = ((double)da.h.x + (double)da.h.y) + ((double)da.l.x + (double)da.l.y);
        j0 = ((double)ja.h.x + (double)ja.h.y) + ((double)ja.l.x + (double)ja.l.y);
        j1 = ((double)jb.h.x + (double)jb.h.y) + ((double)jb.l.x + (double)jb.l.y);
        j2 = ((double)jc.h.x + (double)jc.h.y) + ((double)jc.l.x + (double)jc.l.y);
        row_store(ring, so, Tp);
        // real values for the stored fields below
        const bool need = p.Xs != nullptr || p.Xd != nullptr;
#pragma unroll
        for (int j = 0; j < KV; ++j) T[j] = need ? dpack_value(Tp[j]) : Real(0);
      } else if constexpr (sizeof(Real) == 4) {
        // FP32: the MFPs in pairs with Blackwell's packed FP32x2 arithmetic (one instruction per two MFPs;
        // each lane of a packed operation rounds like the scalar one)
        const float2 C0 = make_float2(c0, c0), C1 = make_float2(c1, c1), C2 = make_float2(c2, c2);
        const float2 C3 = make_float2(c3, c3), DD = make_float2(D, D), BB = make_float2(b, b);
        const float2 PW = make_float2(pw, pw), ONE = make_float2(1.0f, 1.0f), NEG = make_float2(-1.0f, -1.0f);
#pragma unroll
        for (int j = 0; j < KV; j += 2) {
          float2 sm = __fmul2_rn(C0, make_float2(v0[j], v0[j + 1]));
          sm = __ffma2_rn(C1, make_float2(v1[j], v1[j + 1]), sm);
          if constexpr (NF > 2) sm = __ffma2_rn(C2, make_float2(v2[j], v2[j + 1]), sm);
          if constexpr (NF > 3) sm = __ffma2_rn(C3, make_float2(v3[j], v3[j + 1]), sm);
          const float2 lm = make_float2(lam[j], lam[j + 1]);
          const float2 num = __ffma2_rn(lm, __ffma2_rn(NEG, sm, PW), BB);    // b + L (pw - sm)
          const float2 den = __ffma2_rn(lm, DD, ONE);                        // 1 + L D
          const float2 t2 = __fmul2_rn(num, make_float2(rcp(den.x), rcp(den.y)));
          T[j] = t2.x;
          T[j + 1] = t2.y;
        }
        row_store(ring, so, T);
        // sum over the chunk's MFPs, even and odd ones apart, in MFP order
        auto wsum = [&](auto weight) -> float {
          float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
          for (int j = 0; j < KV; j += 2) acc = __ffma2_rn(weight(j), make_float2(T[j], T[j + 1]), acc);
          return acc.x + acc.y;
        };
        dacc = wsum([&](int j) { return make_float2(tt[j], tt[j + 1]); });
        if (FINAL) {
          j0 = wsum([&](int j) { return make_float2(sg0[j], sg0[j + 1]); });
          j1 = wsum([&](int j) { return make_float2(sg1[j], sg1[j + 1]); });
          if (p.ds > 2) j2 = wsum([&](int j) { return make_float2(sg2[j], sg2[j + 1]); });
        }
      } else {
        if (gain_qc) {
          // T = b + G (p - D b - sum g T_up) with G = L / (1 + L D): five FP64 operations per unknown (four
          // and the weighted sum) instead of the seven of the quotient form times the reciprocal
          const Real y = fma(-D, b, pw);
#pragma unroll
          for (int j = 0; j < KV; ++j) {
            Real z = fma(-c0, v0[j], y);
            z = fma(-c1, v1[j], z);
            if constexpr (NF > 2) z = fma(-c2, v2[j], z);
            if constexpr (NF > 3) z = fma(-c3, v3[j], z);
            T[j] = fma((Real)gn[kGain ? j : 0], z, b);
          }
        } else {
#pragma unroll
          for (int j = 0; j < KV; ++j) {
            Real sm = c0 * v0[j] + c1 * v1[j];
            if constexpr (NF > 2) sm += c2 * v2[j];
            if constexpr (NF > 3) sm += c3 * v3[j];
            T[j] = quot(b + lam[j] * (pw - sm), Real(1) + lam[j] * D);
          }
        }
#pragma unroll
        for (int j = 0; j < KV; ++j) {
          dacc += tt[j] * T[j];
          if (FINAL) {
            j0 += sg0[j] * T[j];
            j1 += sg1[j] * T[j];
            if (p.ds > 2) j2 += sg2[j] * T[j];
          }
        }
      }
      if constexpr (!DF && sizeof(Real) == 8) row_store(ring, so, T);
      if (FINAL && p.Xs != nullptr) {
#pragma unroll
        for (int j = 0; j < KV; ++j)
          if (j < mc) {
            float* xs = p.Xs + ((int64_t)q * p.n + c) * p.n_mfp + m0 + j;
            *xs = p.xs_add ? *xs + (float)T[j] : (float)T[j];
          }
      }
      if (FINAL && p.Xd != nullptr) {
#pragma unroll
        for (int j = 0; j < KV; ++j)
          if (j < mc) p.Xd[((int64_t)q * p.n + c) * p.n_mfp + m0 + j] = (double)T[j];
      }
      if (p.det) p.dpart[(int64_t)cta * p.n + hd.y + el] = dacc;
      else atomicAdd(&dT_out[c], widen(dacc));
      if (FINAL) {
        if (p.det) {
          Real* jp = p.jpart + ((int64_t)cta * p.n + hd.y + el) * p.ds;
          jp[0] = j0;
          if (p.ds > 1) jp[1] = j1;
          if (p.ds > 2) jp[2] = j2;
        } else {
          atomicAdd(&p.Jraw[(int64_t)c * p.ds], widen(j0));
          if (p.ds > 1) atomicAdd(&p.Jraw[(int64_t)c * p.ds + 1], widen(j1));
          if (p.ds > 2) atomicAdd(&p.Jraw[(int64_t)c * p.ds + 2], widen(j2));
        }
      }
      el += nthr;
      if (el < n_el) {           // units wider than the CTA
        fetch(st, hd.x >> 16, el);
        rows();
      }
    }
    if (counts) outputs(smem + p.out0 + oi * p.out, counts);
    counts = hd.z;
    if (u > 0 && ++oi > nbuf) oi = 0;
    // unit u + 1: its records (not its rows) before the barrier
    if (++bi == nbuf) { bi = 0; phase ^= 1u; }
    st = smem + p.stage0 + bi * p.stage;
    if (u + 1 < nlev) arrive(u + 1);
    __syncthreads();
  }
  if (counts) outputs(smem + p.out0 + oi * p.out, counts);
  if (FINAL && !p.det && cj >= 0 && cj < mc) {
    p.K[(int64_t)(m0 + cj) * p.n_dir + q] = kTwoOrders ? 0.5 * ((double)ksum + (double)ksum2) : (double)ksum;
    p.S_out[(int64_t)(m0 + cj) * p.n_dir + q] = kTwoOrders ? 0.5 * ((double)ssum + (double)ssum2) : (double)ssum;
  }
}

// ---- deterministic reductions -------------------------------------------------------
// Every sum below runs in a fixed order (chunks, then directions; a wall's entries in entry order; a
// direction's contact entries in order), so the result does not depend on which CTA ran first.

// S[q][pos] = sum over chunks of the lattice-temperature partials (and the flux partials)
template <typename Real>
__global__ void det_pos_sum_kernel(const Real* __restrict__ dpart, const Real* __restrict__ jpart, int n_chunks,
                                   int64_t n, int64_t total, int ds, double* __restrict__ S, double* __restrict__ SJ) {
  for (int64_t it = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; it < total; it += (int64_t)gridDim.x * blockDim.x) {
    const int64_t q = it / n, pos = it - q * n;
    const int64_t b0 = q * n_chunks * n + pos;
    double acc = 0;
    for (int ch = 0; ch < n_chunks; ++ch) acc += (double)dpart[b0 + (int64_t)ch * n];
    S[it] = acc;
    if (jpart)
      for (int d = 0; d < ds; ++d) {
        double aj = 0;
        for (int ch = 0; ch < n_chunks; ++ch) aj += (double)jpart[(b0 + (int64_t)ch * n) * ds + d];
        SJ[it * ds + d] = aj;
      }
  }
}

// element sums over the directions, through the position of the element in each direction's order
__global__ void det_elem_sum_kernel(const double* __restrict__ S, const double* __restrict__ SJ,
                                    const int32_t* __restrict__ inv, int n_dir, int64_t n, int ds,
                                    double* __restrict__ dT_out, double* __restrict__ Jraw) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
    double acc = 0, a0 = 0, a1 = 0, a2 = 0;
    for (int q = 0; q < n_dir; ++q) {
      const int64_t it = (int64_t)q * n + inv[(int64_t)q * n + c];
      acc += S[it];
      if (SJ) {
        a0 += SJ[it * ds];
        if (ds > 1) a1 += SJ[it * ds + 1];
        if (ds > 2) a2 += SJ[it * ds + 2];
      }
    }
    dT_out[c] = acc;
    if (SJ) {
      Jraw[c * ds] = a0;
      if (ds > 1) Jraw[c * ds + 1] = a1;
      if (ds > 2) Jraw[c * ds + 2] = a2;
    }
  }
}

template <typename Real>
__global__ void det_wall_sum_kernel(const Real* __restrict__ wpart, int n_chunks, int64_t n_wo,
                                    const int32_t* __restrict__ wptr, const int32_t* __restrict__ went, int64_t nd,
                                    double* __restrict__ TB_out) {
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < nd; w += (int64_t)gridDim.x * blockDim.x) {
    double acc = 0;
    for (int k = wptr[w]; k < wptr[w + 1]; ++k)
      for (int ch = 0; ch < n_chunks; ++ch) acc += (double)wpart[(int64_t)ch * n_wo + went[k]];
    TB_out[w] = acc;
  }
}

template <typename Real>
__global__ void det_contact_sum_kernel(const Real* __restrict__ kpart, const Real* __restrict__ spart,
                                       const int32_t* __restrict__ ce_off, int n_dir, int n_mfp, int m_pad,
                                       double* __restrict__ K, double* __restrict__ S) {
  const int64_t total = (int64_t)n_mfp * n_dir;
  for (int64_t it = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; it < total; it += (int64_t)gridDim.x * blockDim.x) {
    const int m = (int)(it / n_dir), q = (int)(it - (int64_t)m * n_dir);
    double ak = 0, as = 0;
    for (int ce = ce_off[q]; ce < ce_off[q + 1]; ++ce) {
      ak += (double)kpart[(int64_t)ce * m_pad + m];
      as += (double)spart[(int64_t)ce * m_pad + m];
    }
    K[it] = ak;
    S[it] = as;
  }
}

// ---- table upload ---------------------------------------------------------------

size_t DevSchedule::bytes() const {
  const DevBuf* all[] = {&blk, &desc, &unit_base, &pfe, &xrow, &mfp, &tco, &sig, &kcoef, &scoef, &hs,
                         &vals, &cellmap, &Pq, &si, &sr, &spec, &lpt, &gain};
  size_t b = 0;
  for (auto* x : all) b += x->bytes;
  return b;
}

template <typename Real>
static obte_status upload_real(DevBuf& b, const std::vector<double>& v, cudaStream_t st) {
  std::vector<Real> h(v.begin(), v.end());
  if (h.empty()) h.push_back(Real(0));
  return upload(b, h, st);
}

// Shared memory a CTA can have and SMs of the device that a layout is for (a GB300's where no device is at hand).
struct DeviceShape {
  size_t smem = 232448;
  int sms = 152;
};

// FP32: the MFPs that share a partial sum.  The grouping is part of the results' rounding, so it stays what it was
// when the rule was made: 8 while a layout of that time (records with a word per side, two staged units of 128
// elements, output entries and prefetch lists, rows read back in their own level) would let at least 4 CTAs
// share an SM, else 4; 4 for at most 4 MFPs.  On the present kernel the other choice costs (4 and 8 MFPs): 2,000
// triangles x 30 x 48 117 and 120 us, 8,000 x 60 x 48 217 and 217, 11,000 x 77 x 48 355 and 281, 60,000 x 100 x 96 1,861
// and 1,178, 120,000 x 60 x 48 1,278 and 977; 8,000 tetrahedra x 30 x 128 304 and 222, 24,000 x 30 x 512 1,652 and 1,539.
static int frozen_mc32(const Schedule& s, const UnitStats& base) {
  if (s.n_mfp <= 4) return 4;
  const int64_t stage = kBaseUnit * rec_words(4, s.nf) * 4 + (kBaseUnit + 2) * 8 + base.unit_wo * 16 +
                        ((base.emax + 3) & ~3) * 4 + base.unit_sx * 16;
  const int64_t rows = s.base_slots + 2 + 2 * base.emax;
  const int64_t smem = 128 + 2 * stage + 8 * 20 + rows * 32;
  return smem + 1024 <= 228 * 1024 / 4 ? 8 : 4;
}

// FP64: four MFPs to a CTA halve the passes over the records, but also the CTAs, and their rows take twice the room.
// They pay while four CTAs still share an SM and the last wave of CTAs is not much emptier than the others.  Two
// against four MFPs, with CTAs of four and how many share an SM: 8,000 triangles x 60 x 48 (720, 5) 506 and 458
// us, 20,000 x 100 x 96 (2,400, 4) 2,754 and 2,594, 60,000 x 100 x 96 (2,400, 4) 6,554 and 6,008, x 100 x 48 (1,200, 4) 3,421
// and 3,119; with 1.03 and 1.18 waves 60,000 x 52 x 48 (624, 4) 2,003 and 2,295, 20,000 x 60 x 48 (720, 4) 958 and
// 1,181; with three to an SM 40,000 x 100 x 96 5,075 and 5,151, with two 180,000 x 60 x 48 5,830 and 6,843; in half a
// wave 2,000 x 30 x 48 (384, 5) 146 and 194; in 1.37 waves an output pass of 128^2 squares x 50 x 64 (832, 4) 3,513 and
// 3,280.  (The line is for a sweep alone: with four streams at once, whose CTAs fill
// each other's waves, four to a CTA were 3 to 20 % faster at each of nine sizes, 20,000 x 60 x 48 among them.)  Only with
// two inflow rows do they fit the registers (8,000 tetrahedra x 30 x 128 704 and 718).
static bool wide64(int64_t ctas, int resident, int sms) {
  const double waves = (double)ctas / ((double)std::max(resident, 1) * sms);
  return resident >= 4 && std::ceil(waves) <= 1.6 * waves;
}

// The units of the base layout and their counts.
struct BaseUnits {
  Units un;
  std::vector<int64_t> unit_base;
  std::vector<int32_t> cnt;
  UnitStats st;
};

// A plan's launch shape and the units it is for.
struct Shaped {
  Units un;
  std::vector<int64_t> unit_base;
  std::vector<int32_t> cnt;
  Layout lay;
  bool fits = false;
};

// Unit size and stages for KV MFPs per CTA and `threads`, by shape alone.  Measured (FP32 sweep calls): 96 and 128
// threads on levels of 53 elements (11,000 triangles) 274 and 278 us, of 102 (60,000) 1,309 and 1,159; two and four
// stages on 11,000 triangles (one or two CTAs an SM either way) 279 and 274 us, two and three where the third costs a
// resident CTA (60,000) 1,159 and 1,422; units of 96, 128 and 192 elements on the 60k benchmark cell 1,549, 1,430 and
// 1,649 us (5, 5 and 4 CTAs an SM).
template <typename Real>
static void shape_units(const Schedule& s, const DeviceShape& dev, const BaseUnits& base, int KV, int threads,
                        int final_threads, Shaped& r) {
  int widest = 0;
  for (int q = 0; q < s.n_dir; ++q) {
    const int32_t* lp = s.lev_ptr.data() + s.lev_off[q];
    for (int L = 0; L < s.nlev[q]; ++L) widest = std::max(widest, (int)(lp[L + 1] - lp[L]));
  }
  const int n_chunks = (s.n_mfp + KV - 1) / KV;
  // CTAs an SM has to run: no more are worth making room for
  const int64_t want = std::max<int64_t>(1, ((int64_t)s.n_dir * n_chunks + dev.sms - 1) / dev.sms);
  Layout shape;
  shape.KV = KV;
  shape.threads = threads;
  shape.final_threads = final_threads;
  UnitStats st = base.st;
  auto layout = [&](const UnitStats& e, int nbuf) { return make_layout<Real>(s, e, shape, nbuf); };
  auto steps = [&](int cap) {
    int64_t c = 0;
    for (int q = 0; q < s.n_dir; ++q) {
      const int32_t* lp = s.lev_ptr.data() + s.lev_off[q];
      for (int L = 0; L < s.nlev[q]; ++L) c += (lp[L + 1] - lp[L] + cap - 1) / cap;
    }
    return (double)c;
  };
  // unit size: a level wider than a unit costs one more step of the chain, a wider unit costs shared memory and
  // so CTAs per SM: the size with the fewest steps per resident CTA
  int cap = kBaseUnit;
  double best = 0;
  for (int c = kBaseUnit; c <= 256; c += 32) {
    UnitStats e = st;                       // what wider units would hold, in proportion
    e.unit_el = std::min(c, widest);
    if (e.unit_sx > kUnitSx) e.unit_out = e.unit_out * c / kBaseUnit;
    if (e.emax > kUnitPf) e.emax = e.emax * c / kBaseUnit;
    const int res = resident<Real>(layout(e, 2));
    if (res < 1) break;
    const double cost = steps(c) / (double)std::min<int64_t>(res, want);
    if (c == kBaseUnit || cost < 0.97 * best) { best = cost; cap = c; }
    if (c >= widest) break;
  }
  if (const char* e = std::getenv("OBTE_SWEEP_UNIT")) cap = std::max(32, std::min(kMaxUnit, std::atoi(e)));
  auto build = [&]() {
    build_units(s, cap, r.un);
    st = count_units(s, r.un, sizeof(Real), r.unit_base, r.cnt);
  };
  if (cap == kBaseUnit) {
    r.un = base.un;
    r.unit_base = base.unit_base;
    r.cnt = base.cnt;
  } else {
    build();
  }
  // smaller units while two stages do not fit a CTA
  while (layout(st, 2).smem > dev.smem && cap > 32) {
    cap /= 2;
    build();
  }
  r.lay = layout(st, 2);
  r.fits = r.lay.smem <= dev.smem;
  if (!r.fits) return;
  // more stages where the extra ones cost no resident CTA
  const char* nb_env = std::getenv("OBTE_SWEEP_NBUF");
  const int64_t have = std::min<int64_t>(resident<Real>(r.lay), want);
  for (int nb = nb_env ? std::max(2, std::min(kMaxBuf, std::atoi(nb_env))) : 4; nb > 2; --nb) {
    const Layout l = layout(st, nb);
    if (l.smem <= dev.smem && (nb_env || std::min<int64_t>(resident<Real>(l), want) >= have)) { r.lay = l; break; }
  }
}

// The launch shape of a plan: MFPs per CTA by the rules above (OBTE_SWEEP_KV forces a compiled value), threads by the
// width of the levels.  A front too wide for that is tried with narrow rows, then with units of 32 elements and as
// many threads, whose stages are a quarter.
template <typename Real>
static obte_status choose_layout(const Schedule& s, const DeviceShape& dev, BaseUnits& base, Shaped& out) {
  constexpr int kNarrow = 16 / (int)sizeof(Real), kWide = 2 * kNarrow;
  build_units(s, kBaseUnit, base.un);
  base.st = count_units(s, base.un, sizeof(Real), base.unit_base, base.cnt);
  if (base.st.bad_wo) {
    set_error("wall re-emission entries are not in sweep order");
    return OBTE_ERR_BAD_ARG;
  }
  int64_t levels = 0;
  for (int q = 0; q < s.n_dir; ++q) levels += s.nlev[q];
  const double width = levels ? (double)s.n_dir * s.n / (double)levels : 1.0;
  int threads = width <= 64 ? 96 : kMaxThreads;
  if (const char* e = std::getenv("OBTE_SWEEP_THREADS")) {
    const int v = std::atoi(e);
    if (v >= 32 && v <= kMaxThreads && v % 32 == 0) threads = v;
  }
  auto attempt = [&](int KV, int thr, int final_thr) {
    out.fits = false;
    shape_units<Real>(s, dev, base, KV, thr, final_thr, out);
    return out.fits;
  };
  const char* kv_env = std::getenv("OBTE_SWEEP_KV");
  const int forced = kv_env ? std::atoi(kv_env) : 0;
  if (forced == kNarrow || forced == kWide) {
    if (attempt(forced, threads, kMaxThreads)) return OBTE_OK;
  } else if constexpr (sizeof(Real) == 4) {
    if (frozen_mc32(s, base.st) == kWide && attempt(kWide, threads, kMaxThreads)) return OBTE_OK;
  } else if (s.n_up == 2) {
    const int64_t ctas = (int64_t)s.n_dir * ((s.n_mfp + kWide - 1) / kWide);
    if (ctas >= 3 * dev.sms && attempt(kWide, threads, kMaxThreads) && wide64(ctas, resident<Real>(out.lay), dev.sms))
      return OBTE_OK;
  }
  if (attempt(kNarrow, threads, kMaxThreads) || attempt(kNarrow, 32, 32)) return OBTE_OK;
  set_error("sweep front needs more shared memory than one CTA can have (" + std::to_string(out.lay.rows) + " rows)");
  return OBTE_ERR_UNSUPPORTED;
}

template <typename Real>
static obte_status upload_tables(obte_plan plan, DevSchedule& d) {
  PhaseTimer timer(sizeof(Real) == 4 ? "upload_tables fp32" : "upload_tables fp64");
  const Schedule& s = plan->sched;
  cudaStream_t st = plan->stream;
  Shaped sh;
  Packed pk;
  {
    PhaseTimer tp("pack");
    BaseUnits base;
    OBTE_TRY(choose_layout<Real>(s, {(size_t)plan->ctx->smem_optin, plan->ctx->num_sms}, base, sh));
    OBTE_TRY(pack<Real>(s, sh.un, base.un, sh.unit_base, sh.cnt, sh.lay, pk));
    OBTE_TRY(upload(d.unit_base, sh.unit_base, st));
    d.n_units = sh.unit_base[s.n_dir];
  }
  const Units& un = sh.un;
  const Layout& l = pk.lay;
  d.mc = l.KV;
  d.n_chunks = (s.n_mfp + d.mc - 1) / d.mc;
  d.threads = l.threads;
  d.final_threads = l.final_threads;
  d.prow0 = l.prow0;
  d.emax = l.emax;
  d.nbuf = l.nbuf;
  d.stage0 = kRingOff + l.rows * d.mc * (int)sizeof(Real);
  d.stage = l.stage();
  d.out0 = d.stage0 + l.nbuf * l.stage();
  d.out = l.out;
  d.val_off = l.blk;
  d.gain_off = l.blk + l.val;
  d.smem = l.smem;
  d.n_pf = pk.n_pf;
  d.row_stride = pk.n_pf * d.n_chunks * d.mc;
  if (timer.on)
    std::fprintf(stderr, "[obte trace] sweep shape %s: KV %d, %d threads, %d chunks x %d directions = %d CTAs, %zu B "
                 "shared memory (%d rows = %d slots + 2 + %d x %d bank rows; %d stages of %d B), <= %d CTAs per SM; %lld "
                 "units, %lld levels\n", sizeof(Real) == 4 ? "fp32" : "fp64", l.KV, l.threads, d.n_chunks, s.n_dir,
                 d.n_chunks * s.n_dir, l.smem, l.rows, s.max_slots, l.nbuf, l.emax, l.nbuf, l.stage(), resident<Real>(l),
                 (long long)d.n_units, (long long)std::accumulate(s.nlev.begin(), s.nlev.end(), (int64_t)0));
  OBTE_TRY(upload(d.blk, pk.blk, st));
  OBTE_TRY(upload(d.desc, pk.desc, st));
  OBTE_TRY(upload(d.pfe, pk.pfe, st));
  OBTE_TRY(d.xrow.alloc(std::max<size_t>((size_t)d.row_stride * sizeof(Real), 32)));
  OBTE_TRY(upload(d.cellmap, pk.cellmap, st));
  OBTE_TRY(upload(d.Pq, pk.P, st));
  OBTE_TRY(upload(d.si, pk.si, st));
  OBTE_TRY(upload(d.spec, pk.spec, st));
  OBTE_TRY(upload_real<Real>(d.sr, pk.sr, st));
  {
    // Each CTA is a serial chain of its direction's units (602-846 per direction on the 60k-triangle
    // cell), and the grid runs in about two waves: launching the longest chains first keeps a slot from
    // drawing two long ones (longest-processing-time-first order; the hardware dispatches blocks in index
    // order).
    // (FP32 only: 1.920 -> 1.855 ms per sweep there, while the FP64 sweep, bound by the FP64 pipe and not
    // by chain latency, was 5 % slower in this order.)
    std::vector<int32_t> dirs(s.n_dir);
    for (int q = 0; q < s.n_dir; ++q) dirs[q] = q;
    if (sizeof(Real) == 4)
      std::stable_sort(dirs.begin(), dirs.end(), [&](int a, int b) { return un.n[a] > un.n[b]; });
    std::vector<int32_t> lpt;
    lpt.reserve((size_t)s.n_dir * d.n_chunks);
    for (int q : dirs)
      for (int c = 0; c < d.n_chunks; ++c) lpt.push_back(q * d.n_chunks + c);
    OBTE_TRY(upload(d.lpt, lpt, st));
  }
  OBTE_TRY(upload_real<Real>(d.mfp, s.mfp, st));
  OBTE_TRY(upload_real<Real>(d.tco, s.tco, st));
  OBTE_TRY(upload_real<Real>(d.sig, s.sig, st));
  OBTE_TRY(upload_real<Real>(d.kcoef, s.kcoef, st));
  OBTE_TRY(upload_real<Real>(d.scoef, s.scoef, st));
  if (!s.hs.empty()) OBTE_TRY(upload(d.hs, s.hs, st));
  // per-sweep values (b, p), padded by 32 B for the aligned TMA window
  OBTE_TRY(d.vals.alloc((size_t)s.n_dir * s.n * 2 * sizeof(Real) + 32));
  OBTE_CUDA(cudaMemsetAsync(d.vals.p, 0, d.vals.bytes, st));
  if (s.tf.ok) {   // transmission plans: keep what refresh_tables rewrites
    d.refreshable = true;
  }
  d.ready = true;
  return OBTE_OK;
}

// Element records of a unit on the device: first record, item of its first element, elements.
struct UnitRecs {
  int64_t item0;
  int64_t word0;
  int n_el, a;
};
template <typename Real>
__device__ __forceinline__ UnitRecs unit_recs(const int32_t* __restrict__ desc, int64_t u) {
  const int4 a = reinterpret_cast<const int4*>(desc)[2 * u], b = reinterpret_cast<const int4*>(desc)[2 * u + 1];
  UnitRecs r;
  r.item0 = (int64_t)(unsigned)b.y * (16 / (2 * (int)sizeof(Real))) + (a.x >> 16);
  r.word0 = (int64_t)(unsigned)b.x * (kBlkUnit / 4) + kHeader / 4;
  r.n_el = a.x & 0xFFFF;
  r.a = a.y;
  return r;
}

// New transmissions: rewrite the coefficient words of the records and the wall inflow coefficients of
// the special entries (the same walk over the inflow entries as pack), then P and the contact
// coefficients; indices, units and launch order stay.
// Coefficient word w of item `it`'s record from inflow slot f: g0 x (t_s, 1 - t_s or 1 by the slot's mode),
// the same arithmetic as set_transmission on the host, rounded to the record's precision; the wall inflow (w = -2)
// goes to the item's special entry, in order.  A warp per unit.  (Formed on the host and uploaded, the wall
// coefficients took 7.5 of the 10 ms between two evaluations on 128^2 pixels x 50 x 64, where every item has some.)
template <typename Real, int NF>
__global__ void refresh_rec_kernel(int64_t n_units, int nf, const int32_t* __restrict__ desc, const double* __restrict__ g0,
                                   const int32_t* __restrict__ mode, const int8_t* __restrict__ word,
                                   const double* __restrict__ t, int32_t* __restrict__ blk,
                                   const int32_t* __restrict__ spec, Real* __restrict__ sr) {
  using RR = Rec<Real, NF>;
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t u = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < n_units; u += nw) {
    const UnitRecs ur = unit_recs<Real>(desc, u);
    for (int el = lane; el < ur.n_el; el += 32) {
      const int32_t sp = spec[ur.item0 + el];
      int j = 0;
      for (int f = 0; f < nf; ++f) {
        const int64_t e = (ur.item0 + el) * nf + f;
        const int w = word[e];
        if (w == -1) continue;
        const int32_t md = mode[e];
        const double g = md >= 0 ? g0[e] * t[md] : md == -1 ? g0[e] * 1.0 : g0[e] * (1.0 - t[-md - 2]);
        if (w < 0) {
          sr[(int64_t)sp * SR + j++] = (Real)g;
          continue;
        }
        int32_t* r = blk + ur.word0 + (int64_t)el * RR::W + RR::COEF + w * RR::CSTEP;
        if constexpr (sizeof(Real) == 4) {
          r[0] = __float_as_int((float)g);
        } else {
          r[0] = __double2loint(g);
          r[1] = __double2hiint(g);
        }
      }
    }
  }
}

// The transmission-free factors of a transmission plan on the device (once), and the new t
static obte_status upload_transmission(obte_plan plan, const double* t) {
  const Schedule& s = plan->sched;
  cudaStream_t st = plan->stream;
  if (!plan->tf_g0.p) {
    const int64_t items = (int64_t)s.n_dir * s.n;
    std::vector<int8_t> word((size_t)items * s.nf, -1);
    parallel_for(items, [&](int64_t it) {
      int k = 0;
      for (int f = 0; f < s.nf; ++f) {
        const int kind = (int)((uint32_t)s.in_idx[it * s.nf + f] >> ITEM_SHIFT);
        if (kind == ITEM_CELL || kind == ITEM_PERIODIC) word[(size_t)it * s.nf + f] = (int8_t)k++;
        else if (kind == ITEM_WALL) word[(size_t)it * s.nf + f] = -2;
      }
    });
    OBTE_TRY(upload(plan->tf_g0, s.tf.g0, st));
    OBTE_TRY(upload(plan->tf_mode, s.tf.mode, st));
    OBTE_TRY(upload(plan->tf_word, word, st));
  }
  std::vector<double> tv(t, t + s.n_sides);
  return upload(plan->tf_t, tv, st);
}

__global__ void narrow_kernel(int64_t n, const double* __restrict__ in, float* __restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (float)in[i];
}

// `done`: the FP64 tables, refreshed just before (the FP32 refresh then copies P and narrows the contact
// coefficients on the device instead of uploading them again)
template <typename Real>
static obte_status refresh_impl(obte_plan plan, DevSchedule& d, int64_t* bytes, const DevSchedule* done = nullptr) {
  const Schedule& s = plan->sched;
  cudaStream_t st = plan->stream;
  if (!d.refreshable) { d.ready = false; return OBTE_OK; }   // rebuilt on next use
  const int64_t items = (int64_t)s.n_dir * s.n;
  // the records' coefficient words, on the device from the transmission-free factors and t
  const int blocks = (int)std::min<int64_t>((items + 255) / 256, (int64_t)plan->ctx->num_sms * 8);
  auto kern = s.n_up == 2 ? refresh_rec_kernel<Real, 2> : s.n_up == 3 ? refresh_rec_kernel<Real, 3> : refresh_rec_kernel<Real, 4>;
  if (s.nf != 3 && s.nf != 4) { d.ready = false; return OBTE_OK; }
  kern<<<blocks, 256, 0, st>>>(d.n_units, s.nf, d.desc.as<int32_t>(), plan->tf_g0.as<double>(), plan->tf_mode.as<int32_t>(),
                               plan->tf_word.as<int8_t>(), plan->tf_t.as<double>(), d.blk.as<int32_t>(),
                               d.spec.as<int32_t>(), d.sr.as<Real>());
  count_launch();
  OBTE_CUDA(cudaGetLastError());
  PhaseTimer th(sizeof(Real) == 4 ? "refresh fp32: uploads" : "refresh fp64: uploads");
  const size_t kc_n = std::max<size_t>(s.kcoef.size(), 1);
  const bool reuse = sizeof(Real) == 4 && done && done->Pq.p && d.Pq.bytes == done->Pq.bytes && done->kcoef.p &&
                     d.kcoef.p && d.kcoef.bytes >= kc_n * sizeof(Real) && done->kcoef.bytes >= kc_n * sizeof(double);
  if (reuse) {
    OBTE_CUDA(cudaMemcpyAsync(d.Pq.p, done->Pq.p, s.P.size() * sizeof(double), cudaMemcpyDeviceToDevice, st));
    narrow_kernel<<<(int)std::min<size_t>((kc_n + 255) / 256, 1024), 256, 0, st>>>(
        (int64_t)kc_n, done->kcoef.as<double>(), d.kcoef.as<float>());
    count_launch();
    OBTE_CUDA(cudaGetLastError());
  } else {
    OBTE_CUDA(cudaMemcpyAsync(d.Pq.p, s.P.data(), s.P.size() * sizeof(double), cudaMemcpyHostToDevice, st));
  }
  OBTE_CUDA(wait_stream(st));
  if (!reuse) OBTE_TRY(upload_real<Real>(d.kcoef, s.kcoef, st));
  if (bytes) *bytes += (int64_t)(reuse ? 0 : s.kcoef.size() * sizeof(Real) + s.P.size() * 8);
  return OBTE_OK;
}

// FNV-1a over the packed tables of one precision, built on the host (no device involved).
namespace {
struct Fnv {
  uint64_t h = 1469598103934665603ull;
  void bytes(const void* p, size_t n) {
    const unsigned char* c = static_cast<const unsigned char*>(p);
    for (size_t i = 0; i < n; ++i) h = (h ^ c[i]) * 1099511628211ull;
  }
  template <typename V>
  void vec(const V& v) {
    const uint64_t n = v.size();
    bytes(&n, sizeof n);
    if (n) bytes(v.data(), n * sizeof(v[0]));
  }
  void i(int64_t x) { bytes(&x, sizeof x); }
};
}  // namespace

template <typename Real>
static obte_status tables_digest_impl(const Schedule& s, uint64_t* digest) {
  Shaped sh;
  Packed pk;
  {
    PhaseTimer tp("pack");
    BaseUnits base;
    OBTE_TRY(choose_layout<Real>(s, DeviceShape(), base, sh));
    OBTE_TRY(pack<Real>(s, sh.un, base.un, sh.unit_base, sh.cnt, sh.lay, pk));
  }
  const Units& un = sh.un;
  const std::vector<int64_t>& unit_base = sh.unit_base;
  Fnv f;
  f.vec(un.ptr); f.vec(un.off); f.vec(un.n);
  f.vec(pk.blk); f.vec(pk.cellmap); f.vec(pk.si); f.vec(pk.spec); f.vec(pk.P); f.vec(pk.sr);
  f.vec(pk.desc); f.vec(pk.pfe); f.vec(unit_base);
  f.i(pk.lay.KV); f.i(pk.lay.threads); f.i(pk.lay.nbuf); f.i(pk.lay.emax); f.i(pk.lay.rows);
  // the schedule's own uploads: contact coefficients, K shifts, wall outputs, periodic sources
  f.vec(s.kcoef); f.vec(s.scoef); f.vec(s.kconst); f.vec(s.kshift); f.vec(s.sshift);
  f.vec(s.wo_wall); f.vec(s.wo_off); f.vec(s.x_cell); f.vec(s.x_base); f.vec(s.ell_B);
  *digest = f.h;
  return OBTE_OK;
}

obte_status tables_digest(obte_plan plan, bool fp32, uint64_t* digest) {
  PhaseTimer timer("tables_digest");
  return fp32 ? tables_digest_impl<float>(plan->sched, digest) : tables_digest_impl<double>(plan->sched, digest);
}

obte_status refresh_tables(obte_plan plan, const double* side_transmission, int64_t* bytes) {
  PhaseTimer timer("refresh_tables");
  if (!plan->d32.ready && !plan->d64.ready) return OBTE_OK;
  {
    PhaseTimer tt("refresh: transmissions to the device");
    OBTE_TRY(upload_transmission(plan, side_transmission));
  }
  if (bytes) *bytes += (int64_t)plan->sched.n_sides * 8;
  if (plan->d64.ready) OBTE_TRY(refresh_impl<double>(plan, plan->d64, bytes));
  if (plan->d32.ready) OBTE_TRY(refresh_impl<float>(plan, plan->d32, bytes, plan->d64.ready ? &plan->d64 : nullptr));
  return OBTE_OK;
}
// mfp_m / (1 + mfp_m D) for every (direction, chunk, position, MFP of the chunk) of the FP64 tables, D read
// from the packed records (padded MFPs: 0, as their mfp is 0).  A warp per unit, elements on the lanes.
template <int NF>
__global__ void gain_build_kernel(int64_t n_units, const int32_t* __restrict__ desc, const int32_t* __restrict__ blk,
                                  int64_t n, int n_chunks, int KV, int n_mfp, const double* __restrict__ mfp,
                                  double* __restrict__ out) {
  using RR = Rec<double, NF>;
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t u = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < n_units; u += nw) {
    const UnitRecs ur = unit_recs<double>(desc, u);
    const int64_t q = ur.item0 / n;
    const int total = ur.n_el * KV;
    for (int chunk = 0; chunk < n_chunks; ++chunk)
      for (int i = lane; i < total; i += 32) {
        const int el = i / KV, j = i - el * KV, m = chunk * KV + j;
        const int32_t* r = blk + ur.word0 + (int64_t)el * RR::W;
        const double D = __hiloint2double(r[RR::D + 1], r[RR::D]);
        const double L = m < n_mfp ? mfp[m] : 0.0;
        out[((q * n_chunks + chunk) * n + ur.a) * KV + i] = L / (1.0 + L * D);
      }
  }
}

// The FP64 gain table, unless OBTE_SWEEP64_RINV=0 or it would exceed OBTE_SWEEP64_RINV_GB (default 32) or
// device memory (the sweep then divides)
static obte_status build_gain(obte_plan plan, DevSchedule& d) {
  const Schedule& s = plan->sched;
  if (const char* e = std::getenv("OBTE_SWEEP64_RINV"))
    if (std::atoi(e) == 0) return OBTE_OK;
  double cap_gb = 32.0;
  if (const char* e = std::getenv("OBTE_SWEEP64_RINV_GB")) cap_gb = std::atof(e);
  const int64_t total = (int64_t)s.n_dir * d.n_chunks * s.n * d.mc;
  if ((double)total * 8.0 > cap_gb * 1e9 || (s.nf != 3 && s.nf != 4)) return OBTE_OK;
  if (d.gain.alloc((size_t)total * sizeof(double)) != OBTE_OK) {
    cudaGetLastError();
    d.gain.release();
    return OBTE_OK;            // no room: the sweep divides
  }
  const int blocks = (int)std::min<int64_t>((d.n_units + 7) / 8, (int64_t)plan->ctx->num_sms * 16);
  auto kern = s.n_up == 2 ? gain_build_kernel<2> : s.n_up == 3 ? gain_build_kernel<3> : gain_build_kernel<4>;
  kern<<<std::max(blocks, 1), 256, 0, plan->stream>>>(d.n_units, d.desc.as<int32_t>(), d.blk.as<int32_t>(), s.n,
                                                      d.n_chunks, d.mc, s.n_mfp, d.mfp.as<double>(), d.gain.as<double>());
  count_launch();
  OBTE_CUDA(cudaGetLastError());
  return OBTE_OK;
}

obte_status ensure_tables(obte_plan plan, bool fp32) {
  if (!plan->err.p) {
    OBTE_TRY(plan->err.alloc(sizeof(int)));
    OBTE_CUDA(cudaMemsetAsync(plan->err.p, 0, sizeof(int), plan->stream));
  }
  if (fp32) {
    if (!plan->d32.ready) return upload_tables<float>(plan, plan->d32);
  } else {
    if (!plan->d64.ready) {
      OBTE_TRY(upload_tables<double>(plan, plan->d64));
      OBTE_TRY(build_gain(plan, plan->d64));
    }
  }
  return OBTE_OK;
}

// ---- launch -----------------------------------------------------------------------
// Deterministic reductions requested (OBTE_DETERMINISTIC=1, read per call).
static bool deterministic() {
  const char* e = std::getenv("OBTE_DETERMINISTIC");
  return e && std::atoi(e) != 0;
}

// Tables and partial buffers of the deterministic reductions (plan-level tables once, buffers per precision).
template <typename Real>
static obte_status ensure_det(obte_plan plan, DevSchedule& d) {
  const Schedule& s = plan->sched;
  cudaStream_t st = plan->stream;
  const int64_t n = s.n, n_wo = (int64_t)s.wo_wall.size();
  if (plan->det_nce < 0) {
    std::vector<int32_t> inv((size_t)s.n_dir * n);
    parallel_for(s.n_dir, [&](int64_t q) {
      for (int64_t pos = 0; pos < n; ++pos) inv[(size_t)q * n + s.cell[(size_t)q * n + pos]] = (int32_t)pos;
    });
    std::vector<int32_t> wptr(s.nd + 1, 0), went(std::max<int64_t>(n_wo, 1), 0);
    for (int64_t e = 0; e < n_wo; ++e) wptr[s.wo_wall[e] + 1]++;
    for (int64_t w = 0; w < s.nd; ++w) wptr[w + 1] += wptr[w];
    {
      std::vector<int32_t> fill(wptr.begin(), wptr.end() - 1);
      for (int64_t e = 0; e < n_wo; ++e) went[fill[s.wo_wall[e]]++] = (int32_t)e;   // entry order within a wall
    }
    std::vector<int32_t> ceoff(s.n_dir + 1, 0);
    for (int q = 0; q < s.n_dir; ++q) {
      int32_t cnt = 0;
      for (int64_t pos = 0; pos < n; ++pos) cnt += s.contact[(size_t)q * n + pos] >= 0 ? 1 : 0;
      ceoff[q + 1] = ceoff[q] + cnt;
    }
    OBTE_TRY(upload(plan->det_inv, inv, st));
    OBTE_TRY(upload(plan->det_wptr, wptr, st));
    OBTE_TRY(upload(plan->det_went, went, st));
    OBTE_TRY(upload(plan->det_ceoff, ceoff, st));
    plan->det_nce = ceoff[s.n_dir];
  }
  if (!d.det_d.p) {
    const size_t parts = (size_t)s.n_dir * d.n_chunks * n;
    OBTE_TRY(d.det_d.alloc(parts * sizeof(Real)));
    OBTE_TRY(d.det_j.alloc(parts * s.ds * sizeof(Real)));
    OBTE_TRY(d.det_w.alloc((size_t)std::max<int64_t>(n_wo, 1) * d.n_chunks * sizeof(Real)));
    OBTE_TRY(d.det_k.alloc((size_t)std::max<int64_t>(plan->det_nce, 1) * s.m_pad * sizeof(Real)));
    OBTE_TRY(d.det_s.alloc((size_t)std::max<int64_t>(plan->det_nce, 1) * s.m_pad * sizeof(Real)));
    OBTE_TRY(d.det_S.alloc((size_t)s.n_dir * n * sizeof(double)));
    OBTE_TRY(d.det_SJ.alloc((size_t)s.n_dir * n * s.ds * sizeof(double)));
    // wall partials of entries a chunk does not reach (MFPs beyond n_mfp) stay zero
    OBTE_CUDA(cudaMemsetAsync(d.det_w.p, 0, d.det_w.bytes, st));
  }
  return OBTE_OK;
}

// Scratch of one sweep: the plan's, or the static array's (obte_bte_sweep_static).
template <typename Real>
struct SweepScratch {
  Real* vals;
  int* err;
  Real* xrow;
};

// The per-sweep inputs and the sweep itself (two launches).
template <typename Real, int NF, int KV, bool FINAL, bool DF = false>
static obte_status launch_impl(obte_plan plan, const DevSchedule& d, const SweepScratch<Real>& sc, bool plain,
                               const double* u_in, double* u_out, bool with_src, double* Jraw, double* K, double* S) {
  const Schedule& s = plan->sched;
  cudaStream_t st = plan->stream;
  const bool subset = !plain && !FINAL && plan->sweep_cta_map != nullptr;
  const int batch = subset && plan->sweep_batch > 1 ? plan->sweep_batch : 1;
  PrepParams<Real> r;
  r.cellmap = d.cellmap.as<int32_t>(); r.Pq = d.Pq.as<double>(); r.spec = d.spec.as<int32_t>();
  r.si = d.si.as<int32_t>(); r.sr = d.sr.as<Real>(); r.hs = s.hs.empty() ? nullptr : d.hs.as<double>();
  r.u_in = u_in; r.n = s.n; r.nd = s.nd; r.total = (int64_t)s.n_dir * s.n; r.with_src = with_src ? 1 : 0;
  r.vals = sc.vals; r.pfe = d.pfe.as<int32_t>(); r.n_pf = d.n_pf; r.n_mfp = s.n_mfp; r.m_row = d.n_chunks * KV;
  r.batch = batch; r.batch_stride = batch > 1 ? plan->sweep_batch_stride : 0; r.row_stride = d.row_stride;
  r.xrow = batch > 1 ? static_cast<Real*>(plan->sweep_batch_rows) : sc.xrow;
  r.zero0 = u_out; r.nz0 = s.n + s.nd;
  r.zero1 = FINAL ? Jraw : nullptr; r.nz1 = FINAL ? s.n * s.ds : 0;
  const int64_t sms = plan->ctx->num_sms;
  r.row_blocks = (int)std::min<int64_t>((d.n_pf * batch + 7) / 8, sms * 4);
  const int vblocks = (int)std::max<int64_t>(1, std::min<int64_t>((r.total + 255) / 256, sms * 8));
  sweep_prep_kernel<Real, KV, DF><<<r.row_blocks + vblocks, 256, 0, st>>>(r);
  count_launch();
  OBTE_CUDA(cudaGetLastError());
  auto kern = bte_sweep_kernel<Real, NF, KV, FINAL, DF>;
  // the limit is per kernel, shared by every plan and thread: always the device maximum, so concurrent
  // plans with different footprints cannot lower it under each other's launches
  OBTE_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)plan->ctx->smem_optin));
  SweepParams<Real> p;
  p.n = s.n; p.nd = s.nd; p.n_mfp = s.n_mfp; p.n_dir = s.n_dir; p.ds = s.ds; p.m_pad = s.m_pad;
  p.n_chunks = d.n_chunks; p.zero_row = s.max_slots; p.prow0 = d.prow0; p.emax = d.emax; p.nbuf = d.nbuf;
  p.stage0 = d.stage0; p.stage = d.stage; p.out0 = d.out0; p.out = d.out; p.val_off = d.val_off; p.gain_off = d.gain_off;
  p.blk = d.blk.as<int32_t>(); p.desc = d.desc.as<int32_t>(); p.unit_base = d.unit_base.as<int64_t>();
  p.vals = sc.vals; p.xrow = r.xrow;
  p.mfp = d.mfp.as<Real>(); p.tco = d.tco.as<Real>(); p.sig = d.sig.as<Real>();
  p.kcoef = d.kcoef.as<Real>(); p.scoef = d.scoef.as<Real>();
  p.u_out = u_out; p.Jraw = Jraw; p.K = K; p.S_out = S;
  p.err = sc.err;
  p.gain = (sizeof(Real) == 8 && !DF) ? d.gain.as<double>() : nullptr;
  p.Xs = FINAL ? plan->xstore : nullptr;
  p.xs_add = plan->xstore_add ? 1 : 0;
  p.Xd = FINAL ? plan->xstore64 : nullptr;
  p.skip_unit = plain ? -1 : plan->test_skip_unit;
  p.wait_limit = !plain && plan->test_wait_limit > 0 ? plan->test_wait_limit : kWaitPolls;
  // deterministic reductions: full sweeps of the FP32 and FP64 kernels (not the probes' subset sweeps, not the
  // double-float pass)
  const bool det = !plain && deterministic() && !subset && !DF;
  p.det = det ? 1 : 0;
  p.dpart = p.jpart = p.wpart = p.kpart = p.spart = nullptr;
  p.n_wo = (int64_t)s.wo_wall.size();
  if (det) {
    OBTE_TRY(ensure_det<Real>(plan, const_cast<DevSchedule&>(d)));
    p.dpart = d.det_d.as<Real>();
    p.jpart = d.det_j.as<Real>();
    p.wpart = d.det_w.as<Real>();
    p.kpart = d.det_k.as<Real>();
    p.spart = d.det_s.as<Real>();
  }
  static const bool index_order = std::getenv("OBTE_SWEEP_NO_LPT") != nullptr;   // plain index order
  p.cta_map = subset ? plan->sweep_cta_map : (index_order || DF ? nullptr : d.lpt.as<int32_t>());
  p.n_cta_batch = batch > 1 ? plan->sweep_n_cta : 0;
  p.batch_stride = r.batch_stride;
  p.row_stride = batch > 1 ? d.row_stride : 0;
  const int grid = subset ? plan->sweep_n_cta * batch : s.n_dir * d.n_chunks;
  kern<<<grid, FINAL ? d.final_threads : d.threads, d.smem, st>>>(p);
  count_launch();
  OBTE_CUDA(cudaGetLastError());
  if (det) {
    const int nb = plan->ctx->num_sms * 8;
    const int64_t total = (int64_t)s.n_dir * s.n;
    det_pos_sum_kernel<Real><<<(int)std::min<int64_t>((total + 255) / 256, nb), 256, 0, st>>>(
        d.det_d.as<Real>(), FINAL ? d.det_j.as<Real>() : nullptr, d.n_chunks, s.n, total, s.ds, d.det_S.as<double>(),
        d.det_SJ.as<double>());
    det_elem_sum_kernel<<<(int)std::min<int64_t>((s.n + 255) / 256, nb), 256, 0, st>>>(
        d.det_S.as<double>(), FINAL ? d.det_SJ.as<double>() : nullptr, plan->det_inv.as<int32_t>(), s.n_dir, s.n, s.ds,
        u_out, Jraw);
    count_launch(2);
    if (s.nd > 0) {
      det_wall_sum_kernel<Real><<<(int)std::min<int64_t>((s.nd + 255) / 256, nb), 256, 0, st>>>(
          d.det_w.as<Real>(), d.n_chunks, p.n_wo, plan->det_wptr.as<int32_t>(), plan->det_went.as<int32_t>(), s.nd,
          u_out + s.n);
      count_launch();
    }
    if (FINAL) {
      const int64_t nk = (int64_t)s.n_mfp * s.n_dir;
      det_contact_sum_kernel<Real><<<(int)std::min<int64_t>((nk + 255) / 256, nb), 256, 0, st>>>(
          d.det_k.as<Real>(), d.det_s.as<Real>(), plan->det_ceoff.as<int32_t>(), s.n_dir, s.n_mfp, s.m_pad, K, S);
      count_launch();
    }
    OBTE_CUDA(cudaGetLastError());
  }
  return OBTE_OK;
}

template <typename Real, int KV>
static obte_status launch_kv(obte_plan plan, const DevSchedule& d, const SweepScratch<Real>& sc, bool plain,
                             const double* u_in, double* u_out, bool with_src, bool final_pass, double* Jraw, double* K,
                             double* S) {
  if (plan->sched.n_up == 2) {
    if (final_pass) return launch_impl<Real, 2, KV, true>(plan, d, sc, plain, u_in, u_out, with_src, Jraw, K, S);
    return launch_impl<Real, 2, KV, false>(plan, d, sc, plain, u_in, u_out, with_src, Jraw, K, S);
  }
  if (plan->sched.n_up == 3) {
    if (final_pass) return launch_impl<Real, 3, KV, true>(plan, d, sc, plain, u_in, u_out, with_src, Jraw, K, S);
    return launch_impl<Real, 3, KV, false>(plan, d, sc, plain, u_in, u_out, with_src, Jraw, K, S);
  }
  if (final_pass) return launch_impl<Real, 4, KV, true>(plan, d, sc, plain, u_in, u_out, with_src, Jraw, K, S);
  return launch_impl<Real, 4, KV, false>(plan, d, sc, plain, u_in, u_out, with_src, Jraw, K, S);
}

// plain: no test hook, no deterministic reductions, every CTA (obte_bte_sweep_static)
template <typename Real>
static obte_status launch_shape(obte_plan plan, const DevSchedule& d, const SweepScratch<Real>& sc, bool plain,
                                const double* u_in, double* u_out, bool with_src, bool final_pass, double* Jraw,
                                double* K, double* S) {
  constexpr int N = 16 / (int)sizeof(Real);
  if (d.mc == N) return launch_kv<Real, N>(plan, d, sc, plain, u_in, u_out, with_src, final_pass, Jraw, K, S);
  return launch_kv<Real, 2 * N>(plan, d, sc, plain, u_in, u_out, with_src, final_pass, Jraw, K, S);
}

static obte_status check_shape(const Schedule& s) {
  if (s.ds > 3) { set_error("sigma with more than 3 components"); return OBTE_ERR_UNSUPPORTED; }
  if (s.nf > 4) { set_error("elements with more than 4 sides are not supported"); return OBTE_ERR_UNSUPPORTED; }
  return OBTE_OK;
}

obte_status launch_sweep(obte_plan plan, bool fp32, const double* u_in, double* u_out, bool with_src,
                         bool final_pass, double* Jraw, double* K, double* S) {
  OBTE_TRY(ensure_tables(plan, fp32));
  OBTE_TRY(check_shape(plan->sched));
  if (fp32)
    return launch_shape<float>(plan, plan->d32, {plan->d32.vals.as<float>(), plan->err.as<int>(), plan->d32.xrow.as<float>()},
                               false, u_in, u_out, with_src, final_pass, Jraw, K, S);
  return launch_shape<double>(plan, plan->d64, {plan->d64.vals.as<double>(), plan->err.as<int>(), plan->d64.xrow.as<double>()},
                              false, u_in, u_out, with_src, final_pass, Jraw, K, S);
}

// The output pass in double-float arithmetic on the FP64 tables (J, K and S accumulated like a final pass).
obte_status launch_sweep_df(obte_plan plan, const double* u_in, double* u_out, bool with_src, double* Jraw, double* K,
                            double* S) {
  OBTE_TRY(ensure_tables(plan, false));
  OBTE_TRY(check_shape(plan->sched));
  const DevSchedule& d = plan->d64;
  const SweepScratch<double> sc{d.vals.as<double>(), plan->err.as<int>(), d.xrow.as<double>()};
  if (d.mc == 2) {
    if (plan->sched.n_up == 2) return launch_impl<double, 2, 2, true, true>(plan, d, sc, false, u_in, u_out, with_src, Jraw, K, S);
    if (plan->sched.n_up == 3) return launch_impl<double, 3, 2, true, true>(plan, d, sc, false, u_in, u_out, with_src, Jraw, K, S);
    return launch_impl<double, 4, 2, true, true>(plan, d, sc, false, u_in, u_out, with_src, Jraw, K, S);
  }
  if (plan->sched.n_up == 2) return launch_impl<double, 2, 4, true, true>(plan, d, sc, false, u_in, u_out, with_src, Jraw, K, S);
  if (plan->sched.n_up == 3) return launch_impl<double, 3, 4, true, true>(plan, d, sc, false, u_in, u_out, with_src, Jraw, K, S);
  return launch_impl<double, 4, 4, true, true>(plan, d, sc, false, u_in, u_out, with_src, Jraw, K, S);
}

// Device error word: nonzero after a bounded wait gave up (cleared on read).
obte_status check_device_error(obte_plan plan) {
  if (!plan->err.p) return OBTE_OK;
  int h = 0;
  OBTE_CUDA(cudaMemcpyAsync(&h, plan->err.p, sizeof(int), cudaMemcpyDeviceToHost, plan->stream));
  OBTE_CUDA(wait_stream(plan->stream));
  if (h) {
    OBTE_CUDA(cudaMemsetAsync(plan->err.p, 0, sizeof(int), plan->stream));
    set_error("a device-side wait timed out in a sweep or a diffusion correction");
    return OBTE_ERR_DEVICE_TIMEOUT;
  }
  return OBTE_OK;
}
}  // namespace obte

// ---- sweep on library-owned static scratch ---------------------------------------------
//
// obte_bte_sweep keeps its per-sweep scratch (the (b, p) values the sweep kernel streams by TMA, the periodic inflow
// rows and the device error word) in buffers the plan allocates on first use.  Some callers
// cannot allocate device memory when they sweep: a host framework that has reserved nearly
// all of the GPU's memory for its own pool (cudaMalloc then fails or forces that pool to give
// memory back), or a latency-bound loop in which cudaMalloc / cudaFree would synchronise the
// device and stall work on other streams.  obte_bte_sweep_static runs the same two kernels
// with the values and the error word in the fixed array below instead and the inflow rows that came with the plan's
// tables, and allocates nothing.
//
// The array is a file-scope __device__ variable: every GPU that loads this library holds
// kStaticScratchBytes of it until the process exits.  Its name in host code is only a
// host-side stand-in, so host code passes the kernels the device address that
// cudaGetSymbolAddress returns, looked up once per device (with that device current) on
// the first call on that device.  Layout: [0, 256) device error word, [256, ...) the values.
// All calls share the array, and it keeps the previous call's contents; each call clears
// the error word before its kernels run, and the values are written in full by
// sweep_prep_kernel before the sweep kernel reads them.
namespace obte {

static constexpr size_t kStaticScratchBytes = (size_t)8 << 20;
static constexpr size_t kStaticValsOffset = 256;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_static_mu;
void* g_static_addr[kMaxDevices] = {};
}  // namespace

// Device address of g_static_scratch on `device`, which must be the current device.
static obte_status static_scratch_address(int device, void** out) {
  if (device < 0 || device >= kMaxDevices) { set_error("device ordinal out of range"); return OBTE_ERR_BAD_ARG; }
  std::lock_guard<std::mutex> lock(g_static_mu);
  if (!g_static_addr[device]) {
    void* p = nullptr;
    OBTE_CUDA(cudaGetSymbolAddress(&p, g_static_scratch));
    g_static_addr[device] = p;
  }
  *out = g_static_addr[device];
  return OBTE_OK;
}

// Runs with the plan's device current; the caller restores its own.
static obte_status sweep_static_on_device(obte_plan plan, bool fp32, const double* u_in, double* u_out,
                                          bool with_src) {
  cudaStream_t st = plan->stream;
  void* base = nullptr;
  OBTE_TRY(static_scratch_address(plan->ctx->device, &base));
  int* err = static_cast<int*>(base);
  void* vals = static_cast<unsigned char*>(base) + kStaticValsOffset;
  OBTE_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
  if (fp32)
    OBTE_TRY(launch_shape<float>(plan, plan->d32, {static_cast<float*>(vals), err, plan->d32.xrow.as<float>()}, true, u_in,
                                 u_out, with_src, false, nullptr, nullptr, nullptr));
  else
    OBTE_TRY(launch_shape<double>(plan, plan->d64, {static_cast<double*>(vals), err, plan->d64.xrow.as<double>()}, true,
                                  u_in, u_out, with_src, false, nullptr, nullptr, nullptr));
  int h = 0;
  OBTE_CUDA(cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, st));
  OBTE_CUDA(cudaStreamSynchronize(st));
  if (h) {
    set_error("a device-side wait timed out in the sweep kernel");
    return OBTE_ERR_DEVICE_TIMEOUT;
  }
  return OBTE_OK;
}

}  // namespace obte

using namespace obte;

extern "C" obte_status obte_bte_sweep_static(obte_plan plan, int32_t precision, const double* u_in, double* u_out,
                                             int32_t with_source) {
  if (!plan || !u_in || !u_out) { set_error("null argument"); return OBTE_ERR_BAD_ARG; }
  if (!plan->ctx) { set_error("host-only plan cannot sweep"); return OBTE_ERR_BAD_ARG; }
  if (precision != OBTE_FP64 && precision != OBTE_FP32 && precision != OBTE_FP32_REFINE) {
    set_error("bad precision"); return OBTE_ERR_BAD_ARG;
  }
  const Schedule& s = plan->sched;
  const bool fp32 = precision != OBTE_FP64;
  const size_t need = kStaticValsOffset + (size_t)s.n_dir * (size_t)s.n * 2 * (fp32 ? sizeof(float) : sizeof(double)) + 32;
  if (need > kStaticScratchBytes) {
    set_error("obte_bte_sweep_static: this problem needs " + std::to_string(need) + " bytes of scratch (n_dir x n_elems x " +
              std::to_string(fp32 ? 8 : 16) + " + 288), more than the " + std::to_string(kStaticScratchBytes) +
              " bytes of static scratch the library holds; use obte_bte_sweep");
    return OBTE_ERR_UNSUPPORTED;
  }
  if (s.ds > 3) { set_error("sigma with more than 3 components"); return OBTE_ERR_UNSUPPORTED; }
  if (s.nf > 4) { set_error("elements with more than 4 sides are not supported"); return OBTE_ERR_UNSUPPORTED; }
  if (!(fp32 ? plan->d32.ready : plan->d64.ready)) {
    set_error("obte_bte_sweep_static: the plan's device tables for this precision are not built yet; building them "
              "allocates, so run obte_bte_sweep or obte_bte_solve once in this precision at set-up");
    return OBTE_ERR_BAD_ARG;
  }
  int prev = -1;
  OBTE_CUDA(cudaGetDevice(&prev));
  if (prev != plan->ctx->device) OBTE_CUDA(cudaSetDevice(plan->ctx->device));
  const obte_status rc = sweep_static_on_device(plan, fp32, u_in, u_out, with_source != 0);
  if (prev != plan->ctx->device) {
    const cudaError_t e = cudaSetDevice(prev);
    if (rc == OBTE_OK && e != cudaSuccess) return cuda_fail(e, "cudaSetDevice", __FILE__, __LINE__);
  }
  return rc;
}
