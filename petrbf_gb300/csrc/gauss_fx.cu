// gauss_fx.cu -- the FP64 truncated Gaussian sums with fixed-point exponents (gauss_fx.cuh).
//
//   w_i = sum_{j in T(c(i))} g_j exp(-|x_i - x_j|^2 / (2 sigma^2)) / (2 pi sigma^2)
//
// The sources carry fixed-point coordinates and 64-bit box-test words, so no FP64 coordinate
// is read and the truncation filter is integer work; a pair's exponential is about forty
// integer instructions (fx_pow2_bits) and FP64 holds what it always held -- the weights, the
// products and the sums, one fused multiply-add per pair and vector.
//
// One CTA works on items (target cell, tile of targets) in rounds of the grid, a tile in passes
// of CfgX::TT targets. A producer warp brings the neighbour columns' sources into shared memory
// (bulk copies on an mbarrier, the next piece in flight while one is filtered), keeps those of
// the cell's truncation set in order, and hands them on in two buffers of CfgX::KC sources. The
// consumer warps own an even share of the pass's targets, at most CfgX::TG each, whose sums
// stay in registers; their lanes stride over a buffer's sources. Nothing but the buffers'
// mbarriers joins the warps: with CTA barriers around the filtering they spent a fifth of their
// time waiting there.
// Measured against the FP64-pipe kernels of gauss.cu (one product, caller order): 2D, 4x10^6
// points 44.7 -> 7.9 ms (79.8 -> 450 Gpairs/s); 3D, 96^3 points 180.7 -> 17.8 ms (39.5 -> 400).
// What bounds it: the FP64 accumulations take 16 of the 23 (2D) to 27 (3D) clocks an SM spends
// per 32 pairs; the shared-memory lookups (14), the integer pipes (10 to 13) and the issue of
// about 50 instructions (12) overlap with them, 24 warps an SM not hiding all of it.
//
// Symmetric form (2D, targets = sources, cells of at most kTileT points): the pair (i, j)
// enters row i when j is in T(c(i)) and row j when i is in T(c(j)), with the same
// exponential. A CTA per cell c1 takes its own points against themselves (both rows, one
// after the other) and against the points of the upper half of its neighbour window, adding
// row j's share into per-warp sums in shared memory; another warp puts their totals into
// part[pass][o][j], o the window offset (one writer per slot), for k_sym_gather to add to the
// rows. A pair of rows then costs one exponential and two fused multiply-adds, and the FP64
// pipe bounds it (85 % busy; a fifth of that is the row-j totals, the trees that end the
// targets' sums and lanes past a buffer's end).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>
#include <vector>

#include "gauss_common.cuh"
#include "gauss_fx.cuh"

namespace prbf {
namespace {

// Warps of a CTA that sum; the next one is the producer and the symmetric form's last one adds
// up the row-j sums. One-sided: 24 warps an SM, 80 registers (9, 10, 11, 12 warps a CTA took
// 8.48, 8.39, 9.00, 8.07 ms on 4x10^6 points in 2D, 5.47, 5.69, 5.75, 5.31 ms on 64^3 in 3D);
// symmetric: 20 warps, 96 registers (10 and 12 warps a CTA: 8.31, 8.59 ms).
template <bool SYM>
constexpr int kCons = SYM ? 8 : 11;
template <bool SYM>
constexpr int kFxThreads = 32 * (kCons<SYM> + (SYM ? 2 : 1));
constexpr int kResident = 2 * 152;  // CTAs resident on the GPU
constexpr int kJoin = 2;            // buffers from one joining of the lanes' sums to the next

__device__ uint2 d_fx_t1[kFxTab], d_fx_t2[kFxTab];

// Targets per consumer warp, sources per buffer and per staged piece, for two CTAs per SM. One
// vector: the sums of up to eight targets stay in registers and the buffer is walked for four
// at a time, whose coordinates (and, symmetric form, weights and words) are reloaded for each
// walk -- with all eight held, the 3D kernel's registers left too few chains in flight. More
// vectors: four targets (the sums are NV times as many).
template <int DIM, int NV, bool SYM>
struct CfgX {
  static constexpr int TG = NV == 1 ? 8 : 4;
  static constexpr int TT = TG * kCons<SYM>;  // targets per pass over the sources
  static constexpr int KC = SYM ? 256 : (NV == 1 ? 512 : 384);
  static constexpr int RC = 256;
};

template <int DIM, int NV, bool SYM>
struct LayoutX {
  using C = CfgX<DIM, NV, SYM>;
  static constexpr int NA = DIM + NV + 1;  // staged arrays: coordinates, weights, box-test word
  static constexpr size_t raw = 0;                                                   // 2 x NA x RC
  static constexpr size_t comp = align16(raw + 8 * (size_t)2 * NA * C::RC);           // 2 x (DIM + NV) x KC
  static constexpr size_t code = align16(comp + 8 * (size_t)2 * (DIM + NV) * C::KC);  // SYM: 2 x KC (M, j)
  static constexpr size_t accj = align16(code + (SYM ? 8 * (size_t)2 * C::KC : 0));   // SYM: 2 x 8 x KC
  static constexpr size_t tab1 = align16(accj + (SYM ? 8 * (size_t)2 * kCons<SYM> * C::KC : 0));
  static constexpr size_t tab2 = align16(tab1 + 8 * (size_t)kFxTab);
  // per consumer warp and target: coordinates and (SYM) weight and box-test word
  static constexpr int TW = DIM + (SYM ? 2 : 0);
  static constexpr size_t tgt = align16(tab2 + 8 * (size_t)kFxTab);
  // one-sided: a target's running totals, each with what its additions rounded away
  static constexpr size_t tot = align16(tgt + 8 * (size_t)TW * C::TT);
  static constexpr size_t total = align16(tot + (SYM ? 0 : 16 * (size_t)NV * C::TT));
};

// exp of a pair: coordinates (l, h) of target and source
template <int DIM, bool WIDE>
__device__ __forceinline__ double fx_pair(const uint2 (&t)[DIM], const uint2 (&s)[DIM], const uint2* t1,
                                          const uint2* t2) {
  const unsigned long long B = fx_exponent<DIM, WIDE>(t, s);
  const unsigned bh = (unsigned)(B >> 32);
  const uint2 p = t1[(bh >> 11) & 2047u], q = t2[bh & 2047u];
  return __longlong_as_double((long long)fx_pow2_bits(bh, (unsigned)B, p, q));
}


// The lanes' sums of N <= 8 values over the warp, by a butterfly that halves the values each
// lane carries while there are two or more (N = 8: 9 FP64 adds a lane instead of 8 x 5). Lane l
// returns the total of value *which (-1: of none). Every value is added up in the same order
// whatever N: neighbouring lanes first.
template <int N>
__device__ __forceinline__ double fx_scatter_sum(const double (&a)[N], int lane, int& which) {
  constexpr unsigned F = 0xffffffffu;
  constexpr int P = N > 4 ? 8 : (N > 2 ? 4 : N);  // values carried, padded with zeros
  double k[P];
#pragma unroll
  for (int i = 0; i < P; i++) k[i] = i < N ? a[i] : 0.0;
  which = 0;
  int bit = 1;
#pragma unroll
  for (int h = P / 2; h >= 1; h /= 2) {
    const bool up = lane & bit;
#pragma unroll
    for (int i = 0; i < h; i++) {
      const double mine = up ? k[i + h] : k[i], other = up ? k[i] : k[i + h];
      k[i] = mine + __shfl_xor_sync(F, other, bit);
    }
    which += up ? h : 0;
    bit <<= 1;
  }
  for (; bit < 32; bit <<= 1) k[0] += __shfl_xor_sync(F, k[0], bit);
  if (lane >= P || which >= N) which = -1;  // (lanes that differ in the other bits hold the same total)
  return k[0];
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// What the warps of a CTA share besides the data.
struct FxShared {
  uint64_t raw_bar[2], full[2], empty[2], drained[2];
  int n[2];        // sources of a buffer
  int last[2];     // the last buffer of a pass
  int self[2];     // symmetric form: the cell's own points (no row-j sums)
  int pass[2];     // symmetric form: the cell's pass, with slots of its own
  double norm[2];  // symmetric form
};

struct FxArgs {
  const uint2 *tx, *ty, *tz, *sx, *sy, *sz;
  const unsigned long long* smask;
  const double* sg;
  long long vs;
  double* w;
  double* part;
  long long pstride;
  int K, n, ncs, tile;
  VecSkip left;
};

// One pass of a consumer warp with N targets from t: buffers until the last one. Returns false
// when a wait gave up.
template <int DIM, int NV, bool SYM, bool WIDE, int N>
__device__ __forceinline__ bool fx_consume(unsigned char* smem, FxShared& sh, const FxArgs& a, const int (&vm)[NV],
                                           int t, double norm, int wid, int lane, int& b, unsigned& ph) {
  using Lay = LayoutX<DIM, NV, SYM>;
  using C = CfgX<DIM, NV, SYM>;
  constexpr int KC = C::KC;
  // sets of targets that share a walk over the buffer
  constexpr int NA_ = N > 4 || SYM ? (N + 1) / 2 : N, NB_ = N - NA_;
  const uint2 *t1 = (const uint2*)(smem + Lay::tab1), *t2 = (const uint2*)(smem + Lay::tab2);
  double acc[NV][N > 0 ? N : 1];
#pragma unroll
  for (int v = 0; v < NV; v++)
#pragma unroll
    for (int k = 0; k < N; k++) acc[v][k] = 0.0;
  constexpr int TW = Lay::TW;
  uint2* tw = (uint2*)(smem + Lay::tgt) + wid * C::TG * TW;
  double2* tot = (double2*)(smem + Lay::tot) + wid * C::TG * NV;
  if (lane < N) {
    if constexpr (!SYM)
#pragma unroll
      for (int v = 0; v < NV; v++) tot[lane * NV + v] = make_double2(0.0, 0.0);
    tw[lane * TW] = a.tx[t + lane];
    tw[lane * TW + 1] = a.ty[t + lane];
    if constexpr (DIM == 3) tw[lane * TW + 2] = a.tz[t + lane];
    if constexpr (SYM) {
      ((double*)tw)[lane * TW + DIM] = a.sg[t + lane];
      tw[lane * TW + DIM + 1] = make_uint2((unsigned)a.smask[t + lane], 0u);
    }
  }
  __syncwarp();
  // after every kJoin buffers (one-sided form) the lanes' sums meet and join their target's
  // running total, which keeps what its additions round away: the lanes' partial sums stay short,
  // as rounding grows with their length (a 3D target has some 10^4 sources), and the additions at
  // the total's full size, one per join, cost nothing of it. (The totals lie in shared memory; in
  // registers the 3D kernel spills, 18.0 against 17.8 ms on 96^3. With joins after 1, 2, 3, 4
  // buffers the product took 18.2, 17.8, 17.7, 17.6 ms; three already lose on 40^3 points what the
  // kept roundings gain.)
  double sum[NV];
  int which = -1, held = 0;
  auto join = [&]() {
    if constexpr (N > 0) {
#pragma unroll
      for (int v = 0; v < NV; v++) {
        sum[v] = fx_scatter_sum<N>(acc[v], lane, which);
#pragma unroll
        for (int k = 0; k < N; k++) acc[v][k] = 0.0;
        if (!SYM && which >= 0) {
          double2 q = tot[which * NV + v];
          const double run = q.x + sum[v], d = run - q.x;
          q.y += (q.x - (run - d)) + (sum[v] - d);
          q.x = run;
          tot[which * NV + v] = q;
        }
      }
    }
  };
  while (true) {
    if (!mbar_wait(&sh.full[b], ph)) return false;
    const int n = sh.n[b];
    const bool last = sh.last[b] != 0, self = SYM && sh.self[b] != 0;
    const uint2* comp = (const uint2*)(smem + Lay::comp) + b * (DIM + NV) * KC;
    const double* cg = (const double*)(comp + DIM * KC);
    if constexpr (N > 0) {
      auto walk = [&](auto k0c, auto cnt, auto row_j) {
        constexpr int K0 = decltype(k0c)::value, CNT = decltype(cnt)::value;
        constexpr bool RJ = decltype(row_j)::value;
        uint2 tc[CNT][DIM];
        double tg[RJ ? CNT : 1];
        unsigned tm[RJ ? CNT : 1];
#pragma unroll
        for (int k = 0; k < CNT; k++) {
#pragma unroll
          for (int d = 0; d < DIM; d++) tc[k][d] = tw[(K0 + k) * TW + d];
          if constexpr (RJ) {
            tg[k] = ((const double*)tw)[(K0 + k) * TW + DIM];
            tm[k] = tw[(K0 + k) * TW + DIM + 1].x;
          }
        }
        for (int j = lane; j < n; j += 32) {
          uint2 sc[DIM];
          double g[NV];
#pragma unroll
          for (int d = 0; d < DIM; d++) sc[d] = comp[d * KC + j];
#pragma unroll
          for (int v = 0; v < NV; v++) g[v] = cg[v * KC + j];
          unsigned M = 0;
          double aj = 0.0;
          double* pj = nullptr;
          if constexpr (RJ) {
            M = ((const unsigned*)(smem + Lay::code))[b * 2 * KC + j];
            pj = (double*)(smem + Lay::accj) + (b * kCons<SYM> + wid) * KC + j;
            if constexpr (K0 > 0) aj = *pj;
          }
#pragma unroll
          for (int k = 0; k < CNT; k++) {
            const double e = fx_pair<DIM, WIDE>(tc[k], sc, t1, t2);
#pragma unroll
            for (int v = 0; v < NV; v++) acc[v][K0 + k] = fma(g[v], e, acc[v][K0 + k]);
            // row j, when target k is in T(c(j)): both its bits at c(j)'s offset
            if constexpr (RJ) aj = fma((~tm[k] & M) == 0 ? tg[k] : 0.0, e, aj);
          }
          if constexpr (RJ) *pj = aj;
        }
      };
      using Z = std::integral_constant<int, 0>;
      using A = std::integral_constant<int, NA_>;
      using B = std::integral_constant<int, NB_>;
      if (!SYM || self) {
        walk(Z(), A(), std::false_type());
        if constexpr (NB_ > 0) walk(A(), B(), std::false_type());
      } else {
        walk(Z(), A(), std::integral_constant<bool, SYM>());
        if constexpr (NB_ > 0) walk(A(), B(), std::integral_constant<bool, SYM>());
      }
    } else if constexpr (SYM) {
      double* pj = (double*)(smem + Lay::accj) + (b * kCons<SYM> + wid) * KC;
      for (int j = lane; j < n; j += 32) pj[j] = 0.0;
    }
    __syncwarp();  // the lanes' reads (and sums) of the buffer are done
    if (lane == 0) mbar_arrive(&sh.empty[b]);
    ph ^= b;
    b ^= 1;
    if constexpr (SYM) {
      if (last) join();
    } else {
      if (last || ++held == kJoin) {
        join();
        held = 0;
      }
    }
    if (last) break;
  }
  if (N > 0 && which >= 0) {
#pragma unroll
    for (int v = 0; v < NV; v++) {
      if constexpr (!SYM) {  // (an infinite total leaves no number in what it rounded away)
        const double2 q = tot[which * NV + v];
        sum[v] = q.y == q.y ? q.x + q.y : q.x;
      }
      a.w[vm[v] * a.vs + t + which] = sum[v] * norm;
    }
  }
  if constexpr (!SYM) __syncwarp();  // the totals are read: the next pass may clear them
  return true;
}

// Range r of the symmetric walk of cell c1 (2D): 0 = c1 itself, 1 = the cells above it in its
// column, then the columns to its right. Sorted positions [pa, pb), column offset dx.
__device__ __forceinline__ void fx_sym_range(const Grid& g, const int* __restrict__ cs, int r, int c1, int ix, int iy,
                                             int jy0, int jy1, int& pa, int& pb, int& dx) {
  dx = r < 2 ? 0 : r - 1;
  if (r == 0) {
    pa = cs[c1];
    pb = cs[c1 + 1];
    return;
  }
  const int y0 = r == 1 ? iy + 1 : jy0;
  pa = pb = 0;
  if (y0 > jy1) return;
  const int ca = g.cbase + cell_of(g, ix + dx, y0, 0);
  pa = cs[ca];
  pb = cs[ca + (jy1 - y0) + 1];
}

template <int DIM, int NV, bool BATCH, bool SYM, bool WIDE>
__global__ void __launch_bounds__(kFxThreads<SYM>, 2) k_gauss_fx(Grid g0, const Grid* __restrict__ grids,
                                                           const int* __restrict__ cprob, SegSkip seg,
                                                           const int2* __restrict__ items, int nitems,
                                                           const int* __restrict__ cs_t,
                                                           const int* __restrict__ cs_s, FxArgs a, unsigned* err,
                                                           const int* __restrict__ skip) {
  if (skip && *skip) return;
  int vm[NV];
  if (!vec_map<NV>(a.left, vm)) return;
  using Lay = LayoutX<DIM, NV, SYM>;
  using C = CfgX<DIM, NV, SYM>;
  constexpr int NA = Lay::NA, RC = C::RC, KC = C::KC, TT = C::TT;
  static_assert(!SYM || (DIM == 2 && NV == 1 && TT == kFxSymTile), "the symmetric form is 2D, one vector");
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ FxShared sh;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int i = tid; i < kFxTab / 2; i += kFxThreads<SYM>) {
    ((uint4*)(smem + Lay::tab1))[i] = ((const uint4*)d_fx_t1)[i];
    ((uint4*)(smem + Lay::tab2))[i] = ((const uint4*)d_fx_t2)[i];
  }
  if (tid == 0)
    for (int q = 0; q < 2; q++) {
      mbar_init(&sh.raw_bar[q], 1);
      mbar_init(&sh.full[q], 1);
      mbar_init(&sh.empty[q], kCons<SYM>);
      mbar_init(&sh.drained[q], 1);
    }
  __syncthreads();
  const int G = gridDim.x;
  int b = 0, rb = 0;             // the buffer, and (producer) the raw piece, in turn
  unsigned ph = 0, rph = 0;      // their phases
  unsigned long long* raw = (unsigned long long*)(smem + Lay::raw);

  // the row-j sums of a buffer that the consumers have left, their warps' shares in warp
  // order, into the slots of the sources' offsets
  auto drain = [&](int bb) {
    if constexpr (SYM) {
      const double* s = (const double*)(smem + Lay::accj) + bb * kCons<SYM> * KC;
      const unsigned *cm = (const unsigned*)(smem + Lay::code) + bb * 2 * KC, *cj = cm + KC;
      const int nb = g0.nb_trunc, W = 2 * nb + 1;  // (a batch's grids have the same window)
      const double norm = sh.norm[bb];
      const int nn = sh.self[bb] ? 0 : sh.n[bb];
      double* part = a.part + (long long)sh.pass[bb] * a.K * a.pstride;
#pragma unroll 2
      for (int i = lane; i < nn; i += 32) {
        const unsigned M = cm[i];
        if (M == 0xffffffffu) continue;  // an own point: its row is summed as a target
        const int ddx = nb - (__ffs(M) - 1), ddy = nb - (31 - __clz(M) - kMaskY);
        const int key = ddx * W + ddy, j = (int)cj[i];  // key > 0 in the upper half of the window
        if (key >= 1 && key <= a.K && j < a.n) {
          double v = s[i];
#pragma unroll
          for (int u = 1; u < kCons<SYM>; u++) v += s[u * KC + i];
          part[(long long)(key - 1) * a.pstride + j] = v * norm;
        } else {
          atomicOr(err, DEV_ERR_INDEX);
        }
      }
      __syncwarp();
    }
  };

  for (int round = 0; (long long)round * G < nitems; round++) {
    const int it = (round & 1) ? round * G + (G - 1 - (int)blockIdx.x) : round * G + (int)blockIdx.x;
    if (it >= nitems) continue;
    const int2 item = items[it];
    const int ic = item.x, t0 = item.y;
    if (ic < 0 || ic + 1 >= a.ncs) {  // bounds check: record and skip the item
      if (tid == 0) atomicOr(err, DEV_ERR_INDEX);
      continue;
    }
    Grid g = g0;
    if constexpr (BATCH) {
      if (seg.cell_done(ic)) continue;  // a stopped problem (uniform over the CTA)
      g = grids[cprob[ic]];
    }
    const int nt_all = min(BATCH ? a.tile : kTileT, cs_t[ic + 1] - t0);
    const int passes = (nt_all + TT - 1) / TT;
    const double norm = g.norm;
    for (int q = blockIdx.y; q < passes; q += gridDim.y) {
      const int ta = nt_all * q / passes, nt = nt_all * (q + 1) / passes - ta;
      if (wid < kCons<SYM>) {
        const int u0 = nt * wid / kCons<SYM>, cnt = nt * (wid + 1) / kCons<SYM> - u0;
        const int t = t0 + ta + u0;
        bool ok;
        switch (cnt) {
          case 0: ok = fx_consume<DIM, NV, SYM, WIDE, 0>(smem, sh, a, vm, t, norm, wid, lane, b, ph); break;
          case 1: ok = fx_consume<DIM, NV, SYM, WIDE, 1>(smem, sh, a, vm, t, norm, wid, lane, b, ph); break;
          case 2: ok = fx_consume<DIM, NV, SYM, WIDE, 2>(smem, sh, a, vm, t, norm, wid, lane, b, ph); break;
          case 3: ok = fx_consume<DIM, NV, SYM, WIDE, 3>(smem, sh, a, vm, t, norm, wid, lane, b, ph); break;
          case 4: ok = fx_consume<DIM, NV, SYM, WIDE, 4>(smem, sh, a, vm, t, norm, wid, lane, b, ph); break;
          default:
            if constexpr (C::TG == 8) {
              switch (cnt) {
                case 5: ok = fx_consume<DIM, NV, SYM, WIDE, 5>(smem, sh, a, vm, t, norm, wid, lane, b, ph); break;
                case 6: ok = fx_consume<DIM, NV, SYM, WIDE, 6>(smem, sh, a, vm, t, norm, wid, lane, b, ph); break;
                case 7: ok = fx_consume<DIM, NV, SYM, WIDE, 7>(smem, sh, a, vm, t, norm, wid, lane, b, ph); break;
                default: ok = fx_consume<DIM, NV, SYM, WIDE, 8>(smem, sh, a, vm, t, norm, wid, lane, b, ph); break;
              }
            } else {
              ok = false;  // (not reached: at most TG targets a warp)
            }
        }
        if (!ok) {
          if (lane == 0) atomicOr(err, DEV_ERR_TIMEOUT);
          return;
        }
        continue;
      }
      if (wid > kCons<SYM>) {  // symmetric form: the row-j sums
        bool last = false;
        while (!last) {
          if (!mbar_wait(&sh.empty[b], ph)) {
            if (lane == 0) atomicOr(err, DEV_ERR_TIMEOUT);
            return;
          }
          last = sh.last[b] != 0;
          drain(b);
          if (lane == 0) mbar_arrive(&sh.drained[b]);
          ph ^= b;
          b ^= 1;
        }
        continue;
      }
      // ---- producer ----------------------------------------------------------------------
      const int cb = g.cbase, nb = g.nb_trunc;
      int ix, iy, iz;
      cell_xyz(g, ic - cb, ix, iy, iz);
      const int c0 = cs_s[ic], c1 = cs_s[ic + 1];
      const int jx0 = max(0, ix - nb), jx1 = min(g.nx - 1, ix + nb);
      const int jy0 = max(0, iy - nb), jy1 = min(g.ny - 1, iy + nb);
      const int jz0 = DIM == 3 ? max(0, iz - nb) : 0, jz1 = DIM == 3 ? min(g.nz - 1, iz + nb) : 0;
      const int ncolx = jx1 - jx0 + 1;
      const int nranges = SYM ? 2 + (jx1 - ix) : ncolx * (jz1 - jz0 + 1);
      unsigned tor = 0;  // symmetric form: the box-test bits any of the cell's points has
      if constexpr (SYM) {
        for (int i = c0 + lane; i < c1; i += 32) tor |= (unsigned)a.smask[i];
        tor = __reduce_or_sync(0xffffffffu, tor);
      }
      // ranges: the source columns of the window, 32 at a time in the lanes' registers
      int ra = 0, re = 0, rbase = -32;
      int r = 0, p = -1;
      auto next_piece = [&](int& s, int& cnt, int& pr) {
        cnt = 0;
        while (r < nranges) {
          if (r >= rbase + 32) {
            rbase = r;
            const int q = r + lane;
            ra = re = 0;
            if (q < nranges) {
              if constexpr (SYM) {
                int dx;
                fx_sym_range(g, cs_s, q, ic, ix, iy, jy0, jy1, ra, re, dx);
              } else {
                const int jx = jx0 + q % ncolx, jz = jz0 + q / ncolx;
                ra = cs_s[cb + cell_of(g, jx, jy0, jz)];
                re = cs_s[cb + cell_of(g, jx, jy1, jz) + 1];
              }
              if (ra < 0 || re > a.n || ra > re) {  // bounds check: record and skip the range
                atomicOr(err, DEV_ERR_INDEX);
                ra = re = 0;
              }
            }
          }
          const int x = __shfl_sync(0xffffffffu, ra, r - rbase), y = __shfl_sync(0xffffffffu, re, r - rbase);
          if (p < 0) p = x;
          if (p >= y) {
            r++;
            p = -1;
            continue;
          }
          s = p;
          pr = r;
          p = min(y, (s & ~1) + RC);
          cnt = p - s;
          return;
        }
      };
      auto issue = [&](int s, int cnt, int slot) {  // 16-byte aligned copies of 8-byte elements
        __syncwarp();
        if (lane == 0) {
          const int s_al = s & ~1, len = ((s + cnt + 1) & ~1) - s_al;
          unsigned long long* dst = raw + slot * NA * RC;
          fence_proxy_async_smem();
          mbar_expect_tx(&sh.raw_bar[slot], (unsigned)len * 8u * NA);
          bulk_g2s(dst, a.sx + s_al, len * 8u, &sh.raw_bar[slot]);
          bulk_g2s(dst + RC, a.sy + s_al, len * 8u, &sh.raw_bar[slot]);
          if (DIM == 3) bulk_g2s(dst + 2 * RC, a.sz + s_al, len * 8u, &sh.raw_bar[slot]);
#pragma unroll
          for (int v = 0; v < NV; v++)
            bulk_g2s(dst + (DIM + v) * RC, a.sg + vm[v] * a.vs + s_al, len * 8u, &sh.raw_bar[slot]);
          bulk_g2s(dst + (DIM + NV) * RC, a.smask + s_al, len * 8u, &sh.raw_bar[slot]);
        }
      };
      int n = -1;  // sources in the buffer being filled (-1: not taken yet)
      bool own_part = true;  // symmetric form: only the cell's own points so far
      auto acquire = [&]() -> bool {
        if (!mbar_wait(SYM ? &sh.drained[b] : &sh.empty[b], ph ^ 1u)) return false;
        n = 0;
        return true;
      };
      auto publish = [&](bool last, bool own = false) {
        __syncwarp();
        if (lane == 0) {
          sh.n[b] = n;
          sh.last[b] = last;
          sh.pass[b] = q;
          sh.self[b] = SYM && own;
          sh.norm[b] = norm;
          mbar_arrive(&sh.full[b]);
        }
        __syncwarp();
        ph ^= b;
        b ^= 1;
        n = -1;
      };

      bool ok = true;
      int s, cnt, pr, s2 = 0, cnt2 = 0, pr2 = 0;
      next_piece(s, cnt, pr);
      if (cnt > 0) issue(s, cnt, rb);
      while (cnt > 0 && ok) {
        next_piece(s2, cnt2, pr2);
        if (cnt2 > 0) issue(s2, cnt2, rb ^ 1);
        ok = mbar_wait(&sh.raw_bar[rb], rph);
        const unsigned long long* src = raw + rb * NA * RC + (s & 1);
        const unsigned long long* msk = src + (DIM + NV) * RC;
        int kx, kz = 0;
        if constexpr (SYM)
          kx = (pr < 2 ? 0 : pr - 1) + nb;
        else {
          kx = jx0 + pr % ncolx - ix + nb;
          kz = jz0 + pr / ncolx - iz + nb;
        }
        if constexpr (SYM) {
          // the own cell's points, whole warps of them, in a buffer of their own (no row-j sums)
          if (own_part && pr > 0) {
            own_part = false;
            const int rest = n & 31, ob = b;
            if (n > rest) {
              n -= rest;
              const int from = n;
              publish(false, true);
              ok = ok && acquire();
              if (ok && lane < rest) {
                const uint2* oc = (const uint2*)(smem + Lay::comp) + ob * (DIM + NV) * KC + from + lane;
                uint2* nc = (uint2*)(smem + Lay::comp) + b * (DIM + NV) * KC + lane;
#pragma unroll
                for (int d = 0; d < DIM + NV; d++) nc[d * KC] = oc[d * KC];
                unsigned* cm = (unsigned*)(smem + Lay::code);
                cm[b * 2 * KC + lane] = 0xffffffffu;
                cm[b * 2 * KC + KC + lane] = 0u;
              }
              if (ok) n = rest;
            }
          }
        }
        // groups of four 32-source chunks: one warp's instructions are all that is in flight
        constexpr int U = 4;
        for (int e0 = 0; e0 < cnt && ok; e0 += 32 * U) {
          bool in[U], fij[U];
          unsigned M[U], bal[U];
          int got = 0;
#pragma unroll
          for (int u = 0; u < U; u++) {
            const int e = e0 + 32 * u + lane;
            in[u] = fij[u] = false;
            M[u] = 0xffffffffu;
            if (e < cnt) {
              const unsigned long long m = msk[e];
              const int j = s + e, ky = (int)(m >> kMaskCellY) - iy + nb;
              // the reference's box test against this cell's centre; the cell's own points
              // unconditionally (2d/get_trunc.h:31-39, 63; 3d/get_trunc.h:70-72)
              unsigned boxin = ((unsigned)m >> kx) & ((unsigned)m >> (kMaskY + ky));
              if (DIM == 3) boxin &= (unsigned)(m >> (kMaskZ + kz));
              fij[u] = (boxin & 1u) || (j >= c0 && j < c1);
              in[u] = fij[u];
              if constexpr (SYM)
                if (pr > 0) {  // the bits a target has when it lies in T(c(j))
                  M[u] = (1u << (2 * nb - kx)) | (1u << (kMaskY + 2 * nb - ky));
                  in[u] = fij[u] || (tor & M[u]) == M[u];
                }
            }
          }
#pragma unroll
          for (int u = 0; u < U; u++) {
            bal[u] = __ballot_sync(0xffffffffu, in[u]);
            got += __popc(bal[u]);
          }
          if (got == 0) continue;
          if (n < 0) ok = acquire();
          if (!ok) break;
          // the group's sources in order; those beyond the buffer's end go to the next one
          int from = 0;  // sources of the group already put
          while (true) {
            const int base = n - from, room = min(got, KC - base);
            uint2* comp = (uint2*)(smem + Lay::comp) + b * (DIM + NV) * KC;
            int pre = 0;
#pragma unroll
            for (int u = 0; u < U; u++) {
              const int e = e0 + 32 * u + lane, at = pre + __popc(bal[u] & ((1u << lane) - 1u));
              pre += __popc(bal[u]);
              if (in[u] && at >= from && at < room) {
#pragma unroll
                for (int d = 0; d < DIM; d++) comp[d * KC + base + at] = ((const uint2*)src)[d * RC + e];
#pragma unroll
                for (int v = 0; v < NV; v++) {
                  const double gj = ((const double*)src)[(DIM + v) * RC + e];
                  ((double*)comp)[(DIM + v) * KC + base + at] = SYM && !fij[u] ? 0.0 : gj;
                }
                if constexpr (SYM) {
                  unsigned* cm = (unsigned*)(smem + Lay::code) + b * 2 * KC;
                  cm[base + at] = M[u];
                  cm[KC + base + at] = (unsigned)(s + e);
                }
              }
            }
            n = base + room;
            from = room;
            if (n == KC) publish(false);
            if (from >= got) break;
            ok = acquire();
            if (!ok) break;
          }
        }
        __syncwarp();
        rph ^= rb;
        rb ^= 1;
        s = s2;
        cnt = cnt2;
        pr = pr2;
      }
      if (ok && n < 0) ok = acquire();
      if (!ok) {
        if (lane == 0) atomicOr(err, DEV_ERR_TIMEOUT);
        // let the copies in flight land (bounded) before the CTA exits
        if (cnt > 0) mbar_wait(&sh.raw_bar[rb], rph, 1u << 20);
        return;
      }
      publish(true, own_part);
    }
  }
}

template <int DIM, int NV, bool BATCH, bool SYM, bool WIDE>
void launch_fx_k(const GaussPlan& P, const PointsView& t, const PointsView& s, const double* gv, double* w,
               long long vstride, unsigned* err, const int* skip, VecSkip left, cudaStream_t st) {
  constexpr size_t sm = LayoutX<DIM, NV, SYM>::total;
  static_assert(sm <= 112 * 1024, "two CTAs of k_gauss_fx per SM");
  static std::atomic<bool> attr_set[64];  // per device: attribute set (idempotent, thread-safe)
  int dev = 0;
  PRBF_CUDA(cudaGetDevice(&dev));
  if (dev >= 64 || !attr_set[dev]) {
    PRBF_CUDA(cudaFuncSetAttribute(k_gauss_fx<DIM, NV, BATCH, SYM, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sm));
    if (dev < 64) attr_set[dev] = true;
  }
  const DevBuf<uint2>* T = P.fx_self ? P.fxs : P.fxt;
  FxArgs a{T[0].get(), T[1].get(), T[2].get(), P.fxs[0].get(), P.fxs[1].get(), P.fxs[2].get(), P.smask.get(), gv,
           vstride,    w,          nullptr,    0,              0,              s.n,            P.fx_ncs, P.max_tile, left};
  const int2* items = P.items.get();
  int nitems = P.nitems, grid = P.grid;
  if constexpr (SYM) {
    a.part = P.sym_part.get();
    a.pstride = P.sym_pstride;
    a.K = P.sym_K;
    if (P.sym_nitems > 0) {  // a batch's list of one item per cell
      items = P.sym_items.get();
      nitems = P.sym_nitems;
      a.tile = kTileT;
      grid = 0;
    }
  }
  // many items: the resident CTAs in rounds, so that the tables are read once per CTA
  if (grid <= 0 && nitems >= 16 * kResident) grid = kResident;
  grid = grid > 0 ? std::min(grid, nitems) : nitems;
  // few items: a cell's passes on CTAs of their own
  const dim3 gd(grid, nitems < kResident ? ceil_div(kTileT, CfgX<DIM, NV, SYM>::TT) : 1);
  k_gauss_fx<DIM, NV, BATCH, SYM, WIDE><<<gd, kFxThreads<SYM>, sm, st>>>(P.g, P.grids.get(), P.cprob.get(), P.seg, items,
                                                               nitems, t.cell_start, s.cell_start, a, err, skip);
  PRBF_CHECK_LAUNCH();
}

template <int DIM, int NV, bool BATCH, bool SYM>
void launch_fx(const GaussPlan& P, const PointsView& t, const PointsView& s, const double* gv, double* w,
               long long vstride, unsigned* err, const int* skip, VecSkip left, cudaStream_t st) {
  if constexpr (DIM == 3)
    if (P.fx_wide) return launch_fx_k<DIM, NV, BATCH, SYM, true>(P, t, s, gv, w, vstride, err, skip, left, st);
  launch_fx_k<DIM, NV, BATCH, SYM, false>(P, t, s, gv, w, vstride, err, skip, left, st);
}

template <int DIM>
void sum_dim(const GaussPlan& P, const PointsView& t, const PointsView& s, const double* gv, double* w, int nv,
             long long vs, unsigned* err, const int* skip, VecSkip left, cudaStream_t st) {
  if (P.batched) {  // the problems are the segments of one vector
    for (int v = 0; v < nv; v++)
      launch_fx<DIM, 1, true, false>(P, t, s, gv + v * vs, w + v * vs, vs, err, skip, VecSkip{}, st);
    return;
  }
  for (int v0 = 0; v0 < nv; v0 += 4) {
    const double* g0 = gv + v0 * vs;
    double* w0 = w + v0 * vs;
    const int k0 = std::min(4, nv - v0);
    const VecSkip l0 = vec_part(left, v0, k0);
    for_counts(l0, k0, [&](int k) {
      switch (k) {
        case 1: launch_fx<DIM, 1, false, false>(P, t, s, g0, w0, vs, err, skip, l0, st); break;
        case 2: launch_fx<DIM, 2, false, false>(P, t, s, g0, w0, vs, err, skip, l0, st); break;
        case 3: launch_fx<DIM, 3, false, false>(P, t, s, g0, w0, vs, err, skip, l0, st); break;
        default: launch_fx<DIM, 4, false, false>(P, t, s, g0, w0, vs, err, skip, l0, st); break;
      }
    });
  }
}

}  // namespace

void gauss_fx_sum(const GaussPlan& P, const PointsView& t, const PointsView& s, const double* gv, double* w,
                  unsigned* err, const int* skip, int nv, long long vstride, VecSkip left, cudaStream_t st) {
  if (P.g.dim == 2)
    sum_dim<2>(P, t, s, gv, w, nv, vstride, err, skip, left, st);
  else
    sum_dim<3>(P, t, s, gv, w, nv, vstride, err, skip, left, st);
}

void gauss_fx_sym(const GaussPlan& P, const PointsView& s, const double* gv, double* w, unsigned* err,
                  const int* skip, cudaStream_t st) {
  if (P.batched)
    launch_fx<2, 1, true, true>(P, s, s, gv, w, 0, err, skip, VecSkip{}, st);
  else
    launch_fx<2, 1, false, true>(P, s, s, gv, w, 0, err, skip, VecSkip{}, st);
}

// The tables of gauss_fx.cuh, uploaded once per device.
void gauss_fx_upload_tables(cudaStream_t s) {
  static std::atomic<bool> ready[64];
  int dev = 0;
  PRBF_CUDA(cudaGetDevice(&dev));
  if (dev < 64 && ready[dev]) return;
  std::vector<uint2> h1(kFxTab), h2(kFxTab);
  fx_tables(h1.data(), h2.data());
  const size_t bytes = sizeof(uint2) * kFxTab;
  PRBF_CUDA(cudaMemcpyToSymbolAsync(d_fx_t1, h1.data(), bytes, 0, cudaMemcpyHostToDevice, s));
  PRBF_CUDA(cudaMemcpyToSymbolAsync(d_fx_t2, h2.data(), bytes, 0, cudaMemcpyHostToDevice, s));
  PRBF_CUDA(cudaStreamSynchronize(s));
  if (dev < 64) ready[dev] = true;
}

}  // namespace prbf
