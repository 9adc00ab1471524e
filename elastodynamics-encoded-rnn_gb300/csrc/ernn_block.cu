// Time-blocked tile kernels (sm_103a): up to four time steps of a tile per
// launch, the tile's state in shared memory.
//
// One step of the scheme on a large grid moves 24 bytes of state per cell
// (adjoint 32) through HBM for some 60 FP32 operations: a launch per step is
// bound by the memory, and on grids of a few hundred cells a side by the
// launches.  Here a CTA loads a tile of both levels with a halo of four
// cells once (TMA, zeros outside the grid), advances it up to four steps,
// and writes the last two levels: 24 -> 8 bytes per cell and step.
//
// Layout: a warp owns RW rows of 128 columns, each lane one quad of four
// columns; a new level overwrites the older one in place.  A row is read once
// per step and kept in registers while it is the upper, middle and lower row
// of the window; the columns beside a quad come by lane shuffles, rows of
// other warps from shared memory (one CTA barrier per step).  The valid region
// shrinks by one cell per step, so the outer quad and the outer four rows of
// the tile are not stored: 120 columns x (W RW - 8) rows are (on grids of at
// most 128 or 64 columns a tile holds whole rows and has no halo columns).  Two
// CTAs per SM (tall tiles): one loads its tile while the other computes.
//
// Measured (16 x 1024^2, us per launch of four steps against four launches of
// the one-step kernels before): forward 173 against 264, adjoint 290 against
// 456.  What bounds it is the FP32 pipe's issue: 40 warp instructions per
// four cells and step, 30 of them the scheme's, at 55-60 % of the issue rate;
// HBM runs at half its measured rate.
//
// Every cell's update is the same sequence of rounded operations as in the
// per-step kernels, so the states agree with theirs bit for bit.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <cmath>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "ernn_block.h"
#include "ernn_launch.h"
#include "ernn_tile.cuh"

namespace ernn {

namespace {

constexpr int kBox = 128;  // columns of a tile with its halo: 32 lanes x 4
constexpr int kH = kBlkSteps;
constexpr unsigned kFull = 0xffffffffu;

// A tile: state plane, instance, first row and column, and the region
// [xs, xe) x [ys, ye) of its instance (the whole grid without instances).
struct BTile {
  int plane, inst, x0, y0, xs, ys, xe, ye;
};

// The tiles first, first + step, ... of a CTA.  Grid: walked in (shot, row
// block, column block) digits, an addition with carries per tile; instances:
// entries of the tile table.
template <bool INST, int H, int C = kBlkCols>
struct BWalk {
  int t, step, shot, xt, yt, ds, dx, dy, tiles_x, tiles_y, nx, ny;
  __device__ __forceinline__ void init(int first, int step_, int tx, int ty, int nx_, int ny_) {
    t = first;
    step = step_;
    if constexpr (!INST) {
      tiles_x = tx;
      tiles_y = ty;
      nx = nx_;
      ny = ny_;
      const int per = tx * ty;
      shot = first / per;
      int r = first - shot * per;
      xt = r / ty;
      yt = r - xt * ty;
      ds = step / per;
      r = step - ds * per;
      dx = r / ty;
      dy = r - dx * ty;
    }
  }
  __device__ __forceinline__ BTile tile(const InstTiles& in) const {
    if constexpr (INST) {
      const int4 e = __ldg(&in.tiles[t]);
      return BTile{0, e.x, (int)((unsigned)e.y & 0xffffu), (int)((unsigned)e.y >> 16), (int)((unsigned)e.z & 0xffffu),
                   (int)((unsigned)e.z >> 16), (int)((unsigned)e.w & 0xffffu), (int)((unsigned)e.w >> 16)};
    } else {
      return BTile{shot, shot, xt * H, yt * C, 0, 0, nx, ny};
    }
  }
  __device__ __forceinline__ void next() {
    t += step;
    if constexpr (!INST) {
      yt += dy;
      if (yt >= tiles_y) { yt -= tiles_y; ++xt; }
      xt += dx;
      if (xt >= tiles_x) { xt -= tiles_x; ++shot; }
      shot += ds;
    }
  }
};

// Four cells of a row.
struct Q4 {
  float v[4];
};
__device__ __forceinline__ Q4 q4(const float4 v) { return Q4{{v.x, v.y, v.z, v.w}}; }
__device__ __forceinline__ float4 f4(const Q4& q) { return make_float4(q.v[0], q.v[1], q.v[2], q.v[3]); }

// One row of a component: the quad (w[1] .. w[4]) and the cells beside it.
struct Row {
  float w[6];
};
__device__ __forceinline__ Row row_of(const Q4& q) {
  return Row{{__shfl_up_sync(kFull, q.v[3], 1), q.v[0], q.v[1], q.v[2], q.v[3], __shfl_down_sync(kFull, q.v[0], 1)}};
}

// The constants in the order of Coef; zero for a lane whose quad lies outside
// the region (its levels are zero, and stay so).
__device__ __forceinline__ Coefs coefs_in(const float* k, bool in) {
  return Coefs{in ? k[0] : 0.f, in ? k[1] : 0.f, in ? k[2] : 0.f, in ? k[3] : 0.f,
               in ? k[4] : 0.f, in ? k[5] : 0.f, in ? k[6] : 0.f, in ? k[7] : 0.f};
}

// Second differences at cell q of the quad of row m, with the rows t above
// and b below:
//   xx = (t + b) - 2 m,  yy = (left + right) - 2 m,
//   xy = (b[+1] + t[-1]) - (b[-1] + t[+1]),
// each with the association and rounding of the per-step kernels.  Scalar
// operations: a packed one (two cells) takes the FP32 pipe twice as long, and
// a scalar one between packed ones as long as they (measured: 3.9 scalar,
// 1.8 packed, 1.9 mixed warp instructions per cycle and SM).
struct Sums {
  float xx, yy, xy;
};
__device__ __forceinline__ Sums sums_of(const Row& t, const Row& m, const Row& b, int q) {
  const int k = q + 1;
  return Sums{fmaf(-2.f, m.w[k], t.w[k] + b.w[k]), fmaf(-2.f, m.w[k], m.w[k - 1] + m.w[k + 1]),
              (b.w[k + 1] + t.w[k - 1]) - (b.w[k - 1] + t.w[k + 1])};
}

// The operator at a cell from the sums of both components.  The first two
// terms of each row are one rounded product and one fused multiply-add; which
// product is rounded is an argument (kOrder*), so that a problem's states
// agree bit for bit with those of the per-step kernels of its size and mode:
// the first in the tiled ones, the second in the plain ones (with constant
// planes: the second of the x row, the first of the y row).  The same for the
// adjoint: its constants' sums cancel to a small part of their terms, and a
// lam of another rounding moved single constants' gradients by up to 3e-5 of
// their value (the plain kernels' own distance from 64 bits is as large).
constexpr int kOrderTiled = 0, kOrderPlain = 3, kOrderFields = 1;
template <int ORDER>
__device__ __forceinline__ void oper(const Coefs& k, const Sums& x, const Sums& y, float& lx, float& ly) {
  lx = (ORDER & 1) ? fmaf(k.k11, x.xx, __fmul_rn(k.k66, x.yy)) : fmaf(k.k66, x.yy, __fmul_rn(k.k11, x.xx));
  lx = fmaf(k.kq12, y.xy, lx);
  lx = fmaf(k.k16h, x.xy, lx);
  lx = fmaf(k.k16, y.xx, lx);
  lx = fmaf(k.k26, y.yy, lx);
  ly = (ORDER & 2) ? fmaf(k.k66, y.xx, __fmul_rn(k.k22, y.yy)) : fmaf(k.k22, y.yy, __fmul_rn(k.k66, y.xx));
  ly = fmaf(k.kq12, x.xy, ly);
  ly = fmaf(k.k16, x.xx, ly);
  ly = fmaf(k.k26, x.yy, ly);
  ly = fmaf(k.k26h, y.xy, ly);
}
// The scaled constants of a cell (C11, C22, C12, C16, C26, C66 planes of n
// cells), zero when it is not `in`.
__device__ __forceinline__ Coefs cell_coefs(const float* f, size_t n, size_t o, bool in, float q) {
  float c[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) c[k] = in ? __ldg(f + k * n + o) : 0.f;
  Coefs r;
  r.k11 = c[0] * q;
  r.k22 = c[1] * q;
  r.k66 = c[5] * q;
  r.k16 = c[3] * q;
  r.k26 = c[4] * q;
  r.k16h = 0.5f * r.k16;
  r.k26h = 0.5f * r.k26;
  r.kq12 = (c[2] + c[5]) * q * 0.25f;
  return r;
}
// (2 c - p) + l
__device__ __forceinline__ float leap(float c, float p, float l) { return fmaf(2.f, c, -p) + l; }

// A CTA's tile: both levels of its rows, both components, with a guard row on
// either side (read for rows that are never stored).  A row takes L lanes, a
// quad each, so a warp holds 32 / L shares of RW rows.  WHOLE: the tile's
// columns are all the grid's (or instance's): no halo columns, zeros beside
// the first and the last.
template <int W_, int RW_, int L = 32, bool WHOLE = false>
struct BlkTile {
  static constexpr int kW = W_, kRW = RW_, kLanes = L, kShares = 32 / L;
  static constexpr bool kWhole = WHOLE;
  static constexpr int kThreads = 32 * W_;
  static constexpr int kRows = W_ * RW_ * kShares;
  static constexpr int kCols = 4 * L;
  static constexpr int kHY = WHOLE ? 0 : kH;         // halo columns
  static constexpr int kUse = kRows - 2 * kH;        // rows stored
  static constexpr int kUseY = kCols - 2 * kHY;      // columns stored
  static constexpr int kPlane = kRows * kCols;       // floats of a component
  static constexpr int kLevel = 2 * kPlane;
  static constexpr int kFloats = 2 * kLevel + 2 * kBox;
  static constexpr int kMeta = 16;
  static constexpr size_t kBytes = (size_t)(kFloats + kMeta) * 4 + 8 + 128;
  static_assert(L == 32 || WHOLE, "shares of a warp: whole rows");
};

// Whether a condition holds for any / every share of the warp.
template <class B>
__device__ __forceinline__ bool any_share(bool c) {
  return B::kShares == 1 ? c : __any_sync(kFull, c) != 0;
}
template <class B>
__device__ __forceinline__ bool every_share(bool c) {
  return B::kShares == 1 ? c : __all_sync(kFull, c) != 0;
}

template <bool V>
struct BoolC {
  static constexpr bool value = V;
};

// Zeroes the cells n .. 3 of a quad.
__device__ __forceinline__ void mask_q(float (&v)[4], int n) {
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = n > q ? v[q] : 0.f;
}

__device__ __forceinline__ Row load_row(const float* p) {  // a row of the tile at the lane's quad
  return row_of(q4(*reinterpret_cast<const float4*>(p)));
}
// A row of a tile of whole rows, whose ends have zeros beside them; ql: the
// lane's quad in its row.
template <class B>
__device__ __forceinline__ Row whole_row(const float* p, int ql) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  const float l = __shfl_up_sync(kFull, v.w, 1, B::kLanes), r = __shfl_down_sync(kFull, v.x, 1, B::kLanes);
  return Row{{ql > 0 ? l : 0.f, v.x, v.y, v.z, v.w, ql < B::kLanes - 1 ? r : 0.f}};
}

// Rows of a warp's share that lie in [lo, hi) of the tile, as bits.
template <int RW>
__device__ __forceinline__ uint32_t rows_in(int rr0, int lo, int hi) {
  lo = max(lo - rr0, 0);
  hi = min(hi - rr0, RW);
  return hi > lo ? ((1u << hi) - 1u) & ~((1u << lo) - 1u) : 0u;
}

// Zeroes the tile's cells outside its instance's region (on a canvas they
// belong to other instances), or all of a level that is a zero state.
template <class B>
__device__ __forceinline__ void clear_cells(float* lev, bool all, const BTile& t) {
  for (int e = threadIdx.x; e < B::kPlane / 4; e += B::kThreads) {
    const int gi = t.x0 - kH + e / B::kLanes, gj = t.y0 - B::kHY + 4 * (e % B::kLanes);
    if (!all && gi >= t.xs && gi < t.xe && gj >= t.ys && gj < t.ye) continue;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(lev + 4 * e) = z;
    *reinterpret_cast<float4*>(lev + B::kPlane + 4 * e) = z;
  }
}

// Both levels of a tile into shared memory: c (u^i, or lam^{m+1}) and p (the
// level before it); a level that is not used is zero.  Every thread calls it;
// the tile is complete after the caller's next CTA barrier.
template <class B, bool INST>
__device__ __forceinline__ void load_tile(float* lev0, float* lev1, const CUtensorMap* cm, const CUtensorMap* pm,
                                          bool has_c, bool has_p, bool use_c, bool use_p, const BTile& t, int k,
                                          uint64_t* bar, PipeGuard* guard, int* err) {
  const uint32_t bytes = (uint32_t)((has_c ? B::kLevel : 0) + (has_p ? B::kLevel : 0)) * 4u;
  if (bytes != 0) {
    if (threadIdx.x == 0 && !pipe_failed(guard)) {
      pipe_issued(guard, k);
      fence_async();
      bar_expect(bar, bytes);
      if (has_c) tma_load3(lev0, cm, t.y0 - B::kHY, t.x0 - kH, 2 * t.plane, bar);
      if (has_p) tma_load3(lev1, pm, t.y0 - B::kHY, t.x0 - kH, 2 * t.plane, bar);
    }
    bar_wait_ok(bar, (uint32_t)k & 1u, err, guard);
  }
  if (INST || !use_c) clear_cells<B>(lev0, !use_c, t);
  if (INST || !use_p) clear_cells<B>(lev1, !use_p, t);
}

// ----------------------------------------------------------------- forward
// Per-cell modes: FIELDS keeps the constants of the thread's cells in registers
// for the launch (one row per thread); DFIELD reads the weights 1 - D of a row
// one row ahead.
template <int MODE, class B, bool INST, int ORDER, int CTAS>
__global__ void __launch_bounds__(B::kThreads, CTAS)
    blk_fwd_kernel(const BlkFwd a, const __grid_constant__ CUtensorMap cur_map,
                   const __grid_constant__ CUtensorMap prev_map, int tiles_x, int tiles_y, int ntiles, int* err) {
  extern __shared__ float sm_raw[];
  float* sm = aligned128(sm_raw);
  constexpr int NT = B::kThreads, RW = B::kRW, kCols = B::kCols;
  float* lev0 = sm + kBox;  // (a guard row before and after the levels)
  float* lev1 = lev0 + B::kLevel;
  float* meta = sm + B::kFloats;
  uint64_t* bar = reinterpret_cast<uint64_t*>(meta + B::kMeta);
  __shared__ PipeGuard guard;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int nx = a.nx, ny = a.ny;
  const size_t N = (size_t)nx * ny, Np = (size_t)nx * a.pitch;
  const bool has_src = a.bx > 0 && a.by > 0;
  grid_dep_trigger();
  if (tid == 0) {
    prefetch_map(&cur_map);
    prefetch_map(&prev_map);
    bar_init(bar);
    pipe_init(&guard);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // (zeros: what rows without a neighbour read stays finite)
  if (tid < kBox) sm[tid] = sm[B::kFloats - kBox + tid] = 0.f;
  BWalk<INST, B::kUse, B::kUseY> walk;
  walk.init((int)blockIdx.x, (int)gridDim.x, tiles_x, tiles_y, nx, ny);
  __syncthreads();
  grid_dep_wait();  // the states of the previous launch are complete from here on

  const int ql = lane % B::kLanes;                           // the lane's quad of its rows
  const int rr0 = (w * B::kShares + lane / B::kLanes) * RW;  // the first of them in the tile
  const int o0 = rr0 * kCols + 4 * ql;
  for (int k = 0; walk.t < ntiles; ++k, walk.next()) {
    const BTile tile = walk.tile(a.inst);
    // per-tile scalars: coefficients, amplitudes of the steps, source origin
    if (w == 0) {
      const Coef* K = a.coef + (size_t)tile.inst * a.coef_stride;
      if (lane < 8) meta[lane] = (&K->k11)[lane];
      if (lane >= 8 && lane < 8 + kBlkSteps && a.i + lane - 8 < a.nt)
        meta[lane] = a.src_signal[(size_t)tile.inst * a.nt + a.i + lane - 8] * K->kappa;
      if (lane >= 12 && lane < 14 && has_src) meta[lane] = __int_as_float(a.src_origin[2 * tile.inst + lane - 12]);
    }
    load_tile<B, INST>(lev0, lev1, &cur_map, &prev_map, a.cur != nullptr, a.prev != nullptr, a.cur != nullptr,
                       a.prev != nullptr, tile, k, bar, &guard, err);
    __syncthreads();
    const int gj = tile.y0 - B::kHY + 4 * ql, gi0 = tile.x0 - kH + rr0;
    // cells of the quad inside the region's columns; rows of the warp inside
    // its rows, and those this lane stores
    const int nq = gj >= tile.ys ? max(0, min(4, tile.ye - gj)) : 0;
    const uint32_t region = rows_in<RW>(rr0, tile.xs - tile.x0 + kH, tile.xe - tile.x0 + kH);
    const uint32_t stored = (B::kWhole || (ql >= 1 && ql <= B::kLanes - 2)) && nq > 0
                                ? region & rows_in<RW>(rr0, kH, B::kRows - kH)
                                : 0u;
    const Coefs ks = coefs_in(meta, nq > 0);
    Coefs kc[MODE == kModeFields ? 4 : 1];
    if constexpr (MODE == kModeFields) {
      static_assert(RW == 1, "one row of constants in registers");
      const float q = a.coef->q;
      const size_t o = (size_t)gi0 * ny + gj;
#pragma unroll
      for (int c = 0; c < 4; ++c) kc[c] = cell_coefs(a.field, N, o + c, region != 0 && c < nq, q);
    }
    auto weights = [&](int r, float(&wv)[4]) {  // 1 - D at the warp's row r (zero outside the grid)
      const float* d = a.field + (ptrdiff_t)(gi0 + r) * ny + gj;
      const bool in = (region >> r) & 1u;
      if (a.vec_field) {
        const float4 v = in && nq > 0 ? __ldg(reinterpret_cast<const float4*>(d)) : make_float4(1.f, 1.f, 1.f, 1.f);
        wv[0] = 1.f - v.x; wv[1] = 1.f - v.y; wv[2] = 1.f - v.z; wv[3] = 1.f - v.w;
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) wv[c] = in && c < nq ? 1.f - __ldg(d + c) : 0.f;
      }
    };
    const int ox = __float_as_int(meta[12]), oy = __float_as_int(meta[13]);
    const bool src = has_src && tile.x0 - kH < ox + a.bx && tile.x0 - kH + B::kRows > ox &&
                     tile.y0 - B::kHY < oy + a.by && tile.y0 - B::kHY + kCols > oy;
    const bool ragged = ((tile.ye - tile.ys) & 3) != 0 && tile.y0 - B::kHY + kCols > tile.ye;
    const int2 recs = a.rec_tile != nullptr ? a.rec_tile[walk.t] : make_int2(0, 0);
    int T = a.T;
    if (INST) T = min(T, a.inst.box[2 * tile.inst + 1].z - a.i);
    const ptrdiff_t off = (ptrdiff_t)tile.plane * 2 * (ptrdiff_t)Np + (ptrdiff_t)gi0 * a.pitch + gj;
    if (a.out[0] != nullptr) {
#pragma unroll
      for (int r = 0; r < RW; ++r)
        if ((stored >> r) & 1u) {
          float* o = a.out[0] + off + (ptrdiff_t)r * a.pitch;
          *reinterpret_cast<float4*>(o) = *reinterpret_cast<const float4*>(lev0 + o0 + r * kCols);
          *reinterpret_cast<float4*>(o + Np) = *reinterpret_cast<const float4*>(lev0 + B::kPlane + o0 + r * kCols);
        }
    }
    for (int t = 1; t <= T; ++t) {
      const float* c0 = ((t & 1) ? lev0 : lev1) + o0;  // u^{i+t-1}
      float* p0 = ((t & 1) ? lev1 : lev0) + o0;        // u^{i+t-2}, becomes u^{i+t}
      const int frame = a.frame[t];
      const bool dense = frame >= 0 && a.record == kRecordFields;
      float* out0 = a.out[t] + off;
      float* out1 = out0 + Np;
      const uint32_t st = a.out[t] != nullptr ? stored : 0u;
      auto rows = [&](auto plain) {
        constexpr bool PLAIN = decltype(plain)::value;
        auto row_at = [&](const float* p) {  // a row of the tile at the lane's quad
          if constexpr (B::kWhole) return whole_row<B>(p, ql);
          else return row_of(q4(*reinterpret_cast<const float4*>(p)));
        };
        [[maybe_unused]] float wn[4], wv[4];
        if constexpr (MODE == kModeDField) weights(0, wn);
        Row t0 = row_at(c0 - kCols), t1 = row_at(c0 + B::kPlane - kCols);
        Row m0 = row_at(c0), m1 = row_at(c0 + B::kPlane);
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          if constexpr (MODE == kModeDField) {
#pragma unroll
            for (int q = 0; q < 4; ++q) wv[q] = wn[q];
            if (r + 1 < RW) weights(r + 1, wn);
          }
          const Row b0 = row_at(c0 + (r + 1) * kCols), b1 = row_at(c0 + B::kPlane + (r + 1) * kCols);
          if (PLAIN || ((region >> r) & 1u)) {  // (rows outside the region stay zero)
            const float4 pv0 = *reinterpret_cast<const float4*>(p0 + r * kCols);
            const float4 pv1 = *reinterpret_cast<const float4*>(p0 + B::kPlane + r * kCols);
            const float q0[4] = {pv0.x, pv0.y, pv0.z, pv0.w}, q1[4] = {pv1.x, pv1.y, pv1.z, pv1.w};
            float v0[4], v1[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              oper<ORDER>(MODE == kModeFields ? kc[MODE == kModeFields ? q : 0] : ks, sums_of(t0, m0, b0, q),
                         sums_of(t1, m1, b1, q), v0[q], v1[q]);
              if constexpr (MODE == kModeDField) {
                v0[q] = __fmul_rn(v0[q], wv[q]);
                v1[q] = __fmul_rn(v1[q], wv[q]);
              }
            }
            if (!PLAIN && src && (unsigned)(gi0 + r - ox) < (unsigned)a.bx) {
              // the load joins the operator sum before the update, as in the
              // reference's (A u + f) / rho
              const float amp = meta[7 + t];
              const float* f = a.src_map + ((size_t)tile.inst * a.bx + (gi0 + r - ox)) * a.by;
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const int sb = gj + q - oy;
                if ((unsigned)sb < (unsigned)a.by && q < nq) {
                  float& l = a.src_comp == 0 ? v0[q] : v1[q];
                  l = fmaf(amp, f[sb], l);  // L + amp f, one rounding
                }
              }
            }
            // (quads outside the region stay zero: their lanes' coefficients are)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              v0[q] = leap(m0.w[q + 1], q0[q], v0[q]);
              v1[q] = leap(m1.w[q + 1], q1[q], v1[q]);
            }
            if (!PLAIN && ragged) {  // the region's last column is inside a quad
              mask_q(v0, nq);
              mask_q(v1, nq);
            }
            const float4 n0 = make_float4(v0[0], v0[1], v0[2], v0[3]), n1 = make_float4(v1[0], v1[1], v1[2], v1[3]);
            *reinterpret_cast<float4*>(p0 + r * kCols) = n0;
            *reinterpret_cast<float4*>(p0 + B::kPlane + r * kCols) = n1;
            if ((st >> r) & 1u) {
              *reinterpret_cast<float4*>(out0) = n0;
              *reinterpret_cast<float4*>(out1) = n1;
            }
            if (!PLAIN && dense && ((stored >> r) & 1u)) {
              const size_t o = ((size_t)tile.plane * a.nt_out + frame) * N + (size_t)(gi0 + r) * ny + gj;
              if (a.vec) {
                *reinterpret_cast<float4*>(a.rec_x + o) = n0;
                *reinterpret_cast<float4*>(a.rec_y + o) = n1;
              } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                  if (q < nq) {
                    a.rec_x[o + q] = v0[q];
                    a.rec_y[o + q] = v1[q];
                  }
              }
            }
          }
          out0 += a.pitch;
          out1 += a.pitch;
          t0 = m0; t1 = m1; m0 = b0; m1 = b1;
        }
      };
      // (warps none of whose rows a later step reads have nothing to do)
      if (any_share<B>(region != 0 && rows_in<RW>(rr0, t, B::kRows - t) != 0)) {
        if (every_share<B>(region == (1u << RW) - 1u) && !src && !ragged && !dense) rows(BoolC<true>{});
        else rows(BoolC<false>{});
      }
      __syncthreads();  // u^{i+t} is complete; its receivers are read beside the next step
      if (frame >= 0 && recs.y > 0) {
        const float* lv = (t & 1) ? lev1 : lev0;
        const size_t o = ((size_t)tile.inst * a.nt_out + frame) * a.nrec;
        for (int e = tid; e < recs.y; e += NT) {
          const int2 v = a.rec_ent[recs.x + e];
          const int rr = v.x / kCols, cc = v.x % kCols;
          if (rr < kH || rr >= B::kRows - kH || cc < B::kHY || cc >= kCols - B::kHY) continue;  // another tile's
          a.rec_x[o + v.y] = lv[v.x];
          a.rec_y[o + v.y] = lv[B::kPlane + v.x];
        }
      }
    }
    __syncthreads();  // the levels and scalars are read: the next tile's may arrive
  }
  if (tid == 0 && pipe_failed(&guard)) pipe_drain(bar, 1, &guard);
}

// Adds the threads' imaging sums (FP32 pairs) to a row of partials and clears
// them; every thread of the CTA calls it.
// The lanes' pairs are added as pairs (a warp's FP64 addition occupies this
// part's FP64 pipe for 16 cycles and more, and thirty of them took longer
// than a step of a small tile), and each exchange halves the values a lane
// still carries: 4 + 2 + 1 additions leave one value in every group of four
// lanes, two more sum it over the group.
// (The per-step kernels add warps and steps in FP64.  The same sums over steps
// and lanes in FP64 here gave the same gradients, in float32, on the five timed
// scalar cases and eight drawn ones, and passes of 1.04 to 1.27 times the time.
// The pair of 96 random terms was their exact sum in each of 400 trials.)
template <int W>
__device__ __forceinline__ void flush_sums(float (&hi)[6], float (&lo)[6], float2 (*red)[6], double* row) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  float h[8], l[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    h[q] = q < 6 ? hi[q < 6 ? q : 0] : 0.f;
    l[q] = q < 6 ? lo[q < 6 ? q : 0] : 0.f;
  }
  auto add = [&](int q, float h2, float l2) {
    const float s = h[q] + h2, bp = s - h[q];
    l[q] = (l[q] + l2) + ((h[q] - (s - bp)) + (h2 - bp));
    h[q] = s;
  };
#pragma unroll
  for (int n = 4; n >= 1; n >>= 1) {  // lanes with bit 4 n set keep values n .. 2 n - 1
    const bool up = (lane & (4 * n)) != 0;
#pragma unroll
    for (int q = 0; q < n; ++q) {
      const float sh = up ? h[q] : h[q + n], sl = up ? l[q] : l[q + n];
      h[q] = up ? h[q + n] : h[q];
      l[q] = up ? l[q + n] : l[q];
      add(q, __shfl_xor_sync(kFull, sh, 4 * n), __shfl_xor_sync(kFull, sl, 4 * n));
    }
  }
  add(0, __shfl_xor_sync(kFull, h[0], 2), __shfl_xor_sync(kFull, l[0], 2));
  add(0, __shfl_xor_sync(kFull, h[0], 1), __shfl_xor_sync(kFull, l[0], 1));
  // (bits 4, 3, 2 of the lane: bits 2, 1, 0 of the value)
  if ((lane & 3) == 0 && lane < 24) red[w][lane >> 2] = make_float2(h[0], l[0]);
#pragma unroll
  for (int q = 0; q < 6; ++q) hi[q] = lo[q] = 0.f;
  __syncthreads();
  if (tid < 6) {
    double v = 0.0;
    for (int x = 0; x < W; ++x) v += (double)red[x][tid].x + (double)red[x][tid].y;
    row[tid] += v;
  }
  __syncthreads();  // red is free again
}

// TwoSum(hi, acc)
__device__ __forceinline__ void fold_sums(float (&hi)[6], float (&lo)[6], const float (&acc)[6]) {
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    const float s = hi[q] + acc[q];
    const float bp = s - hi[q];
    lo[q] += (hi[q] - (s - bp)) + (acc[q] - bp);
    hi[q] = s;
  }
}

// The six sums' terms of a cell.
__device__ __forceinline__ void image(float (&acc)[6], float ux, float uy, const Sums& sx, const Sums& sy) {
  acc[0] = fmaf(ux, sx.xx, acc[0]);
  acc[1] = fmaf(uy, sy.yy, acc[1]);
  acc[2] = fmaf(ux, sy.xy, fmaf(uy, sx.xy, acc[2]));
  acc[3] = fmaf(uy, sx.xx, fmaf(ux, fmaf(0.5f, sx.xy, sy.xx), acc[3]));
  acc[4] = fmaf(ux, sy.yy, fmaf(uy, fmaf(0.5f, sy.xy, sx.yy), acc[4]));
  acc[5] = fmaf(uy, sy.xx, fmaf(ux, sx.yy, acc[5]));
}

// ----------------------------------------------------------------- adjoint
// As the forward, with lam^{m+1}, lam^{m+2} in the levels' place and no
// load: the recorded residuals enter at the receivers' cells (subtracted
// from lam^{m+2} before the update, as the tiled per-step kernels do; added
// to lam^m after it in the plain kernels' order) or at every cell (dense
// history).  The
// six imaging sums sum_cells lam . (dA/dC_k u) are formed in the transposed
// form sum_cells u . (dA/dC_k lam) (the second differences with zero ghosts
// are symmetric), which needs u^m only at the cell itself, read from global
// memory one row ahead.
template <class B, bool INST, int ORDER, int CTAS>
__global__ void __launch_bounds__(B::kThreads, CTAS)
    blk_adj_kernel(const BlkAdj a, const __grid_constant__ CUtensorMap cur_map,
                   const __grid_constant__ CUtensorMap prev_map, int tiles_x, int tiles_y, int ntiles, int* err) {
  extern __shared__ float sm_raw[];
  float* sm = aligned128(sm_raw);
  constexpr int NT = B::kThreads, RW = B::kRW, kCols = B::kCols;
  float* lev0 = sm + kBox;
  float* lev1 = lev0 + B::kLevel;
  float* meta = sm + B::kFloats;
  uint64_t* bar = reinterpret_cast<uint64_t*>(meta + B::kMeta);
  __shared__ PipeGuard guard;
  __shared__ float2 red[B::kW][6];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int nx = a.nx, ny = a.ny;
  const size_t N = (size_t)nx * ny, Np = (size_t)nx * a.pitch;
  grid_dep_trigger();
  if (tid == 0) {
    prefetch_map(&cur_map);
    prefetch_map(&prev_map);
    bar_init(bar);
    pipe_init(&guard);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // This CTA's tiles: strided over the grid, or with per-shot constants a
  // contiguous chunk (its sums are flushed whenever it enters another shot)
  const bool per_shot = a.coef_stride != 0;
  const int b = (int)blockIdx.x, nb = (int)gridDim.x;
  const int t_end = per_shot ? (int)((long long)(b + 1) * ntiles / nb) : ntiles;
  // (zeros: what rows without a neighbour read stays finite)
  if (tid < kBox) sm[tid] = sm[B::kFloats - kBox + tid] = 0.f;
  BWalk<INST, B::kUse, B::kUseY> walk;
  walk.init(per_shot ? (int)((long long)b * ntiles / nb) : b, per_shot ? 1 : nb, tiles_x, tiles_y, nx, ny);
  __syncthreads();
  grid_dep_wait();  // the states of the previous launch are complete from here on
  const float gs = a.coef->gscale;  // one scale for every shot

  // Imaging sums: FP32 over a thread's cells of one step, over steps and
  // tiles as FP32 pairs (TwoSum; the sum does not depend on how the steps
  // are split over launches), FP64 across warps and launches.
  float hi[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, lo[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  auto flush = [&](int shot) {  // CTA-uniform
    flush_sums<B::kW>(hi, lo, red, a.partials + (per_shot ? (size_t)shot * kTiledRowsPerShot + b : (size_t)b) * 8);
  };
  int acc_shot = -1;

  const int ql = lane % B::kLanes;                           // the lane's quad of its rows
  const int rr0 = (w * B::kShares + lane / B::kLanes) * RW;  // the first of them in the tile
  const int o0 = rr0 * kCols + 4 * ql;
  for (int k = 0; walk.t < t_end; ++k, walk.next()) {
    const BTile tile = walk.tile(a.inst);
    if (per_shot && tile.inst != acc_shot) {
      if (acc_shot >= 0) flush(acc_shot);
      acc_shot = tile.inst;
    }
    // steps of the tile's instance; lam beyond the last is zero, and its
    // imaging pairs are m <= steps - 1
    const int steps = INST ? min(a.inst.box[2 * tile.inst + 1].z, a.nt) : a.nt;
    if (w == 0 && lane < 8) meta[lane] = (&(a.coef + (size_t)tile.inst * a.coef_stride)->k11)[lane];
    load_tile<B, INST>(lev0, lev1, &cur_map, &prev_map, a.cur != nullptr, a.prev != nullptr,
                       a.cur != nullptr && steps >= a.m_hi + 1, a.prev != nullptr && steps >= a.m_hi + 2, tile, k, bar,
                       &guard, err);
    __syncthreads();
    const int gj = tile.y0 - B::kHY + 4 * ql, gi0 = tile.x0 - kH + rr0;
    const int nq = gj >= tile.ys ? max(0, min(4, tile.ye - gj)) : 0;
    const uint32_t region = rows_in<RW>(rr0, tile.xs - tile.x0 + kH, tile.xe - tile.x0 + kH);
    const uint32_t stored = (B::kWhole || (ql >= 1 && ql <= B::kLanes - 2)) && nq > 0
                                ? region & rows_in<RW>(rr0, kH, B::kRows - kH)
                                : 0u;
    const Coefs ks = coefs_in(meta, nq > 0);
    const bool ragged = ((tile.ye - tile.ys) & 3) != 0 && tile.y0 - B::kHY + kCols > tile.ye;
    const int2 recs = a.rec_tile != nullptr ? a.rec_tile[walk.t] : make_int2(0, 0);
    const ptrdiff_t off = (ptrdiff_t)tile.plane * 2 * (ptrdiff_t)Np + (ptrdiff_t)gi0 * a.pitch + gj;
    for (int t = max(1, a.m_hi - steps + 1); t <= a.T; ++t) {
      const int m = a.m_hi - t + 1;
      // the frame whose residuals enter lam^m
      const int frame = (m - 1) % a.stride == 0 ? (m - 1) / a.stride : -1;
      const bool dense = frame >= 0 && a.record == kRecordFields;
      float* lc = (t & 1) ? lev0 : lev1;
      float* lp = (t & 1) ? lev1 : lev0;
      const bool inject = frame >= 0 && recs.y > 0;
      auto add_residuals = [&](float gss) {
        const size_t o = ((size_t)tile.inst * a.nt_out + frame) * a.nrec;
        for (int e = tid; e < recs.y; e += NT) {
          const int2 v = a.rec_ent[recs.x + e];
          atomicAdd(&lp[v.x], gss * a.g_x[o + v.y]);
          atomicAdd(&lp[B::kPlane + v.x], gss * a.g_y[o + v.y]);
        }
        __syncthreads();
      };
      if (ORDER == kOrderTiled && inject) add_residuals(-gs);  // lam^m = ... - (lam^{m+2} - g) + ...
      const float* c0 = lc + o0;  // lam^{m+1}
      float* p0 = lp + o0;        // lam^{m+2}, becomes lam^m
      float* out = t == a.T ? a.out_last : (t == a.T - 1 ? a.out_before : nullptr);
      const uint32_t st = out != nullptr ? stored : 0u;
      // cells with an imaging pair; the others' u is taken as zero
      const uint32_t im = m <= steps - 1 ? stored : 0u;
      float* out0 = out + off;
      float* out1 = out0 + Np;
      const float* u0 = a.u_base + (ptrdiff_t)(m - a.m_base) * (ptrdiff_t)a.u_stride + off;
      const float* u1 = u0 + Np;
      float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      auto rows = [&](auto plain) {
        constexpr bool PLAIN = decltype(plain)::value;
        auto row_at = [&](const float* p) {  // a row of the tile at the lane's quad
          if constexpr (B::kWhole) return whole_row<B>(p, ql);
          else return row_of(q4(*reinterpret_cast<const float4*>(p)));
        };
        auto load_u = [&](int r, float4& x, float4& y) {
          x = y = make_float4(0.f, 0.f, 0.f, 0.f);
          if ((im >> r) & 1u) {
            x = __ldcg(reinterpret_cast<const float4*>(u0));
            y = __ldcg(reinterpret_cast<const float4*>(u1));
          }
          u0 += a.pitch;
          u1 += a.pitch;
        };
        float4 ux4, uy4, nx4, ny4;
        load_u(0, nx4, ny4);
        Row t0 = row_at(c0 - kCols), t1 = row_at(c0 + B::kPlane - kCols);
        Row m0 = row_at(c0), m1 = row_at(c0 + B::kPlane);
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          ux4 = nx4;
          uy4 = ny4;
          if (r + 1 < RW) load_u(r + 1, nx4, ny4);
          const Row b0 = row_at(c0 + (r + 1) * kCols), b1 = row_at(c0 + B::kPlane + (r + 1) * kCols);
          if (PLAIN || ((region >> r) & 1u)) {  // (rows outside the region stay zero)
            const float4 pv0 = *reinterpret_cast<const float4*>(p0 + r * kCols);
            const float4 pv1 = *reinterpret_cast<const float4*>(p0 + B::kPlane + r * kCols);
            const float q0[4] = {pv0.x, pv0.y, pv0.z, pv0.w}, q1[4] = {pv1.x, pv1.y, pv1.z, pv1.w};
            const float ux[4] = {ux4.x, ux4.y, ux4.z, ux4.w}, uy[4] = {uy4.x, uy4.y, uy4.z, uy4.w};
            float v0[4], v1[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const Sums sx = sums_of(t0, m0, b0, q), sy = sums_of(t1, m1, b1, q);
              oper<ORDER>(ks, sx, sy, v0[q], v1[q]);
              image(acc, ux[q], uy[q], sx, sy);
              // (quads outside the region stay zero: their lanes' coefficients are)
              v0[q] = leap(m0.w[q + 1], q0[q], v0[q]);
              v1[q] = leap(m1.w[q + 1], q1[q], v1[q]);
            }
            if (!PLAIN && dense) {
              const size_t o = ((size_t)tile.plane * a.nt_out + frame) * N + (size_t)(gi0 + r) * ny + gj;
#pragma unroll
              for (int q = 0; q < 4; ++q)
                if (q < nq) {
                  v0[q] = fmaf(gs, a.g_x[o + q], v0[q]);
                  v1[q] = fmaf(gs, a.g_y[o + q], v1[q]);
                }
            }
            if (!PLAIN && ragged) {  // the region's last column is inside a quad
              mask_q(v0, nq);
              mask_q(v1, nq);
            }
            const float4 n0 = make_float4(v0[0], v0[1], v0[2], v0[3]), n1 = make_float4(v1[0], v1[1], v1[2], v1[3]);
            *reinterpret_cast<float4*>(p0 + r * kCols) = n0;
            *reinterpret_cast<float4*>(p0 + B::kPlane + r * kCols) = n1;
            if ((st >> r) & 1u) {
              *reinterpret_cast<float4*>(out0) = n0;
              *reinterpret_cast<float4*>(out1) = n1;
            }
          }
          out0 += a.pitch;
          out1 += a.pitch;
          t0 = m0; t1 = m1; m0 = b0; m1 = b1;
        }
      };
      if (any_share<B>(region != 0 && rows_in<RW>(rr0, t, B::kRows - t) != 0)) {
        if (every_share<B>(region == (1u << RW) - 1u) && !ragged && !dense) rows(BoolC<true>{});
        else rows(BoolC<false>{});
        fold_sums(hi, lo, acc);
      }
      __syncthreads();  // lam^m is complete
      if (ORDER != kOrderTiled && inject) {  // ... but for the residuals: lam^m = (...) + g
        add_residuals(gs);
        if (out != nullptr) {
          for (int e = tid; e < recs.y; e += NT) {
            const int c = a.rec_ent[recs.x + e].x, rr = c / kCols, cc = c % kCols;
            if (rr < kH || rr >= B::kRows - kH || cc < B::kHY || cc >= kCols - B::kHY) continue;  // another tile's
            float* o = out + (ptrdiff_t)tile.plane * 2 * (ptrdiff_t)Np + (ptrdiff_t)(tile.x0 - kH + rr) * a.pitch +
                       (tile.y0 - B::kHY + cc);
            o[0] = lp[c];
            o[Np] = lp[B::kPlane + c];
          }
        }
      }
    }
    if (ORDER != kOrderTiled) __syncthreads();  // the stored receivers' cells are read: the next tile may arrive
  }
  if (tid == 0 && pipe_failed(&guard)) pipe_drain(bar, 1, &guard);
  flush(per_shot ? acc_shot : 0);
}

// ------------------------------------------------------------ runs of passes
// Grids whose tiles fit the chip, one per CTA: one cooperative launch makes
// several passes of up to four steps.  A launch per pass costs such a grid as
// much as its arithmetic (a CTA of 512 threads cannot start before the
// previous launch's has left).  Here a tile's state stays in registers: a warp holds RW rows, a lane
// four columns of them; rows beside another warp's go through shared memory
// (one barrier per step), and between passes a CTA waits only for the tiles
// around it, by a flag per tile that counts passes, and reloads its halo.
// A pass writes the two states, of four, that the pass before it has read; the
// tiles around it that read them have counted that pass before it starts, so a
// neighbour is at most one pass ahead.
// Measured, us per pass of four steps, forward / adjoint: 301^2 (8-row tiles)
// 6.0 / 7.5 against 7.5 / 11 with a launch each, 512^2 (24-row tiles) 7.0 /
// 11.1 against 9.4 / 14.  Without waiting for neighbours, halo loads and
// stores a forward pass of 301^2 takes 4.2: what bounds it is the chain of a
// step (exchange, barrier, window, operator) with four warps per scheduler.
struct NoRun {};
__device__ __forceinline__ int passes_of(const NoRun&) { return 1; }
template <class R>
__device__ __forceinline__ int passes_of(const R& r) { return r.n; }

// The passes of a run, copied to shared memory at its start: read from the
// kernel's arguments, every pass would begin with misses of the constant
// cache.  Without a run the launch's arguments are the pass.
template <class R>
struct Passes {
  decltype(R::p) p;
};
template <>
struct Passes<NoRun> {};
template <class A>
__device__ __forceinline__ const A& pass_of(const A& a, const Passes<NoRun>&, int) { return a; }
template <class A, class R>
__device__ __forceinline__ const auto& pass_of(const A&, const Passes<R>& s, int k) { return s.p[k]; }
__device__ __forceinline__ void copy_passes(Passes<NoRun>&, const NoRun&) {}
template <class R>
__device__ __forceinline__ void copy_passes(Passes<R>& s, const R& r) {  // (visible after the next CTA barrier)
  static_assert(sizeof(r.p[0]) % 8 == 0, "copied by words of 8 bytes");
  const uint64_t* src = reinterpret_cast<const uint64_t*>(r.p);
  uint64_t* dst = reinterpret_cast<uint64_t*>(s.p);
  for (int e = threadIdx.x; e < (int)(r.n * sizeof(r.p[0]) / 8); e += blockDim.x) dst[e] = src[e];
}

// A neighbour that has not started yet is waited for (its SM may still be
// busy with another stream's kernel), but not for ever.
constexpr long long kRunWaitCycles = 1ll << 34;

// Waits until the tiles around tile t of a shot's tiles_x x tiles_y have
// counted k passes of this run.  Every thread of the CTA calls it.
template <class R>
__device__ __forceinline__ void wait_neighbours(const R& run, int k, int t, int tiles_x, int tiles_y, int* err) {
  if (k > 0 && threadIdx.x < 9) {
    const int r = t % (tiles_x * tiles_y), xt = r / tiles_y, yt = r - xt * tiles_y;
    const int i = (int)threadIdx.x / 3 - 1, j = (int)threadIdx.x % 3 - 1;
    if (xt + i >= 0 && xt + i < tiles_x && yt + j >= 0 && yt + j < tiles_y) {
      const int* f = run.flags + t + i * tiles_y + j;
      const long long t0 = clock64();
      for (bool done = false; !done;) {
        for (int n = 0; n < 64 && !done; ++n) {
          int v;
          asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
          done = v >= run.epoch + k;
        }
        if (done || *(volatile int*)err != 0) break;
        if (clock64() - t0 > kRunWaitCycles) {
          atomicExch(err, kDeviceTimeout);
          break;
        }
      }
    }
  }
  __syncthreads();
}
__device__ __forceinline__ void wait_neighbours(const NoRun&, int, int, int, int, int*) {}

// Counts the pass once every thread's stores are made.
template <class R>
__device__ __forceinline__ void count_pass(const R& run, int k, int t) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(run.flags + t), "r"(run.epoch + k + 1) : "memory");
  }
}
__device__ __forceinline__ void count_pass(const NoRun&, int, int) {}

constexpr int kRunW = 16;  // warps of a run's CTA

// A warp's part of a run's tile.
template <int RW>
struct RunTile {
  static constexpr int kRows = kRunW * RW;
  static constexpr int kUse = kRows - 2 * kH;
  static constexpr int kPlane = kRows * kBox;
  static constexpr size_t kBytes = (size_t)2 * 2 * kPlane * 4 + 128;  // [parity][component][row][column]
  BTile tile;
  int lane, w, rr0, gi0, gj, nq, pitch;
  uint32_t region, stored;
  bool ragged;
  ptrdiff_t off;
  size_t Np;
  float* ex;  // the lane's quad of the warp's first row, parity 0

  template <class A>
  __device__ __forceinline__ RunTile(const A& a, int t, int tiles_x, int tiles_y, float* sm) {
    lane = threadIdx.x & 31;
    w = threadIdx.x >> 5;
    const int per = tiles_x * tiles_y, shot = t / per, r = t - shot * per, xt = r / tiles_y;
    tile = BTile{shot, shot, xt * kUse, (r - xt * tiles_y) * kBlkCols, 0, 0, a.nx, a.ny};
    rr0 = w * RW;
    gi0 = tile.x0 - kH + rr0;
    gj = tile.y0 - kH + 4 * lane;
    nq = gj >= 0 ? max(0, min(4, a.ny - gj)) : 0;
    region = rows_in<RW>(rr0, kH - tile.x0, a.nx - tile.x0 + kH);
    stored = lane >= 1 && lane <= 30 && nq > 0 ? region & rows_in<RW>(rr0, kH, kRows - kH) : 0u;
    ragged = (a.ny & 3) != 0 && tile.y0 - kH + kBox > a.ny;
    pitch = a.pitch;
    Np = (size_t)a.nx * a.pitch;
    off = (ptrdiff_t)tile.plane * 2 * (ptrdiff_t)Np + (ptrdiff_t)gi0 * a.pitch + gj;
    ex = sm + rr0 * kBox + 4 * lane;
  }
  // Whether a step t later still reads one of the warp's rows.
  __device__ __forceinline__ bool active(int t) const {
    return region != 0 && rr0 + RW > t && rr0 < kRows - t;
  }
  __device__ __forceinline__ float* row(int parity, int c, int r) const {  // r: -1 .. RW
    return ex + parity * 2 * kPlane + c * kPlane + r * kBox;
  }
  // Cells of a state that the tile does not store itself (all: every cell).
  __device__ __forceinline__ void load(const float* s, bool all, Q4 (&x)[RW], Q4 (&y)[RW]) const {
#pragma unroll
    for (int r = 0; r < RW; ++r) {
      if (!all && ((stored >> r) & 1u)) continue;
      const bool on = s != nullptr && nq > 0 && ((region >> r) & 1u);
      const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
      x[r] = q4(on ? __ldcg(reinterpret_cast<const float4*>(s + off + (ptrdiff_t)r * pitch)) : z);
      y[r] = q4(on ? __ldcg(reinterpret_cast<const float4*>(s + off + (ptrdiff_t)r * pitch + Np)) : z);
    }
  }
  // The rows that other warps read (or every row) to shared memory.
  __device__ __forceinline__ void put(int parity, bool all, const Q4 (&x)[RW], const Q4 (&y)[RW]) const {
#pragma unroll
    for (int r = 0; r < RW; ++r) {
      if (r != 0 && r != RW - 1 && !all) continue;
      *reinterpret_cast<float4*>(row(parity, 0, r)) = f4(x[r]);
      *reinterpret_cast<float4*>(row(parity, 1, r)) = f4(y[r]);
    }
  }
  __device__ __forceinline__ Row above(int parity, int c) const {
    return w > 0 ? load_row(row(parity, c, -1)) : Row{{0.f, 0.f, 0.f, 0.f, 0.f, 0.f}};
  }
  __device__ __forceinline__ Row below(int parity, int c) const {
    return w < kRunW - 1 ? load_row(row(parity, c, RW)) : Row{{0.f, 0.f, 0.f, 0.f, 0.f, 0.f}};
  }
  __device__ __forceinline__ void store(float* s, int r, const Q4& x, const Q4& y) const {
    *reinterpret_cast<float4*>(s + off + (ptrdiff_t)r * pitch) = f4(x);
    *reinterpret_cast<float4*>(s + off + (ptrdiff_t)r * pitch + Np) = f4(y);
  }
};

template <int MODE, int RW, int ORDER>
__global__ void __launch_bounds__(32 * kRunW, 1)
    run_fwd_kernel(const BlkFwd a, const __grid_constant__ FwdRun run, int tiles_x, int tiles_y, int* err) {
  extern __shared__ float sm_raw[];
  using R = RunTile<RW>;
  __shared__ Passes<FwdRun> pass;
  copy_passes(pass, run);
  const int t0 = (int)blockIdx.x, ny = a.ny;
  const R g(a, t0, tiles_x, tiles_y, aligned128(sm_raw));
  const size_t N = (size_t)a.nx * ny;
  const Coef* K = a.coef + (size_t)g.tile.inst * a.coef_stride;
  const Coefs ks = coefs_in(&K->k11, g.nq > 0);
  Coefs kc[MODE == kModeFields ? 4 : 1];
  if constexpr (MODE == kModeFields) {
    static_assert(RW == 1, "one row of constants in registers");
    const float q = K->q;
#pragma unroll
    for (int c = 0; c < 4; ++c)
      kc[c] = cell_coefs(a.field, N, (size_t)g.gi0 * ny + g.gj + c, g.region != 0 && c < g.nq, q);
  }
  const bool has_src = a.bx > 0 && a.by > 0;
  const int ox = has_src ? a.src_origin[2 * g.tile.inst] : 0, oy = has_src ? a.src_origin[2 * g.tile.inst + 1] : 0;
  const bool src = has_src && g.gi0 < ox + a.bx && g.gi0 + RW > ox && g.tile.y0 - kH < oy + a.by &&
                   g.tile.y0 - kH + kBox > oy;
  const float kappa = K->kappa;
  const int2 recs = a.rec_tile != nullptr ? a.rec_tile[t0] : make_int2(0, 0);
  Q4 cx[RW], cy[RW], px[RW], py[RW];
  int pending = -1;  // the frame of the newest level, whose receivers are not read yet
  float fs[RW][4];     // the load of the thread's cells
  uint32_t loaded = 0;  // cells inside the load's box, bit 4 r + q
#pragma unroll
  for (int r = 0; r < RW; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int sa = g.gi0 + r - ox, sb = g.gj + q - oy;
      const bool in = src && q < g.nq && (unsigned)sa < (unsigned)a.bx && (unsigned)sb < (unsigned)a.by;
      fs[r][q] = in ? a.src_map[((size_t)g.tile.inst * a.bx + sa) * a.by + sb] : 0.f;
      loaded |= (in ? 1u : 0u) << (4 * r + q);
    }
  auto receivers = [&](int parity) {  // of the level in ex[parity]
    const float* lv = aligned128(sm_raw) + parity * 2 * R::kPlane;
    const size_t o = ((size_t)g.tile.inst * a.nt_out + pending) * a.nrec;
    for (int e = threadIdx.x; e < recs.y; e += 32 * kRunW) {
      const int2 v = a.rec_ent[recs.x + e];
      const int rr = v.x / kBox, cc = v.x % kBox;
      if (rr < kH || rr >= R::kRows - kH || cc < kH || cc >= kBox - kH) continue;  // another tile's
      a.rec_x[o + v.y] = lv[v.x];
      a.rec_y[o + v.y] = lv[R::kPlane + v.x];
    }
  };
  __syncthreads();  // the passes are copied
  for (int k = 0; k < run.n; ++k) {
    const FwdPass& ps = pass.p[k];
    float amp[kBlkSteps];
#pragma unroll
    for (int t = 0; t < kBlkSteps; ++t)  // (in flight over the wait)
      amp[t] = src && t < ps.T ? a.src_signal[(size_t)g.tile.inst * a.nt + ps.i + t] * kappa : 0.f;
    wait_neighbours(run, k, t0, tiles_x, tiles_y, err);
    g.load(ps.cur, k == 0, cx, cy);
    g.load(ps.prev, k == 0, px, py);
    if (ps.out[0] != nullptr) {
#pragma unroll
      for (int r = 0; r < RW; ++r)
        if ((g.stored >> r) & 1u) g.store(ps.out[0], r, cx[r], cy[r]);
    }
    // one step: the new level into the older one's registers
    auto step = [&](int t, float am, const Q4(&ux)[RW], const Q4(&uy)[RW], Q4(&vx)[RW], Q4(&vy)[RW]) {
      const int e = (t - 1) & 1;
      const bool read = pending >= 0 && recs.y > 0;
      g.put(e, read, ux, uy);
      __syncthreads();
      if (read) receivers(e);
      const int frame = ps.frame[t];
      const bool dense = frame >= 0 && a.record == kRecordFields;
      float* out = ps.out[t];
      if (g.active(t)) {
        Row tx = g.above(e, 0), ty = g.above(e, 1), mx = row_of(ux[0]), my = row_of(uy[0]);
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          const Row bx = r + 1 < RW ? row_of(ux[r + 1 < RW ? r + 1 : r]) : g.below(e, 0);
          const Row by = r + 1 < RW ? row_of(uy[r + 1 < RW ? r + 1 : r]) : g.below(e, 1);
          if ((g.region >> r) & 1u) {  // (rows outside the grid stay zero)
            float lx[4], ly[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
              oper<ORDER>(MODE == kModeFields ? kc[MODE == kModeFields ? q : 0] : ks, sums_of(tx, mx, bx, q),
                          sums_of(ty, my, by, q), lx[q], ly[q]);
            if (src) {
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                float& l = a.src_comp == 0 ? lx[q] : ly[q];
                if ((loaded >> (4 * r + q)) & 1u) l = fmaf(am, fs[r][q], l);  // L + amp f, one rounding
              }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              vx[r].v[q] = leap(ux[r].v[q], vx[r].v[q], lx[q]);
              vy[r].v[q] = leap(uy[r].v[q], vy[r].v[q], ly[q]);
            }
            if (g.ragged) {  // the grid's last column is inside a quad
              mask_q(vx[r].v, g.nq);
              mask_q(vy[r].v, g.nq);
            }
            if ((g.stored >> r) & 1u) {
              if (out != nullptr) g.store(out, r, vx[r], vy[r]);
              if (dense) {
                const size_t o = ((size_t)g.tile.plane * a.nt_out + frame) * N + (size_t)(g.gi0 + r) * ny + g.gj;
                if (a.vec) {
                  *reinterpret_cast<float4*>(a.rec_x + o) = f4(vx[r]);
                  *reinterpret_cast<float4*>(a.rec_y + o) = f4(vy[r]);
                } else {
#pragma unroll
                  for (int q = 0; q < 4; ++q)
                    if (q < g.nq) {
                      a.rec_x[o + q] = vx[r].v[q];
                      a.rec_y[o + q] = vy[r].v[q];
                    }
                }
              }
            }
          }
          tx = mx; ty = my; mx = bx; my = by;
        }
      }
      pending = frame;
    };
#pragma unroll
    for (int t = 1; t <= kBlkSteps; t += 2) {
      if (t > ps.T) break;
      step(t, amp[t - 1], cx, cy, px, py);
      if (t == ps.T) {  // (odd: the newest level goes to c)
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          Q4 s = cx[r]; cx[r] = px[r]; px[r] = s;
          s = cy[r]; cy[r] = py[r]; py[r] = s;
        }
        break;
      }
      step(t + 1, amp[t], px, py, cx, cy);
    }
    count_pass(run, k, t0);
  }
  if (pending >= 0 && recs.y > 0) {
    g.put(0, true, cx, cy);
    __syncthreads();
    receivers(0);
  }
}

// As the forward run; the imaging pairs' u is read a step ahead.  The sums
// leave the registers once, at the end of the run.
template <int RW, int ORDER>
__global__ void __launch_bounds__(32 * kRunW, 1)
    run_adj_kernel(const BlkAdj a, const __grid_constant__ AdjRun run, int tiles_x, int tiles_y, int* err) {
  extern __shared__ float sm_raw[];
  using R = RunTile<RW>;
  __shared__ Passes<AdjRun> pass;
  __shared__ float2 red[kRunW][6];
  copy_passes(pass, run);
  const int t0 = (int)blockIdx.x, ny = a.ny;
  const R g(a, t0, tiles_x, tiles_y, aligned128(sm_raw));
  const size_t N = (size_t)a.nx * ny;
  const Coefs ks = coefs_in(&(a.coef + (size_t)g.tile.inst * a.coef_stride)->k11, g.nq > 0);
  const float gs = a.coef->gscale;
  const int2 recs = a.rec_tile != nullptr ? a.rec_tile[t0] : make_int2(0, 0);
  Q4 cx[RW], cy[RW], px[RW], py[RW], ux[RW], uy[RW];
  float hi[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, lo[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  // u^m of the cells with an imaging pair, zero for the others; read from
  // m_base on (what a run's last step would read next is not used)
#pragma unroll
  for (int r = 0; r < RW; ++r) ux[r] = uy[r] = Q4{{0.f, 0.f, 0.f, 0.f}};
  const float* up = nullptr;
  auto load_u = [&](int m, int r) {
    if (m >= a.m_base && ((g.stored >> r) & 1u)) {
      ux[r] = q4(__ldcg(reinterpret_cast<const float4*>(up + (ptrdiff_t)r * g.pitch)));
      uy[r] = q4(__ldcg(reinterpret_cast<const float4*>(up + (ptrdiff_t)r * g.pitch + g.Np)));
    }
  };
  __syncthreads();  // the passes are copied
  {
    const int m = pass.p[0].m_hi;
    up = a.u_base + (ptrdiff_t)(m - a.m_base) * (ptrdiff_t)a.u_stride + g.off;
    if (m <= a.nt - 1) {
#pragma unroll
      for (int r = 0; r < RW; ++r) load_u(m, r);
    }
  }
  for (int k = 0; k < run.n; ++k) {
    const AdjPass& ps = pass.p[k];
    wait_neighbours(run, k, t0, tiles_x, tiles_y, err);
    g.load(ps.cur, k == 0, cx, cy);
    g.load(ps.prev, k == 0, px, py);
    auto step = [&](int t, const Q4(&lx)[RW], const Q4(&ly)[RW], Q4(&vx)[RW], Q4(&vy)[RW]) {
      const int m = ps.m_hi - t + 1, e = (t - 1) & 1;
      const int frame = (m - 1) % a.stride == 0 ? (m - 1) / a.stride : -1;
      const bool dense = frame >= 0 && a.record == kRecordFields;
      g.put(e, false, lx, ly);
      up -= a.u_stride;  // u^{m-1}
      __syncthreads();
      float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (g.active(t)) {
        Row tx = g.above(e, 0), ty = g.above(e, 1), mx = row_of(lx[0]), my = row_of(ly[0]);
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          const Row bx = r + 1 < RW ? row_of(lx[r + 1 < RW ? r + 1 : r]) : g.below(e, 0);
          const Row by = r + 1 < RW ? row_of(ly[r + 1 < RW ? r + 1 : r]) : g.below(e, 1);
          if ((g.region >> r) & 1u) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const Sums sx = sums_of(tx, mx, bx, q), sy = sums_of(ty, my, by, q);
              float ax, ay;
              oper<ORDER>(ks, sx, sy, ax, ay);
              image(acc, ux[r].v[q], uy[r].v[q], sx, sy);
              vx[r].v[q] = leap(lx[r].v[q], vx[r].v[q], ax);
              vy[r].v[q] = leap(ly[r].v[q], vy[r].v[q], ay);
            }
            if (dense) {
              const size_t o = ((size_t)g.tile.plane * a.nt_out + frame) * N + (size_t)(g.gi0 + r) * ny + g.gj;
#pragma unroll
              for (int q = 0; q < 4; ++q)
                if (q < g.nq) {
                  vx[r].v[q] = fmaf(gs, a.g_x[o + q], vx[r].v[q]);
                  vy[r].v[q] = fmaf(gs, a.g_y[o + q], vy[r].v[q]);
                }
            }
            if (g.ragged) {  // the grid's last column is inside a quad
              mask_q(vx[r].v, g.nq);
              mask_q(vy[r].v, g.nq);
            }
          }
          load_u(m - 1, r);
          tx = mx; ty = my; mx = bx; my = by;
        }
        fold_sums(hi, lo, acc);
      } else {
#pragma unroll
        for (int r = 0; r < RW; ++r) load_u(m - 1, r);
      }
      if (frame >= 0 && recs.y > 0) {  // lam^m = (...) + g at the receivers' cells
        g.put(e ^ 1, true, vx, vy);
        __syncthreads();
        float* lv = aligned128(sm_raw) + (e ^ 1) * 2 * R::kPlane;
        const size_t o = ((size_t)g.tile.inst * a.nt_out + frame) * a.nrec;
        for (int i = threadIdx.x; i < recs.y; i += 32 * kRunW) {
          const int2 v = a.rec_ent[recs.x + i];
          atomicAdd(&lv[v.x], gs * a.g_x[o + v.y]);
          atomicAdd(&lv[R::kPlane + v.x], gs * a.g_y[o + v.y]);
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          vx[r] = q4(*reinterpret_cast<const float4*>(g.row(e ^ 1, 0, r)));
          vy[r] = q4(*reinterpret_cast<const float4*>(g.row(e ^ 1, 1, r)));
        }
      }
      float* out = t == ps.T ? ps.out_last : (t == ps.T - 1 ? ps.out_before : nullptr);
      if (out != nullptr) {
#pragma unroll
        for (int r = 0; r < RW; ++r)
          if ((g.stored >> r) & 1u) g.store(out, r, vx[r], vy[r]);
      }
    };
#pragma unroll
    for (int t = 1; t <= kBlkSteps; t += 2) {
      if (t > ps.T) break;
      step(t, cx, cy, px, py);
      if (t == ps.T) {
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          Q4 s = cx[r]; cx[r] = px[r]; px[r] = s;
          s = cy[r]; cy[r] = py[r]; py[r] = s;
        }
        break;
      }
      step(t + 1, px, py, cx, cy);
    }
    count_pass(run, k, t0);
  }
  const size_t row = a.coef_stride != 0 ? (size_t)g.tile.inst * kTiledRowsPerShot + blockIdx.x : (size_t)blockIdx.x;
  flush_sums<kRunW>(hi, lo, red, a.partials + row * 8);
}

// ------------------------------------------- adjoint, degradation map
// A^T lam = A0((1 - D) lam): the update's stencils run over the weighted
// lam^{m+1}, its centre stays unweighted.  The imaging sum is kept per cell,
// lam^{m+1} . (A0 u^m), so u's own stencils are needed: a second pass over the
// warp's rows, with u's rows read from global memory (halo columns by the
// outer lanes) one row ahead.
template <int W, int RW, int CTAS>
__global__ void __launch_bounds__(32 * W, CTAS)
    blk_adj_d_kernel(const BlkAdj a, const __grid_constant__ CUtensorMap cur_map,
                     const __grid_constant__ CUtensorMap prev_map, int tiles_x, int tiles_y, int ntiles, int* err) {
  extern __shared__ float sm_raw[];
  float* sm = aligned128(sm_raw);
  using B = BlkTile<W, RW>;
  constexpr int NT = B::kThreads;
  float* lev0 = sm + kBox;
  float* lev1 = lev0 + B::kLevel;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + B::kFloats + B::kMeta);
  __shared__ PipeGuard guard;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int nx = a.nx, ny = a.ny;
  const size_t N = (size_t)nx * ny, Np = (size_t)nx * a.pitch;
  grid_dep_trigger();
  if (tid == 0) {
    prefetch_map(&cur_map);
    prefetch_map(&prev_map);
    bar_init(bar);
    pipe_init(&guard);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < kBox) sm[tid] = sm[B::kFloats - kBox + tid] = 0.f;
  BWalk<false, B::kUse> walk;
  walk.init((int)blockIdx.x, (int)gridDim.x, tiles_x, tiles_y, nx, ny);
  __syncthreads();
  grid_dep_wait();  // the states of the previous launch are complete from here on
  const float gs = a.coef->gscale;
  const int rr0 = w * RW;  // first row of the warp in the tile
  const int o0 = rr0 * kBox + 4 * lane;
  for (int k = 0; walk.t < ntiles; ++k, walk.next()) {
    const BTile tile = walk.tile(a.inst);
    const int2 recs = a.rec_tile != nullptr ? a.rec_tile[walk.t] : make_int2(0, 0);
    load_tile<B, false>(lev0, lev1, &cur_map, &prev_map, a.cur != nullptr, a.prev != nullptr, a.cur != nullptr,
                        a.prev != nullptr, tile, k, bar, &guard, err);
    __syncthreads();
    const int gj = tile.y0 - kH + 4 * lane, gi0 = tile.x0 - kH + rr0;
    const int nq = gj >= 0 ? max(0, min(4, ny - gj)) : 0;
    const uint32_t region = rows_in<RW>(rr0, kH - tile.x0, nx - tile.x0 + kH);
    const uint32_t rows_st = region & rows_in<RW>(rr0, kH, B::kRows - kH);
    const uint32_t stored = lane >= 1 && lane <= 30 && nq > 0 ? rows_st : 0u;
    const Coefs ks = coefs_in(&a.coef->k11, nq > 0);
    const bool ragged = (ny & 3) != 0 && tile.y0 - kH + kBox > ny;
    const ptrdiff_t off = (ptrdiff_t)tile.plane * 2 * (ptrdiff_t)Np + (ptrdiff_t)gi0 * a.pitch + gj;
    auto weights = [&](int gi, float(&wv)[4]) {  // 1 - D (zero outside the grid)
      const float* d = a.field + (ptrdiff_t)gi * ny + gj;
      const bool in = gi >= 0 && gi < nx;
      if (a.vec_field) {
        const float4 v = in && nq > 0 ? __ldg(reinterpret_cast<const float4*>(d)) : make_float4(1.f, 1.f, 1.f, 1.f);
        wv[0] = 1.f - v.x; wv[1] = 1.f - v.y; wv[2] = 1.f - v.z; wv[3] = 1.f - v.w;
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) wv[c] = in && c < nq ? 1.f - __ldg(d + c) : 0.f;
      }
    };
    for (int t = 1; t <= a.T; ++t) {
      const int m = a.m_hi - t + 1;
      const int frame = (m - 1) % a.stride == 0 ? (m - 1) / a.stride : -1;
      const bool dense = frame >= 0 && a.record == kRecordFields;
      float* lc = (t & 1) ? lev0 : lev1;
      float* lp = (t & 1) ? lev1 : lev0;
      if (frame >= 0 && recs.y > 0) {  // lam^m = ... - (lam^{m+2} - g) + ...
        const size_t o = ((size_t)tile.inst * a.nt_out + frame) * a.nrec;
        for (int e = tid; e < recs.y; e += NT) {
          const int2 v = a.rec_ent[recs.x + e];
          atomicAdd(&lp[v.x], -gs * a.g_x[o + v.y]);
          atomicAdd(&lp[B::kPlane + v.x], -gs * a.g_y[o + v.y]);
        }
        __syncthreads();
      }
      const float* c0 = lc + o0;  // lam^{m+1}
      float* p0 = lp + o0;        // lam^{m+2}, becomes lam^m
      float* out = t == a.T ? a.out_last : (t == a.T - 1 ? a.out_before : nullptr);
      const uint32_t st = out != nullptr ? stored : 0u;
      if (region != 0 && rows_in<RW>(rr0, t, B::kRows - t) != 0) {
        float* out0 = out + off;
        float* out1 = out0 + Np;
        // a row of lam^{m+1}: the quads, and their weighted windows
        struct LRow {
          Q4 x, y;
          Row wx, wy;
        };
        float wn[4];
        auto lam_row = [&](int r) {
          LRow l;
          l.x = q4(*reinterpret_cast<const float4*>(c0 + r * kBox));
          l.y = q4(*reinterpret_cast<const float4*>(c0 + B::kPlane + r * kBox));
          Q4 vx, vy;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            vx.v[q] = __fmul_rn(wn[q], l.x.v[q]);
            vy.v[q] = __fmul_rn(wn[q], l.y.v[q]);
          }
          l.wx = row_of(vx);
          l.wy = row_of(vy);
          return l;
        };
        weights(gi0 - 1, wn);
        LRow tr = lam_row(-1);
        weights(gi0, wn);
        LRow mr = lam_row(0);
        weights(gi0 + 1, wn);
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          const LRow br = lam_row(r + 1);
          if (r + 1 < RW) weights(gi0 + r + 2, wn);
          if ((region >> r) & 1u) {
            const float4 pv0 = *reinterpret_cast<const float4*>(p0 + r * kBox);
            const float4 pv1 = *reinterpret_cast<const float4*>(p0 + B::kPlane + r * kBox);
            const float q0[4] = {pv0.x, pv0.y, pv0.z, pv0.w}, q1[4] = {pv1.x, pv1.y, pv1.z, pv1.w};
            float v0[4], v1[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              oper<kOrderTiled>(ks, sums_of(tr.wx, mr.wx, br.wx, q), sums_of(tr.wy, mr.wy, br.wy, q), v0[q], v1[q]);
              v0[q] = leap(mr.x.v[q], q0[q], v0[q]);
              v1[q] = leap(mr.y.v[q], q1[q], v1[q]);
            }
            if (dense) {
              const size_t o = ((size_t)tile.plane * a.nt_out + frame) * N + (size_t)(gi0 + r) * ny + gj;
#pragma unroll
              for (int q = 0; q < 4; ++q)
                if (q < nq) {
                  v0[q] = fmaf(gs, a.g_x[o + q], v0[q]);
                  v1[q] = fmaf(gs, a.g_y[o + q], v1[q]);
                }
            }
            if (ragged) {  // the grid's last column is inside a quad
              mask_q(v0, nq);
              mask_q(v1, nq);
            }
            const float4 n0 = make_float4(v0[0], v0[1], v0[2], v0[3]), n1 = make_float4(v1[0], v1[1], v1[2], v1[3]);
            *reinterpret_cast<float4*>(p0 + r * kBox) = n0;
            *reinterpret_cast<float4*>(p0 + B::kPlane + r * kBox) = n1;
            if ((st >> r) & 1u) {
              *reinterpret_cast<float4*>(out0) = n0;
              *reinterpret_cast<float4*>(out1) = n1;
            }
          }
          out0 += a.pitch;
          out1 += a.pitch;
          tr = mr;
          mr = br;
        }
      }
      if (m <= a.nt - 1 && rows_st != 0) {
        const float* u0 = a.u_base + (ptrdiff_t)(m - a.m_base) * (ptrdiff_t)a.u_stride + off;
        auto load_u = [&](int r, float4& x, float4& y) {
          x = y = make_float4(0.f, 0.f, 0.f, 0.f);
          if (gi0 + r >= 0 && gi0 + r < nx && nq > 0) {
            const float* u = u0 + (ptrdiff_t)r * a.pitch;
            x = __ldcg(reinterpret_cast<const float4*>(u));
            y = __ldcg(reinterpret_cast<const float4*>(u + Np));
          }
        };
        float* ga = a.gacc + (size_t)tile.plane * N + (ptrdiff_t)gi0 * ny + gj;
        float4 nx4, ny4, tx4, ty4;
        load_u(-1, tx4, ty4);
        load_u(0, nx4, ny4);
        Row t0 = row_of(q4(tx4)), t1 = row_of(q4(ty4));
        load_u(1, tx4, ty4);
        Row m0 = row_of(q4(nx4)), m1 = row_of(q4(ny4));
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          const Row b0 = row_of(q4(tx4)), b1 = row_of(q4(ty4));
          if (r + 1 < RW) load_u(r + 2, tx4, ty4);
          if ((stored >> r) & 1u) {
            const float4 lx = *reinterpret_cast<const float4*>(c0 + r * kBox);
            const float4 ly = *reinterpret_cast<const float4*>(c0 + B::kPlane + r * kBox);
            const float l0[4] = {lx.x, lx.y, lx.z, lx.w}, l1[4] = {ly.x, ly.y, ly.z, ly.w};
            float gv[4];
            if (a.vec_field) {
              const float4 g = *reinterpret_cast<const float4*>(ga);
              gv[0] = g.x; gv[1] = g.y; gv[2] = g.z; gv[3] = g.w;
            } else {
#pragma unroll
              for (int q = 0; q < 4; ++q) gv[q] = q < nq ? ga[q] : 0.f;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              float Lx, Ly;
              oper<kOrderPlain>(ks, sums_of(t0, m0, b0, q), sums_of(t1, m1, b1, q), Lx, Ly);
              gv[q] += fmaf(l0[q], Lx, __fmul_rn(l1[q], Ly));
            }
            if (a.vec_field) {
              *reinterpret_cast<float4*>(ga) = make_float4(gv[0], gv[1], gv[2], gv[3]);
            } else {
#pragma unroll
              for (int q = 0; q < 4; ++q)
                if (q < nq) ga[q] = gv[q];
            }
          }
          ga += ny;
          t0 = m0; t1 = m1; m0 = b0; m1 = b1;
        }
      }
      __syncthreads();  // lam^m is complete
    }
  }
  if (tid == 0 && pipe_failed(&guard)) pipe_drain(bar, 1, &guard);
}

// ------------------------------------------- adjoint, six constant planes
// One row of 128 columns per warp; the thread keeps its cells' two levels,
// constants and six running gradients in registers for the launch.  A^T
// applies the stencils to products of each cell's own constants with lam:
// the four products whose vertical or diagonal neighbours are needed go
// through shared memory (one CTA barrier per step), the others' column
// neighbours come by lane shuffles.  Recorded residuals are summed per cell in
// shared memory, the thread's receiver and its residual loaded before the
// step's first barrier (us per forward and adjoint step, every thread looking
// for its own cells in the tile's list / the plain kernels / here: 301^2 with
// 1536 receivers in a corner 97 / 15.7 / 6.1, with every cell 132 / 412 / 9.3,
// with 256 spread over it 4.9 / 9.9 / 4.3).
template <int W, bool RUN>
__global__ void __launch_bounds__(32 * W, 1)
    blk_adj_f_kernel(const BlkAdj a, const __grid_constant__ std::conditional_t<RUN, AdjRun, NoRun> run, int tiles_x,
                     int tiles_y, int ntiles, int* err) {
  extern __shared__ float sm_raw[];
  float* ex = aligned128(sm_raw);  // [parity][product][row][128]
  constexpr int kRows = W, kUse = W - 2 * kH;
  float* res = ex + 2 * 4 * kRows * kBox;  // [component][row][128], with receivers
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int nx = a.nx, ny = a.ny;
  const size_t N = (size_t)nx * ny, Np = (size_t)nx * a.pitch;
  grid_dep_trigger();
  BWalk<false, kUse> walk;
  walk.init((int)blockIdx.x, (int)gridDim.x, tiles_x, tiles_y, nx, ny);
  const float qf = a.coef->q;
  __shared__ Passes<std::conditional_t<RUN, AdjRun, NoRun>> pass;
  copy_passes(pass, run);
  for (; walk.t < ntiles; walk.next()) {
    const BTile tile = walk.tile(a.inst);
    const int2 recs = a.rec_tile != nullptr ? a.rec_tile[walk.t] : make_int2(0, 0);
    const int gj = tile.y0 - kH + 4 * lane, gi = tile.x0 - kH + w;
    const bool row_in = gi >= 0 && gi < nx;
    const int nq = row_in && gj >= 0 ? max(0, min(4, ny - gj)) : 0;
    const bool stored = w >= kH && w < kRows - kH && lane >= 1 && lane <= 30 && nq > 0;
    float C[6][4];
#pragma unroll
    for (int c = 0; c < 6; ++c)
#pragma unroll
      for (int q = 0; q < 4; ++q) C[c][q] = q < nq ? __ldg(a.field + c * N + (size_t)gi * ny + gj + q) : 0.f;
    grid_dep_wait();  // the states of the previous launch are complete from here on
    const float gs = a.coef->gscale;
    const ptrdiff_t off = (ptrdiff_t)tile.plane * 2 * (ptrdiff_t)Np + (ptrdiff_t)gi * a.pitch + gj;
    auto load_state = [&](const float* s, ptrdiff_t o, bool in, float(&x)[4], float(&y)[4]) {
      const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 vx = in ? __ldcg(reinterpret_cast<const float4*>(s + o)) : z;
      const float4 vy = in ? __ldcg(reinterpret_cast<const float4*>(s + o + Np)) : z;
      x[0] = vx.x; x[1] = vx.y; x[2] = vx.z; x[3] = vx.w;
      y[0] = vy.x; y[1] = vy.y; y[2] = vy.z; y[3] = vy.w;
    };
    float cx[4], cy[4], px[4], py[4], ga[6][4];
    // the running sums of the thread's cells, a step's terms added to them one
    // by one as in the per-step kernels
    float* const gc = a.gacc + (size_t)tile.plane * 6 * N + (size_t)gi * ny + gj;
#pragma unroll
    for (int c = 0; c < 6; ++c)
#pragma unroll
      for (int q = 0; q < 4; ++q) ga[c][q] = stored && q < nq ? gc[c * N + q] : 0.f;
    int n = 0;  // steps so far
    for (int k = 0; k < passes_of(run); ++k) {
    if (RUN) wait_neighbours(run, k, walk.t, tiles_x, tiles_y, err);
    const auto& ps = pass_of(a, pass, k);
    if (!(k > 0 && stored)) {
      load_state(ps.cur, off, ps.cur != nullptr && nq > 0, cx, cy);
      load_state(ps.prev, off, ps.prev != nullptr && nq > 0, px, py);
    }
    for (int t = 1; t <= ps.T; ++t, ++n) {
      const int m = ps.m_hi - t + 1;
      const int frame = (m - 1) % a.stride == 0 ? (m - 1) / a.stride : -1;
      // the products of this row, those the rows above and below need in
      // shared memory (which of a sum's products is rounded is as in the plain
      // kernels: the states are theirs bit for bit)
      Q4 s0, s1, s2, s3, s4, s5;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float lx = cx[q], ly = cy[q], c1266 = C[2][q] + C[5][q];
        s0.v[q] = fmaf(C[0][q], lx, __fmul_rn(C[3][q], ly));
        s1.v[q] = fmaf(C[4][q], ly, __fmul_rn(C[5][q], lx));
        s2.v[q] = fmaf(2.f * C[3][q], lx, __fmul_rn(c1266, ly));
        s3.v[q] = fmaf(C[3][q], lx, __fmul_rn(C[5][q], ly));
        s4.v[q] = fmaf(C[1][q], ly, __fmul_rn(C[4][q], lx));
        s5.v[q] = fmaf(2.f * C[4][q], ly, __fmul_rn(c1266, lx));
      }
      float* e = ex + (n & 1) * (4 * kRows * kBox) + w * kBox + 4 * lane;
      *reinterpret_cast<float4*>(e) = f4(s0);
      *reinterpret_cast<float4*>(e + kRows * kBox) = f4(s2);
      *reinterpret_cast<float4*>(e + 2 * kRows * kBox) = f4(s3);
      *reinterpret_cast<float4*>(e + 3 * kRows * kBox) = f4(s5);
      const bool inject = frame >= 0 && recs.y > 0;
      float* const my_res = res + w * kBox + 4 * lane;
      int2 rv = make_int2(0, 0);
      float rgx = 0.f, rgy = 0.f;  // the thread's first receiver, in flight over the barrier
      if (inject) {
        *reinterpret_cast<float4*>(my_res) = *reinterpret_cast<float4*>(my_res + kRows * kBox) =
            make_float4(0.f, 0.f, 0.f, 0.f);
        if (tid < recs.y) {
          rv = a.rec_ent[recs.x + tid];
          const size_t o = ((size_t)tile.inst * a.nt_out + frame) * a.nrec + rv.y;
          rgx = gs * a.g_x[o];
          rgy = gs * a.g_y[o];
        }
      }
      // (the u rows of the imaging sums, in flight over the barrier)
      const bool im = m <= a.nt - 1 && w >= kH && w < kRows - kH && row_in;
      float ux[3][4], uy[3][4];
      if (im) {
        const float* u = a.u_base + (ptrdiff_t)(m - a.m_base) * (ptrdiff_t)a.u_stride;
#pragma unroll
        for (int d = 0; d < 3; ++d)
          load_state(u, off + (ptrdiff_t)(d - 1) * a.pitch, nq > 0 && gi + d - 1 >= 0 && gi + d - 1 < nx, ux[d], uy[d]);
      }
      __syncthreads();
      if (inject) {
        if (tid < recs.y) {
          atomicAdd(&res[rv.x], rgx);
          atomicAdd(&res[kRows * kBox + rv.x], rgy);
        }
        const size_t o = ((size_t)tile.inst * a.nt_out + frame) * a.nrec;
        for (int r = tid + 32 * W; r < recs.y; r += 32 * W) {
          const int2 v = a.rec_ent[recs.x + r];
          atomicAdd(&res[v.x], gs * a.g_x[o + v.y]);
          atomicAdd(&res[kRows * kBox + v.x], gs * a.g_y[o + v.y]);
        }
        __syncthreads();
      }
      if (row_in && w >= t && w < kRows - t) {
        const float* up = e - (w > 0 ? kBox : 0);
        const float* dn = e + (w < kRows - 1 ? kBox : 0);
        auto quad = [](const float* p) { return q4(*reinterpret_cast<const float4*>(p)); };
        const Row r1 = row_of(s1), r4 = row_of(s4);
        float vx[4], vy[4];
        {
          const Q4 t0 = quad(up), b0 = quad(dn);
          const Row t2 = row_of(quad(up + kRows * kBox)), b2 = row_of(quad(dn + kRows * kBox));
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float xx = fmaf(-2.f, s0.v[q], t0.v[q] + b0.v[q]);
            const float yy = fmaf(-2.f, s1.v[q], r1.w[q] + r1.w[q + 2]);
            const float xy = (b2.w[q + 2] + t2.w[q]) - (b2.w[q] + t2.w[q + 2]);
            vx[q] = fmaf(qf, fmaf(0.25f, xy, xx + yy), fmaf(2.f, cx[q], -px[q]));
          }
        }
        {
          const Q4 t3 = quad(up + 2 * kRows * kBox), b3 = quad(dn + 2 * kRows * kBox);
          const Row t5 = row_of(quad(up + 3 * kRows * kBox)), b5 = row_of(quad(dn + 3 * kRows * kBox));
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float xx = fmaf(-2.f, s3.v[q], t3.v[q] + b3.v[q]);
            const float yy = fmaf(-2.f, s4.v[q], r4.w[q] + r4.w[q + 2]);
            const float xy = (b5.w[q + 2] + t5.w[q]) - (b5.w[q] + t5.w[q + 2]);
            vy[q] = fmaf(qf, fmaf(0.25f, xy, xx + yy), fmaf(2.f, cy[q], -py[q]));
          }
        }
        if (frame >= 0 && a.record == kRecordFields) {
          const size_t o = ((size_t)tile.plane * a.nt_out + frame) * N + (size_t)gi * ny + gj;
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (q < nq) {
              vx[q] = fmaf(gs, a.g_x[o + q], vx[q]);
              vy[q] = fmaf(gs, a.g_y[o + q], vy[q]);
            }
        }
        if (inject) {
          const Q4 rx = q4(*reinterpret_cast<const float4*>(my_res));
          const Q4 ry = q4(*reinterpret_cast<const float4*>(my_res + kRows * kBox));
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            vx[q] += rx.v[q];
            vy[q] += ry.v[q];
          }
        }
        mask_q(vx, nq);  // cells outside the grid stay zero
        mask_q(vy, nq);
        if (im) {  // lam^{m+1} against the derivatives of A u^m
          const Row t0 = row_of(Q4{{ux[0][0], ux[0][1], ux[0][2], ux[0][3]}});
          const Row m0 = row_of(Q4{{ux[1][0], ux[1][1], ux[1][2], ux[1][3]}});
          const Row b0 = row_of(Q4{{ux[2][0], ux[2][1], ux[2][2], ux[2][3]}});
          const Row t1 = row_of(Q4{{uy[0][0], uy[0][1], uy[0][2], uy[0][3]}});
          const Row m1 = row_of(Q4{{uy[1][0], uy[1][1], uy[1][2], uy[1][3]}});
          const Row b1 = row_of(Q4{{uy[2][0], uy[2][1], uy[2][2], uy[2][3]}});
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const Sums sx = sums_of(t0, m0, b0, q), sy = sums_of(t1, m1, b1, q);
            const float lx = cx[q], ly = cy[q];
            ga[0][q] = fmaf(lx, sx.xx, ga[0][q]);
            ga[1][q] = fmaf(ly, sy.yy, ga[1][q]);
            ga[2][q] += fmaf(ly, sx.xy, __fmul_rn(lx, sy.xy));
            ga[3][q] += fmaf(ly, sx.xx, __fmul_rn(lx, fmaf(0.5f, sx.xy, sy.xx)));
            ga[4][q] += fmaf(lx, sy.yy, __fmul_rn(ly, fmaf(0.5f, sy.xy, sx.yy)));
            ga[5][q] += fmaf(lx, sx.yy, __fmul_rn(ly, sy.xx));
          }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          px[q] = cx[q];
          py[q] = cy[q];
          cx[q] = vx[q];
          cy[q] = vy[q];
        }
      }
    }
    if (stored) {
      // cur holds lam of the last step, prev of the one before
      *reinterpret_cast<float4*>(ps.out_last + off) = make_float4(cx[0], cx[1], cx[2], cx[3]);
      *reinterpret_cast<float4*>(ps.out_last + off + Np) = make_float4(cy[0], cy[1], cy[2], cy[3]);
      if (ps.out_before != nullptr) {
        *reinterpret_cast<float4*>(ps.out_before + off) = make_float4(px[0], px[1], px[2], px[3]);
        *reinterpret_cast<float4*>(ps.out_before + off + Np) = make_float4(py[0], py[1], py[2], py[3]);
      }
    }
    if (RUN) count_pass(run, k, walk.t);
    }
    if (stored) {
#pragma unroll
      for (int c = 0; c < 6; ++c)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (q < nq) gc[c * N + q] = ga[c][q];
    }
    __syncthreads();  // the products are read: the next tile's may be written
  }
}

// ------------------------------------------------------- instance tiles
// Block b writes the tiles of instance d.id[b] (entry base[b] + xt * tiles_y
// + yt for the tile at rows x0 + tile_rows xt, columns y0 + tile_cols yt) and
// its box.
__global__ void inst_table_kernel(const InstDesc d, int4* __restrict__ tiles, int4* __restrict__ box) {
  const int b = blockIdx.x;
  const int k = d.id[b];
  const int tiles_y = (d.ny[b] + d.tile_cols - 1) / d.tile_cols;
  const int n = tiles_y * ((d.nx[b] + d.tile_rows - 1) / d.tile_rows);
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    const int xt = t / tiles_y, yt = t - xt * tiles_y;
    // the entry: instance, tile origin, instance region (16-bit pairs)
    const unsigned rx = (unsigned)(d.x0[b] + d.tile_rows * xt), ry = (unsigned)(d.y0[b] + d.tile_cols * yt);
    const unsigned xs = (unsigned)d.x0[b], ys = (unsigned)d.y0[b];
    const unsigned xe = xs + (unsigned)d.nx[b], ye = ys + (unsigned)d.ny[b];
    tiles[d.base[b] + t] = make_int4(k, (int)(rx | (ry << 16)), (int)(xs | (ys << 16)), (int)(xe | (ye << 16)));
  }
  if (threadIdx.x == 0) {
    box[2 * k] = make_int4(d.x0[b], d.y0[b], d.x0[b] + d.nx[b], d.y0[b] + d.ny[b]);
    box[2 * k + 1] = make_int4(d.base[b], tiles_y, d.nt[b], 0);
  }
}

// ------------------------------------------------- receivers of the tiles
// The receivers whose cells lie in a tile with its halo, for every tile of a
// call: tile[t] = (first entry, entries), an entry = (cell in the tile's
// planes, receiver number).  Counted, given room and filled by three small
// kernels (the order inside a tile does not matter).  A receiver outside the
// grid is in no tile: the counting kernel writes its nt_out frames (zeros).
struct RecPlace {  // the tiles (at most 2 x 2) around a cell
  int x0, x1, y0, y1, base, tiles_y, oi, oj;
  __device__ __forceinline__ bool find(int idx, int s, int nx, int ny, const BlkShape& g, int tiles_x, int ty,
                                       const int4* box) {
    if (idx < 0 || (int64_t)idx >= (int64_t)nx * ny) return false;  // out of range: ignored
    int gi = idx / ny, gj = idx - gi * ny;
    if (box != nullptr) {
      const int4 r = box[2 * s], m = box[2 * s + 1];
      if (gi < r.x || gi >= r.z || gj < r.y || gj >= r.w) return false;
      gi -= r.x;
      gj -= r.y;
      base = m.x;
      tiles_y = m.y;
      tiles_x = (r.z - r.x + g.rows - 1) / g.rows;
    } else {
      base = s * tiles_x * ty;
      tiles_y = ty;
    }
    oi = gi + kH;
    oj = gj + g.hy;
    x1 = min(oi / g.rows, tiles_x - 1);
    x0 = max((oi - 2 * kH) / g.rows, 0);  // first tile whose last row reaches the cell
    y1 = min(oj / g.cols, tiles_y - 1);
    y0 = max((oj - 2 * g.hy) / g.cols, 0);
    return true;
  }
};

template <bool FILL>
__global__ void rec_tiles_kernel(const int32_t* __restrict__ rec_idx, int S, int nrec, int nx, int ny, const BlkShape g,
                                 int tiles_x, int tiles_y, const int4* __restrict__ box, int* __restrict__ count,
                                 int2* __restrict__ tile, int2* __restrict__ ent, float* __restrict__ tr_x,
                                 float* __restrict__ tr_y, int nt_out) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= S * nrec) return;
  const int s = e / nrec;
  RecPlace p;
  if (!p.find(rec_idx[e], s, nx, ny, g, tiles_x, tiles_y, box)) {
    if (!FILL && tr_x != nullptr)
      for (int k = 0; k < nt_out; ++k) {
        const size_t o = ((size_t)s * nt_out + k) * nrec + (e - s * nrec);
        tr_x[o] = tr_y[o] = 0.f;
      }
    return;
  }
  const int width = g.cols + 2 * g.hy;
  for (int xt = p.x0; xt <= p.x1; ++xt)
    for (int yt = p.y0; yt <= p.y1; ++yt) {
      const int rr = p.oi - xt * g.rows, cc = p.oj - yt * g.cols;
      if (rr < 0 || rr >= g.rows + 2 * kH || cc < 0 || cc >= width) continue;
      const int t = p.base + xt * p.tiles_y + yt;
      if (FILL) ent[tile[t].x + atomicAdd(&tile[t].y, 1)] = make_int2(rr * width + cc, e - s * nrec);
      else atomicAdd(&count[t], 1);
    }
}

__global__ void rec_base_kernel(int* __restrict__ count, int ntiles, int2* __restrict__ tile) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntiles) return;
  const int n = count[t];
  tile[t] = make_int2(n > 0 ? atomicAdd(&count[ntiles], n) : 0, 0);
}

// ----------------------------------------------------------------- host
PFN_cuTensorMapEncodeTiled_v12000 blk_encode_fn() {
  static std::mutex mu;
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  std::lock_guard<std::mutex> lock(mu);
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

// Tensor map over S shots of [comp][nx][pitch] floats, columns ny .. pitch - 1
// read as zeros: dims (ny, nx, 2 S).
bool blk_map(CUtensorMap* m, const float* base, int nx, int ny, int pitch, int S, int bw, int bh) {
  auto fn = blk_encode_fn();
  if (fn == nullptr || base == nullptr) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)ny, (cuuint64_t)nx, (cuuint64_t)2 * S};
  const cuuint64_t strides[2] = {(cuuint64_t)pitch * 4, (cuuint64_t)nx * pitch * 4};
  const cuuint32_t box[3] = {(cuuint32_t)bw, (cuuint32_t)bh, 2};
  const cuuint32_t estr[3] = {1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int MODE, class B, int CTAS, bool INST, int ORDER>
cudaError_t fwd_t(const BlkFwd& a, int* err, cudaStream_t st) {
  constexpr size_t smem = B::kBytes;
  static OncePerDevice once;
  const cudaError_t ready = once([] {
    return cudaFuncSetAttribute(blk_fwd_kernel<MODE, B, INST, ORDER, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  });
  if (ready != cudaSuccess) return ready;
  const int planes = INST ? 1 : a.S;
  const float* any = a.cur ? a.cur : a.out[a.T];  // (a level that is zero is not loaded)
  CUtensorMap cm, pm;
  if (!blk_map(&cm, any, a.nx, a.ny, a.pitch, planes, B::kCols, B::kRows) ||
      !blk_map(&pm, a.prev ? a.prev : any, a.nx, a.ny, a.pitch, planes, B::kCols, B::kRows))
    return cudaErrorNotSupported;
  const int tiles_x = (a.nx + B::kUse - 1) / B::kUse, tiles_y = (a.ny + B::kUseY - 1) / B::kUseY;
  const int ntiles = INST ? a.inst.ntiles : a.S * tiles_x * tiles_y;
  const int grid = ntiles < CTAS * device_info().sms ? ntiles : CTAS * device_info().sms;
  const double cells = INST ? (double)ntiles * B::kUse * B::kUseY : (double)a.S * a.nx * a.ny;
  int stores = 0;
  for (int t = 0; t <= a.T; ++t) stores += a.out[t] != nullptr ? 1 : 0;
  return tracked_launch(kProfForward, st, [&] {
    launch_step_kernel(blk_fwd_kernel<MODE, B, INST, ORDER, CTAS>, dim3(grid), dim3(B::kThreads), smem, st, a.chained != 0, a, cm, pm,
                       tiles_x, tiles_y, ntiles, err);
  }, cells * 8.0 * (stores + (a.cur ? 1 : 0) + (a.prev ? 1 : 0)));
}

template <class B, int CTAS, bool INST, int ORDER>
cudaError_t adj_t(const BlkAdj& a, int* err, cudaStream_t st) {
  constexpr size_t smem = B::kBytes;
  static OncePerDevice once;
  const cudaError_t ready = once([] {
    return cudaFuncSetAttribute(blk_adj_kernel<B, INST, ORDER, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  });
  if (ready != cudaSuccess) return ready;
  const int planes = INST ? 1 : a.S;
  const float* any = a.cur ? a.cur : a.out_last;  // (a level that is zero is not loaded)
  CUtensorMap cm, pm;
  if (!blk_map(&cm, any, a.nx, a.ny, a.pitch, planes, B::kCols, B::kRows) ||
      !blk_map(&pm, a.prev ? a.prev : any, a.nx, a.ny, a.pitch, planes, B::kCols, B::kRows))
    return cudaErrorNotSupported;
  const int tiles_x = (a.nx + B::kUse - 1) / B::kUse, tiles_y = (a.ny + B::kUseY - 1) / B::kUseY;
  const int ntiles = INST ? a.inst.ntiles : a.S * tiles_x * tiles_y;
  const int all = CTAS * device_info().sms, slots = all < kTiledRowsPerShot ? all : kTiledRowsPerShot;  // a partial row each
  const int grid = ntiles < slots ? ntiles : slots;
  const double cells = INST ? (double)ntiles * B::kUse * B::kUseY : (double)a.S * a.nx * a.ny;
  return tracked_launch(kProfAdjoint, st, [&] {
    launch_step_kernel(blk_adj_kernel<B, INST, ORDER, CTAS>, dim3(grid), dim3(B::kThreads), smem, st, a.chained != 0, a, cm, pm,
                       tiles_x, tiles_y, ntiles, err);
  }, cells * 8.0 * (a.T + (a.T > 1 ? 2 : 1) + (a.cur ? 1 : 0) + (a.prev ? 1 : 0)));
}

// The per-cell modes' adjoint launches.
template <int W, int RW, int CTAS>
cudaError_t adj_d_t(const BlkAdj& a, int* err, cudaStream_t st) {
  using B = BlkTile<W, RW>;
  static OncePerDevice once;
  const cudaError_t ready = once([] {
    return cudaFuncSetAttribute(blk_adj_d_kernel<W, RW, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)B::kBytes);
  });
  if (ready != cudaSuccess) return ready;
  const float* any = a.cur ? a.cur : a.out_last;  // (a level that is zero is not loaded)
  CUtensorMap cm, pm;
  if (!blk_map(&cm, any, a.nx, a.ny, a.pitch, a.S, kBox, B::kRows) ||
      !blk_map(&pm, a.prev ? a.prev : any, a.nx, a.ny, a.pitch, a.S, kBox, B::kRows))
    return cudaErrorNotSupported;
  const int tiles_x = (a.nx + B::kUse - 1) / B::kUse, tiles_y = (a.ny + kBlkCols - 1) / kBlkCols;
  const int ntiles = a.S * tiles_x * tiles_y, slots = CTAS * device_info().sms;
  return tracked_launch(kProfAdjoint, st, [&] {
    launch_step_kernel(blk_adj_d_kernel<W, RW, CTAS>, dim3(ntiles < slots ? ntiles : slots), dim3(32 * W), B::kBytes,
                       st, a.chained != 0, a, cm, pm, tiles_x, tiles_y, ntiles, err);
  }, (double)a.S * a.nx * a.ny * (16.0 * a.T + 32.0 + 4.0));
}

// A run: one CTA per tile, launched cooperatively.
template <class Kernel, class... Args>
cudaError_t launch_run(int cls, Kernel kernel, int ntiles, size_t smem, double bytes, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ntiles);
  cfg.blockDim = dim3(32 * kRunW);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaSuccess;
  const cudaError_t l = tracked_launch(cls, st, [&] { e = cudaLaunchKernelEx(&cfg, kernel, args...); }, bytes);
  return e != cudaSuccess ? e : l;
}

template <int MODE, int RW, int ORDER>
cudaError_t fwd_run(const BlkFwd& a, const FwdRun& r, int* err, cudaStream_t st) {
  using R = RunTile<RW>;
  static OncePerDevice once;
  const cudaError_t ready = once([] {
    return cudaFuncSetAttribute(run_fwd_kernel<MODE, RW, ORDER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)R::kBytes);
  });
  if (ready != cudaSuccess) return ready;
  const int tiles_x = (a.nx + R::kUse - 1) / R::kUse, tiles_y = (a.ny + kBlkCols - 1) / kBlkCols;
  return launch_run(kProfForward, run_fwd_kernel<MODE, RW, ORDER>, a.S * tiles_x * tiles_y, R::kBytes,
                    (double)a.S * a.nx * a.ny * 8.0 * kBlkSteps * r.n, st, a, r, tiles_x, tiles_y, err);
}

template <int RW, int ORDER>
cudaError_t adj_run(const BlkAdj& a, const AdjRun& r, int* err, cudaStream_t st) {
  using R = RunTile<RW>;
  static OncePerDevice once;
  const cudaError_t ready = once([] {
    return cudaFuncSetAttribute(run_adj_kernel<RW, ORDER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)R::kBytes);
  });
  if (ready != cudaSuccess) return ready;
  const int tiles_x = (a.nx + R::kUse - 1) / R::kUse, tiles_y = (a.ny + kBlkCols - 1) / kBlkCols;
  return launch_run(kProfAdjoint, run_adj_kernel<RW, ORDER>, a.S * tiles_x * tiles_y, R::kBytes,
                    (double)a.S * a.nx * a.ny * 8.0 * (kBlkSteps + 2) * r.n, st, a, r, tiles_x, tiles_y, err);
}

template <bool RUN>
cudaError_t adj_f(const BlkAdj& a, const std::conditional_t<RUN, AdjRun, NoRun>& r, int* err, cudaStream_t st) {
  constexpr int W = kRunW, H = W - 2 * kH;
  constexpr size_t smem = (size_t)(2 * 4 + 2) * W * kBox * 4 + 128;
  static OncePerDevice once;
  const cudaError_t ready = once([] {
    return cudaFuncSetAttribute(blk_adj_f_kernel<W, RUN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  });
  if (ready != cudaSuccess) return ready;
  const int tiles_x = (a.nx + H - 1) / H, tiles_y = (a.ny + kBlkCols - 1) / kBlkCols;
  const int ntiles = a.S * tiles_x * tiles_y;
  if constexpr (RUN) {
    return launch_run(kProfAdjoint, blk_adj_f_kernel<W, true>, ntiles, smem,
                      (double)a.S * a.nx * a.ny * (8.0 * (kBlkSteps + 2) * r.n + 72.0), st, a, r, tiles_x, tiles_y,
                      ntiles, err);
  } else {
    return tracked_launch(kProfAdjoint, st, [&] {
      launch_step_kernel(blk_adj_f_kernel<W, false>, dim3(ntiles < device_info().sms ? ntiles : device_info().sms), dim3(32 * W), smem,
                         st, a.chained != 0, a, r, tiles_x, tiles_y, ntiles, err);
    }, (double)a.S * a.nx * a.ny * (8.0 * a.T + 32.0 + 72.0));
  }
}

}  // namespace

// Tile geometries.  kBlkTall: eight warps of six rows, two CTAs per SM (one
// loads its tile while the other computes), 40 of 48 rows stored: the best
// use of the FP32 pipe, for grids of several tiles per SM; kBlkTall5 and
// kBlkTall4, with five and four rows a warp, where these fill their last wave
// of tiles better.  kBlkShort: sixteen warps of two rows, one CTA per SM, 24
// of 32 rows stored, and kBlkFlat: sixteen warps of one row, 8 of 16 stored,
// whose tiles take a half and a quarter as long, for grids that would leave
// SMs idle.
// kBlkRow128 and kBlkRow64: grids of at most 128 or 64 columns, whose rows a
// tile holds whole: the tall tile without halo columns, and with two rows
// side by side in a warp (96 rows, 88 stored).  With 120-column tiles most
// lanes would be idle there, or a second tile hold a few columns: us per
// forward and adjoint step, one-step tiles / 120-column tiles / these: 64 x
// 4000x40 194 / 243 / 131, 64 x 4000x64 217 / 247 / 139, 30 x 3000x124
// 160 / 183 / 113.
BlkShape blk_shape(int geo) {
  switch (geo) {
    case kBlkShort: return {16 * 2 - 2 * kH, kBlkCols, kH};
    case kBlkFlat: return {16 - 2 * kH, kBlkCols, kH};
    case kBlkTall5: return {8 * 5 - 2 * kH, kBlkCols, kH};
    case kBlkTall4: return {8 * 4 - 2 * kH, kBlkCols, kH};
    case kBlkRow128: return {8 * 6 - 2 * kH, 128, 0};
    case kBlkRow64: return {8 * 6 * 2 - 2 * kH, 64, 0};
    default: return {8 * 6 - 2 * kH, kBlkCols, kH};
  }
}

size_t blk_tiles(int geo, int nx, int ny) {
  const BlkShape g = blk_shape(geo);
  return (size_t)((nx + g.rows - 1) / g.rows) * ((ny + g.cols - 1) / g.cols);
}

// The geometry whose waves of tiles take the least time: us per wave on 152
// SMs, mean of a forward and an adjoint launch of four steps (measured at
// one shot of 301^2 and 512^2, three of 501 x 389, eight of 640 x 720; low
// grids: 100 to 500 shots of 1 to 16 rows and 4000 to 8000 columns).  From sizes
// alone, as the workspace layout depends on it.
double blk_cost(int geo, int nx, int ny, int S) {
  const double sms = 152.0, tiles = S * (double)blk_tiles(geo, nx, ny);
  if (blk_shape(geo).hy == 0 && ny > blk_shape(geo).cols) return HUGE_VAL;  // not the whole row
  if (geo == kBlkTall || geo == kBlkRow128 || geo == kBlkRow64) return tiles <= sms ? 21.0 : 20.0 * std::ceil(tiles / (2.0 * sms));
  if (geo == kBlkTall5) return 17.3 * std::ceil(tiles / (2.0 * sms));
  // (a grid lower than the tile leaves warps idle and takes as much less time:
  // 4.3 us a wave at one row, 7.1 at 8, 8.4 at 16)
  if (geo == kBlkTall4)
    return 14.6 * (nx < 24 ? 0.4 + 0.6 * nx / 24.0 : 1.0) * std::ceil(tiles / (2.0 * sms));
  return (geo == kBlkShort ? 9.4 : 5.0) * std::ceil(tiles / sms);
}

int blk_geometry(int mode, int nx, int ny, int S) {
  int best = kBlkTall;
  // (the five- and four-row tiles, and those of whole rows: scalar constants)
  for (int geo : {kBlkShort, kBlkFlat, kBlkTall5, kBlkTall4, kBlkRow128, kBlkRow64})
    if ((mode == kModeScalar || geo < kBlkTall5) && blk_cost(geo, nx, ny, S) < blk_cost(best, nx, ny, S)) best = geo;
  return best;
}

bool blk_available() { return blk_encode_fn() != nullptr; }

cudaError_t launch_inst_table(const InstDesc& d, int4* tiles, int4* box, cudaStream_t st) {
  if (d.count < 1) return cudaSuccess;
  return tracked_launch(kProfOther, st, [&] { inst_table_kernel<<<d.count, 256, 0, st>>>(d, tiles, box); });
}

size_t blk_rec_bytes(size_t ntiles, int S, int nrec) {
  return (ntiles + 2) / 2 * 8 + ntiles * sizeof(int2) + 4 * (size_t)S * nrec * sizeof(int2);
}

cudaError_t launch_rec_tiles(int geo, const int32_t* rec_idx, int S, int nrec, int nx, int ny, const int4* box,
                             size_t ntiles, void* ws, const int2** tile, const int2** ent, float* tr_x, float* tr_y,
                             int nt_out, cudaStream_t st) {
  const BlkShape g = blk_shape(geo);
  int* count = static_cast<int*>(ws);
  int2* tl = reinterpret_cast<int2*>(static_cast<char*>(ws) + (ntiles + 2) / 2 * 8);
  int2* en = tl + ntiles;
  *tile = tl;
  *ent = en;
  cudaError_t e = cudaMemsetAsync(count, 0, (ntiles + 1) * sizeof(int), st);
  if (e != cudaSuccess) return e;
  const int n = S * nrec, tx = (nx + g.rows - 1) / g.rows, ty = (ny + g.cols - 1) / g.cols;
  const int nt = (int)ntiles;
  e = tracked_launch(kProfOther, st, [&] {
    rec_tiles_kernel<false><<<(n + 255) / 256, 256, 0, st>>>(rec_idx, S, nrec, nx, ny, g, tx, ty, box, count, tl, en, tr_x,
                                                             tr_y, nt_out);
  });
  if (e != cudaSuccess) return e;
  e = tracked_launch(kProfOther, st, [&] { rec_base_kernel<<<(nt + 255) / 256, 256, 0, st>>>(count, nt, tl); });
  if (e != cudaSuccess) return e;
  return tracked_launch(kProfOther, st, [&] {
    rec_tiles_kernel<true><<<(n + 255) / 256, 256, 0, st>>>(rec_idx, S, nrec, nx, ny, g, tx, ty, box, count, tl, en, tr_x,
                                                            tr_y, nt_out);
  });
}

namespace {
template <int MODE, int ORDER>
cudaError_t fwd_geo(const BlkFwd& a, int* err, cudaStream_t st) {
  if (a.geo == kBlkFlat) return fwd_t<MODE, BlkTile<16, 1>, 1, false, ORDER>(a, err, st);
  if (a.geo == kBlkShort) return fwd_t<MODE, BlkTile<16, 2>, 1, false, ORDER>(a, err, st);
  if constexpr (MODE == kModeScalar) {
    if (a.geo == kBlkTall5) return fwd_t<MODE, BlkTile<8, 5>, 2, false, ORDER>(a, err, st);
    if (a.geo == kBlkTall4) return fwd_t<MODE, BlkTile<8, 4>, 2, false, ORDER>(a, err, st);
    if (a.geo == kBlkRow128) return fwd_t<MODE, BlkTile<8, 6, 32, true>, 2, false, ORDER>(a, err, st);
    if (a.geo == kBlkRow64) return fwd_t<MODE, BlkTile<8, 6, 16, true>, 2, false, ORDER>(a, err, st);
  }
  return fwd_t<MODE, BlkTile<8, 6>, 2, false, ORDER>(a, err, st);
}

template <int ORDER>
cudaError_t adj_geo(const BlkAdj& a, int* err, cudaStream_t st) {
  if (a.geo == kBlkFlat) return adj_t<BlkTile<16, 1>, 1, false, ORDER>(a, err, st);
  if (a.geo == kBlkShort) return adj_t<BlkTile<16, 2>, 1, false, ORDER>(a, err, st);
  if (a.geo == kBlkTall5) return adj_t<BlkTile<8, 5>, 2, false, ORDER>(a, err, st);
  if (a.geo == kBlkTall4) return adj_t<BlkTile<8, 4>, 2, false, ORDER>(a, err, st);
  if (a.geo == kBlkRow128) return adj_t<BlkTile<8, 6, 32, true>, 2, false, ORDER>(a, err, st);
  if (a.geo == kBlkRow64) return adj_t<BlkTile<8, 6, 16, true>, 2, false, ORDER>(a, err, st);
  return adj_t<BlkTile<8, 6>, 2, false, ORDER>(a, err, st);
}
}  // namespace

cudaError_t launch_blk_fwd(int mode, const BlkFwd& a, int* err, cudaStream_t st) {
  if (a.inst.tiles != nullptr)
    return a.geo == kBlkRow64 ? fwd_t<kModeScalar, BlkTile<8, 6, 16, true>, 2, true, kOrderTiled>(a, err, st)
                              : fwd_t<kModeScalar, BlkTile<8, 6>, 2, true, kOrderTiled>(a, err, st);
  if (mode == kModeFields) return fwd_t<kModeFields, BlkTile<16, 1>, 1, false, kOrderFields>(a, err, st);
  if (mode == kModeDField) return fwd_geo<kModeDField, kOrderPlain>(a, err, st);
  return a.plain_order ? fwd_geo<kModeScalar, kOrderPlain>(a, err, st) : fwd_geo<kModeScalar, kOrderTiled>(a, err, st);
}

cudaError_t launch_blk_adj(int mode, const BlkAdj& a, int* err, cudaStream_t st) {
  if (mode == kModeFields) return adj_f<false>(a, NoRun{}, err, st);
  if (mode == kModeDField) {
    if (a.geo == kBlkFlat) return adj_d_t<16, 1, 1>(a, err, st);
    if (a.geo == kBlkShort) return adj_d_t<16, 2, 1>(a, err, st);
    return adj_d_t<8, 6, 2>(a, err, st);
  }
  if (a.inst.tiles != nullptr)
    return a.geo == kBlkRow64 ? adj_t<BlkTile<8, 6, 16, true>, 2, true, kOrderTiled>(a, err, st)
                              : adj_t<BlkTile<8, 6>, 2, true, kOrderTiled>(a, err, st);
  return a.plain_order ? adj_geo<kOrderPlain>(a, err, st) : adj_geo<kOrderTiled>(a, err, st);
}

// Runs: the tiles of a flat or short geometry that are resident at the same
// time, one per SM, scalar constants in the plain kernels' order and constant
// planes.
bool blk_run_fits(int mode, int geo, int nx, int ny, int S) {
  if (mode == kModeDField || (geo != kBlkFlat && geo != kBlkShort)) return false;
  const DeviceInfo d = device_info();
  return d.cooperative && S * blk_tiles(geo, nx, ny) <= (size_t)d.sms;
}

cudaError_t launch_blk_fwd_run(int mode, const BlkFwd& a, const FwdRun& r, int* err, cudaStream_t st) {
  if (mode == kModeFields) return fwd_run<kModeFields, 1, kOrderFields>(a, r, err, st);
  return a.geo == kBlkFlat ? fwd_run<kModeScalar, 1, kOrderPlain>(a, r, err, st)
                           : fwd_run<kModeScalar, 2, kOrderPlain>(a, r, err, st);
}

cudaError_t launch_blk_adj_run(int mode, const BlkAdj& a, const AdjRun& r, int* err, cudaStream_t st) {
  if (mode == kModeFields) return adj_f<true>(a, r, err, st);
  return a.geo == kBlkFlat ? adj_run<1, kOrderPlain>(a, r, err, st) : adj_run<2, kOrderPlain>(a, r, err, st);
}

}  // namespace ernn
