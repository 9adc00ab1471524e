// Per-step kernels for degradation maps on large grids (sm_103a), TMA-pipelined.
//
// One launch per time step; each CTA is persistent over a list of 64 (y) x 32
// (x) tiles of the step and streams them through a two-stage shared-memory
// pipeline: while a tile is computed, the tensor-memory-accelerator loads of
// the next tile are in flight (cp.async.bulk.tensor, completion on an
// mbarrier per stage).  (The other modes, and smaller grids of this one, take
// several steps per launch: ernn_block.cu.)
//
// The halo box of a tile is 72 x 34 cells: rows x0-1 .. x0+32 and columns
// y0-4 .. y0+67 (the innermost coordinate must be a multiple of four floats,
// so the box reaches four columns to the left where one is needed).  Cells
// outside the grid are filled with zeros by the copy engine: that is the zero
// ghost ring of the scheme, with no predicated loads.  ny % 4 == 0.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <mutex>

#include "ernn_launch.h"
#include "ernn_tile.cuh"
#include "ernn_tma.h"

namespace ernn {

namespace {

constexpr int kTY = 64;                    // tile columns (y); rows per kernel layout
constexpr int kBW = kTY + 8;               // halo box width: tile + 4 columns each side
constexpr int kThreads = 256;              // 16 column quads x 16 rows


// End of a warp's reads of stage k & 1: the last of the CTA's warps to get
// there starts the loads of tile k + 2 into it, so no warp waits on the
// others between tiles.  The values read from the stage are all consumed
// (in registers) before a lane arrives.
template <typename F>
__device__ __forceinline__ void release_stage(int* done, int stage, F&& refill) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
    const int old = atomicAdd(&done[stage], 1);
    if (old % (kThreads / 32) == kThreads / 32 - 1) refill();
  }
}
template <typename F>
__device__ __forceinline__ void release(int* done, int k, F&& refill) {
  release_stage(done, k & 1, refill);
}


// window [j-1 .. j+4] of halo-box row r (box column of cell column j is j + 4)
__device__ __forceinline__ void win(const float* __restrict__ box, int r, int j, float w[6]) {
  const float* p = box + r * kBW + j + 4;
  const float4 m = *reinterpret_cast<const float4*>(p);
  w[0] = p[-1];
  w[1] = m.x;
  w[2] = m.y;
  w[3] = m.z;
  w[4] = m.w;
  w[5] = p[4];
}

struct Sums4 {
  float cx[4], cy[4], xx_x[4], yy_x[4], xy_x[4], xx_y[4], yy_y[4], xy_y[4];
};

// Second differences of one component at the four cells of a window row
// (cell q at window column q + 1):
//   xx = (u[0][k] + u[2][k]) - 2 u[1][k],  yy = (u[1][k-1] + u[1][k+1]) - 2 u[1][k],
//   xy = (u[2][k+1] + u[0][k-1]) - (u[2][k-1] + u[0][k+1]).
__device__ __forceinline__ void comp_sums(const float u[3][6], float xx[4], float yy[4], float xy[4]) {
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const int k = 2 * p + 1;
    const float2 m0 = make_float2(u[0][k], u[0][k + 1]);
    const float2 m1 = make_float2(u[1][k], u[1][k + 1]);
    const float2 m2 = make_float2(u[2][k], u[2][k + 1]);
    put(xx, p, fma2(dup2(-2.f), m1, __fadd2_rn(m0, m2)));
    put(yy, p, fma2(dup2(-2.f), m1, make_float2(u[1][k - 1] + u[1][k + 1], u[1][k] + u[1][k + 2])));
    const float2 a = make_float2(u[2][k + 1] + u[0][k - 1], u[2][k + 2] + u[0][k]);
    const float2 b = make_float2(u[2][k - 1] + u[0][k + 1], u[2][k] + u[0][k + 2]);
    put(xy, p, __fadd2_rn(a, neg2(b)));
  }
}

__device__ __forceinline__ void sums4(const float ux[3][6], const float uy[3][6], Sums4& s) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    s.cx[q] = ux[1][q + 1];
    s.cy[q] = uy[1][q + 1];
  }
  comp_sums(ux, s.xx_x, s.yy_x, s.xy_x);
  comp_sums(uy, s.xx_y, s.yy_y, s.xy_y);
}

__device__ __forceinline__ void apply(const Coefs& k, const Sums4& s, int q, float& lx, float& ly) {
  lx = k.k11 * s.xx_x[q] + k.k66 * s.yy_x[q] + k.kq12 * s.xy_y[q] + k.k16h * s.xy_x[q] +
       k.k16 * s.xx_y[q] + k.k26 * s.yy_y[q];
  ly = k.k66 * s.xx_y[q] + k.k22 * s.yy_y[q] + k.kq12 * s.xy_x[q] + k.k16 * s.xx_x[q] +
       k.k26 * s.yy_x[q] + k.k26h * s.xy_y[q];
}

__device__ __forceinline__ void shift(float u[3][6]) {
#pragma unroll
  for (int k = 0; k < 6; ++k) { u[0][k] = u[1][k]; u[1][k] = u[2][k]; }
}

__device__ __forceinline__ float g4(const float4& v, int q) {
  return q == 0 ? v.x : q == 1 ? v.y : q == 2 ? v.z : v.w;
}

// (L u) of cells 2p and 2p+1: the terms of apply() in the same order.
__device__ __forceinline__ void apply2(const Coefs& k, const Sums4& s, int p, float2& lx, float2& ly) {
  lx = __fmul2_rn(dup2(k.k11), pair(s.xx_x, p));
  lx = fma2(dup2(k.k66), pair(s.yy_x, p), lx);
  lx = fma2(dup2(k.kq12), pair(s.xy_y, p), lx);
  lx = fma2(dup2(k.k16h), pair(s.xy_x, p), lx);
  lx = fma2(dup2(k.k16), pair(s.xx_y, p), lx);
  lx = fma2(dup2(k.k26), pair(s.yy_y, p), lx);
  ly = __fmul2_rn(dup2(k.k66), pair(s.xx_y, p));
  ly = fma2(dup2(k.k22), pair(s.yy_y, p), ly);
  ly = fma2(dup2(k.kq12), pair(s.xy_x, p), ly);
  ly = fma2(dup2(k.k16), pair(s.xx_x, p), ly);
  ly = fma2(dup2(k.k26), pair(s.yy_x, p), ly);
  ly = fma2(dup2(k.k26h), pair(s.xy_y, p), ly);
}

// The forward update in two parts, so that the load joins the operator sum
// before the update, as in the reference's (A u + f) / rho: oper4 writes the
// operator terms w (L u) of a quad into vx, vy, the
// caller adds the load there, and update4 turns them into v = (2 c - p) +
// (w (L u) + f), one rounding of the increment into 2 c - p.  (Added after
// the update instead, the forward's rounding near the source projects onto
// the gradient: ten times the FP32 reference's gradient error close to
// convergence.)
__device__ __forceinline__ void oper4(const Coefs& k, const Sums4& s, const float4& w, float vx[4], float vy[4]) {
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    float2 lx, ly;
    apply2(k, s, p, lx, ly);
    lx = __fmul2_rn(lx, pair4(w, p));
    ly = __fmul2_rn(ly, pair4(w, p));
    vx[2 * p] = lx.x;
    vx[2 * p + 1] = lx.y;
    vy[2 * p] = ly.x;
    vy[2 * p + 1] = ly.y;
  }
}
__device__ __forceinline__ void update4(const float cx[4], const float cy[4], const float4& pvx, const float4& pvy,
                                        float vx[4], float vy[4]) {
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const float2 px = pair4(pvx, p), py = pair4(pvy, p);
    const float2 ax = __fadd2_rn(fma2(dup2(2.f), pair(cx, p), neg2(px)), make_float2(vx[2 * p], vx[2 * p + 1]));
    const float2 ay = __fadd2_rn(fma2(dup2(2.f), pair(cy, p), neg2(py)), make_float2(vy[2 * p], vy[2 * p + 1]));
    vx[2 * p] = ax.x;
    vx[2 * p + 1] = ax.y;
    vy[2 * p] = ay.x;
    vy[2 * p + 1] = ay.y;
  }
}

// Leapfrog update of a quad without a load: v = (2 c - p) + L u (2 c is
// exact, so 2 c - p is one rounding either way).
__device__ __forceinline__ void leap4(const Coefs& k, const Sums4& s, const float cx[4], const float cy[4],
                                      const float4& pvx, const float4& pvy, float vx[4], float vy[4]) {
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    float2 lx, ly;
    apply2(k, s, p, lx, ly);
    const float2 px = pair4(pvx, p), py = pair4(pvy, p);
    const float2 ax = __fadd2_rn(fma2(dup2(2.f), pair(cx, p), neg2(px)), lx);
    const float2 ay = __fadd2_rn(fma2(dup2(2.f), pair(cy, p), neg2(py)), ly);
    vx[2 * p] = ax.x;
    vx[2 * p + 1] = ax.y;
    vy[2 * p] = ay.x;
    vy[2 * p + 1] = ay.y;
  }
}

// A tile: its shot and origin.
struct TileId {
  int shot, x0, y0;
};

// The tiles t = first, first + stride, ... of a CTA, walked in (shot, row
// block, column block) coordinates: the stride is split once into the same
// mixed radix, so a step is an addition with two carries, not a division.
template <int TR>
struct TileWalk {
  int shot, xt, yt, ds, dx, dy, tiles_x, tiles_y;
  __device__ __forceinline__ void init(int first, int stride, int tx, int ty) {
    tiles_x = tx;
    tiles_y = ty;
    const int per = tx * ty;
    shot = first / per;
    int r = first - shot * per;
    xt = r / ty;
    yt = r - xt * ty;
    ds = stride / per;
    r = stride - ds * per;
    dx = r / ty;
    dy = r - dx * ty;
  }
  __device__ __forceinline__ TileId id() const { return TileId{shot, xt * TR, yt * kTY}; }
  __device__ __forceinline__ void next() {
    yt += dy;
    if (yt >= tiles_y) { yt -= tiles_y; ++xt; }
    xt += dx;
    if (xt >= tiles_x) { xt -= tiles_x; ++shot; }
    shot += ds;
  }
};

template <int TR>  // tile rows
__device__ __forceinline__ TileId tile_of(int t, int tiles_x, int tiles_y) {
  const int per_shot = tiles_x * tiles_y;
  TileId id;
  id.shot = t / per_shot;
  const int r = t - id.shot * per_shot;
  id.x0 = (r / tiles_y) * TR;
  id.y0 = (r % tiles_y) * kTY;
  return id;
}

// ----------------------------------------------------------------- forward
// Stage: halo box of u^i, own box of u^{i-1}.  The weights 1 - D are read
// straight from global memory (one plane shared by every shot, L2 resident).
// 64 x 32 tiles, two rows per thread, three CTAs per SM (64 x 16 tiles at
// four measured slower: 8 x 512^2, 81.3 against 75.6 ms per iteration).
struct FwdLayout {
  static constexpr int kTR = 32;         // tile rows
  static constexpr int kRT = kTR / 16;   // rows per thread
  static constexpr int kBHa = kTR + 2;   // halo box rows
  static constexpr int kHalo = 2 * kBHa * kBW;
  static constexpr int kOwn = 2 * kTR * kTY;
  static constexpr int kStage = (kHalo + kOwn + 31) / 32 * 32;  // 128-byte multiple
  static constexpr int kCtasPerSm = 3;
};

__global__ void __launch_bounds__(kThreads, FwdLayout::kCtasPerSm)
    tma_fwd_kernel(const FwdStep a, const __grid_constant__ CUtensorMap cur_map,
                   const __grid_constant__ CUtensorMap prev_map, int tiles_x, int tiles_y, int has_prev,
                   int* err) {
  extern __shared__ float sm_raw[];
  float* sm = aligned128(sm_raw);
  using F = FwdLayout;
  constexpr int kStage = F::kStage;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + 2 * kStage);
  const int tid = threadIdx.x;
  const int nx = a.nx, ny = a.ny;
  const size_t N = (size_t)nx * ny;
  const int ntiles = a.S * tiles_x * tiles_y;
  const uint32_t bytes = (uint32_t)(F::kHalo + (has_prev ? F::kOwn : 0)) * 4u;
  grid_dep_trigger();
  __shared__ int done[2];
  __shared__ PipeGuard guard;
  if (tid == 0) {
    prefetch_map(&cur_map);
    prefetch_map(&prev_map);
    bar_init(&bar[0]);
    bar_init(&bar[1]);
    done[0] = done[1] = 0;
    pipe_init(&guard);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  grid_dep_wait();  // the state of the previous step is complete from here on

  // receiver gather of the input state u^i, spread over the grid
  if (a.gframe >= 0) {
    for (int e = blockIdx.x * kThreads + tid; e < a.S * a.nrec; e += gridDim.x * kThreads) {
      const int s = e / a.nrec, r = e - s * a.nrec;
      const int32_t idx = a.rec_idx[e];
      const size_t o = ((size_t)s * a.nt_out + a.gframe) * a.nrec + r;
      const size_t plane = (size_t)s * 2 * N;
      const bool ok = a.cur != nullptr && idx >= 0 && (size_t)idx < N;
      a.tr_x[o] = ok ? a.cur[plane + idx] : 0.f;
      a.tr_y[o] = ok ? a.cur[plane + N + idx] : 0.f;
    }
  }
  __syncthreads();
  const bool has_src = a.bx > 0 && a.by > 0;
  auto issue = [&](int k) {  // loads of this CTA's k-th tile into stage k & 1
    const int t = blockIdx.x + k * gridDim.x;
    if (t >= ntiles || pipe_failed(&guard)) return;
    pipe_issued(&guard, k);
    const TileId id = tile_of<F::kTR>(t, tiles_x, tiles_y);
    float* st = sm + (k & 1) * kStage;
    fence_async();
    bar_expect(&bar[k & 1], bytes);
    tma_load3(st, &cur_map, id.y0 - 4, id.x0 - 1, 2 * id.shot, &bar[k & 1]);
    if (has_prev) tma_load3(st + F::kHalo, &prev_map, id.y0, id.x0, 2 * id.shot, &bar[k & 1]);
  };
  if (tid == 0) {
    issue(0);
    issue(1);
  }
  const int qc = tid & 15, rg = tid >> 4;
  const int j = 4 * qc;
  const Coefs ks = coefs(a.coef);
  TileWalk<F::kTR> walk;
  walk.init(blockIdx.x, gridDim.x, tiles_x, tiles_y);
  for (int k = 0;; ++k) {
    const int t = blockIdx.x + k * gridDim.x;
    if (t >= ntiles) break;
    const TileId id = walk.id();
    walk.next();
    // per-tile scalars, loaded before the wait
    const float amp = a.src_signal[(size_t)id.shot * a.nt + a.i] * a.coef->kappa;
    const int ox = has_src ? a.src_origin[2 * id.shot] : 0, oy = has_src ? a.src_origin[2 * id.shot + 1] : 0;
    const int gj = id.y0 + j;
    const int r0 = F::kRT * rg;  // tile row r0 + q2 -> box row r0 + q2 + 1
    float4 w4[F::kRT];
#pragma unroll
    for (int q2 = 0; q2 < F::kRT; ++q2) {  // issued before the wait: overlaps the tile's loads
      const int gi = id.x0 + r0 + q2;
      w4[q2] = (gi < nx && gj < ny)
                   ? one_minus(__ldg(reinterpret_cast<const float4*>(a.field + (size_t)gi * ny + gj)))
                   : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    bar_wait_ok(&bar[k & 1], (uint32_t)(k >> 1) & 1u, err, &guard);
    const float* hb = sm + (k & 1) * kStage;
    const float* pb = hb + F::kHalo;
    float* out = a.out + (size_t)id.shot * 2 * N;
    float wx[3][6], wy[3][6];
    win(hb, r0, j, wx[0]);
    win(hb + F::kBHa * kBW, r0, j, wy[0]);
    win(hb, r0 + 1, j, wx[1]);
    win(hb + F::kBHa * kBW, r0 + 1, j, wy[1]);
#pragma unroll
    for (int q2 = 0; q2 < F::kRT; ++q2) {
      const int r = r0 + q2;
      win(hb, r + 2, j, wx[2]);
      win(hb + F::kBHa * kBW, r + 2, j, wy[2]);
      Sums4 st;
      sums4(wx, wy, st);
      const int gi = id.x0 + r;
      // computed for every cell of the tile (the boxes are zero outside the
      // grid); only the stores are guarded
      float4 pvx = make_float4(0.f, 0.f, 0.f, 0.f), pvy = pvx;
      if (has_prev) {
        pvx = *reinterpret_cast<const float4*>(pb + r * kTY + j);
        pvy = *reinterpret_cast<const float4*>(pb + F::kTR * kTY + r * kTY + j);
      }
      float vx[4], vy[4];
      // source box: rows and columns of this thread's 4 cells inside it
      const int sa = gi - ox;
      oper4(ks, st, w4[q2], vx, vy);
      if (has_src && (unsigned)sa < (unsigned)a.bx && gj + 3 >= oy && gj < oy + a.by) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int sb = gj + q - oy;
          if ((unsigned)sb < (unsigned)a.by) {
            const float f = a.src_map[((size_t)id.shot * a.bx + sa) * a.by + sb];  // L + amp f, one rounding
            if (a.src_comp == 0) vx[q] = fmaf(amp, f, vx[q]); else vy[q] = fmaf(amp, f, vy[q]);
          }
        }
      }
      update4(st.cx, st.cy, pvx, pvy, vx, vy);
      if (gi < nx && gj < ny) {
        const float4 nvx = make_float4(vx[0], vx[1], vx[2], vx[3]);
        const float4 nvy = make_float4(vy[0], vy[1], vy[2], vy[3]);
        const size_t o = (size_t)gi * ny + gj;
        *reinterpret_cast<float4*>(out + o) = nvx;
        *reinterpret_cast<float4*>(out + N + o) = nvy;
        if (a.copy0) {
          *reinterpret_cast<float4*>(a.copy0 + (size_t)id.shot * 2 * N + o) = nvx;
          *reinterpret_cast<float4*>(a.copy0 + (size_t)id.shot * 2 * N + N + o) = nvy;
        }
        if (a.copy1) {
          *reinterpret_cast<float4*>(a.copy1 + (size_t)id.shot * 2 * N + o) = nvx;
          *reinterpret_cast<float4*>(a.copy1 + (size_t)id.shot * 2 * N + N + o) = nvy;
        }
        if (a.frame >= 0) {
          const size_t ho = ((size_t)id.shot * a.nt_out + a.frame) * N + o;
          *reinterpret_cast<float4*>(a.hist_x + ho) = nvx;
          *reinterpret_cast<float4*>(a.hist_y + ho) = nvy;
        }
      }
      shift(wx);
      shift(wy);
    }
    release(done, k, [&] { issue(k + 2); });
  }
  if (tid == 0 && pipe_failed(&guard)) pipe_drain(bar, 2, &guard);
}

// ----------------------------------------------------------------- adjoint
// Stage: halo boxes of lam^{m+1}, u^m and D (the imaging is per cell, so u's
// stencils are needed); lam^{m+2} is read into registers before the wait
// (keeps two CTAs per SM within shared memory).  Two rows per thread: with
// one row the three halo windows per output row (lam, u, D) cost more than a
// third CTA gains (24.4 against 21.5 us per step of 8 x 512^2).
struct AdjLayout {
  static constexpr int kTR = 32;                               // tile rows
  static constexpr int kRT = kTR / 16;                         // rows per thread
  static constexpr int kBHa = kTR + 2;                         // halo box rows
  static constexpr int kHalo = 2 * kBHa * kBW;
  static constexpr int kU = kHalo;
  static constexpr int kD = kU + kHalo;
  static constexpr int kStage = (kD + kBHa * kBW + 31) / 32 * 32;  // 128-byte multiple
  static constexpr int kStages = 2;
  static constexpr int kCtasPerSm = 2;
};

__global__ void __launch_bounds__(kThreads, AdjLayout::kCtasPerSm)
    tma_adj_kernel(const AdjStep a, const __grid_constant__ CUtensorMap cur_map,
                   const __grid_constant__ CUtensorMap u_map, const __grid_constant__ CUtensorMap d_map, int tiles_x,
                   int tiles_y, int has_u, int* err) {
  using L = AdjLayout;
  extern __shared__ float sm_raw[];
  float* sm = aligned128(sm_raw);
  constexpr int NS = L::kStages;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + NS * L::kStage);
  const int tid = threadIdx.x;
  const int nx = a.nx, ny = a.ny;
  const size_t N = (size_t)nx * ny;
  const int ntiles = a.S * tiles_x * tiles_y;
  const uint32_t bytes = (uint32_t)(L::kHalo + L::kBHa * kBW + (has_u ? L::kHalo : 0)) * 4u;
  grid_dep_trigger();
  __shared__ int done[NS];
  __shared__ PipeGuard guard;
  if (tid == 0) {
    prefetch_map(&cur_map);
    prefetch_map(&d_map);
    if (has_u) prefetch_map(&u_map);
    for (int q = 0; q < NS; ++q) {
      bar_init(&bar[q]);
      done[q] = 0;
    }
    pipe_init(&guard);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  grid_dep_wait();  // the state of the previous step is complete from here on
  const float gs = a.coef->gscale;
  auto issue = [&](int k) {  // loads of this CTA's k-th tile
    const int t = blockIdx.x + k * gridDim.x;
    if (t >= ntiles || pipe_failed(&guard)) return;
    pipe_issued(&guard, k);
    const TileId id = tile_of<L::kTR>(t, tiles_x, tiles_y);
    const int sg = k % NS;
    float* st = sm + sg * L::kStage;
    fence_async();
    bar_expect(&bar[sg], bytes);
    tma_load3(st, &cur_map, id.y0 - 4, id.x0 - 1, 2 * id.shot, &bar[sg]);
    tma_load2(st + L::kD, &d_map, id.y0 - 4, id.x0 - 1, &bar[sg]);
    if (has_u) tma_load3(st + L::kU, &u_map, id.y0 - 4, id.x0 - 1, 2 * id.shot, &bar[sg]);
  };
  if (tid == 0)
    for (int q = 0; q < NS; ++q) issue(q);
  const int qc = tid & 15, rg = tid >> 4;
  const int j = 4 * qc;
  const bool inject = a.frame >= 0 && a.record == kRecordReceivers;
  const Coefs ks = coefs(a.coef);
  TileWalk<L::kTR> walk;
  walk.init(blockIdx.x, gridDim.x, tiles_x, tiles_y);
  for (int k = 0;; ++k) {
    const int t = blockIdx.x + k * gridDim.x;
    if (t >= ntiles) break;
    const TileId id = walk.id();
    walk.next();
    const int gj = id.y0 + j;
    const int r0 = L::kRT * rg;
    // receivers in this tile (uniform over the CTA): the injection and its
    // barrier only run where the per-call table says there are some
    const bool tile_inject = inject && (a.tile_flags == nullptr || a.tile_flags[t] != 0);
    float4 pv[L::kRT][2];  // lam^{m+2} of the thread's rows (x, y)
#pragma unroll
    for (int q2 = 0; q2 < L::kRT; ++q2) {
      const int gi = id.x0 + r0 + q2;
      const size_t o = (size_t)id.shot * 2 * N + (size_t)gi * ny + gj;
      const bool in = gi < nx && gj < ny;
      pv[q2][0] = in ? *reinterpret_cast<const float4*>(a.prev + o) : make_float4(0.f, 0.f, 0.f, 0.f);
      pv[q2][1] = in ? *reinterpret_cast<const float4*>(a.prev + N + o) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const int stage = k % NS;
    bar_wait_ok(&bar[stage], (uint32_t)(k / NS) & 1u, err, &guard);
    const float* hb = sm + stage * L::kStage;
    const float* ub = hb + L::kU;
    const float* db = hb + L::kD;
    float* out = a.out + (size_t)id.shot * 2 * N;
    // lam windows for the stencils, weighted by 1 - D (A^T lam =
    // A0((1 - D) lam)); the centre value itself stays unweighted
    auto lam_win = [&](int r, float wx_[6], float wy_[6]) {
      win(hb, r, j, wx_);
      win(hb + L::kBHa * kBW, r, j, wy_);
      float dw[6];
      win(db, r, j, dw);
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        const float w = 1.f - dw[c];
        wx_[c] = w * wx_[c];
        wy_[c] = w * wy_[c];
      }
    };
    float wx[3][6], wy[3][6], vx_[3][6], vy_[3][6];
    lam_win(r0, wx[0], wy[0]);
    lam_win(r0 + 1, wx[1], wy[1]);
    if (has_u) {
      win(ub, r0, j, vx_[0]);
      win(ub + L::kBHa * kBW, r0, j, vy_[0]);
      win(ub, r0 + 1, j, vx_[1]);
      win(ub + L::kBHa * kBW, r0 + 1, j, vy_[1]);
    }
#pragma unroll
    for (int q2 = 0; q2 < L::kRT; ++q2) {
      const int r = r0 + q2;
      lam_win(r + 2, wx[2], wy[2]);
      Sums4 st;
      sums4(wx, wy, st);
      const int gi = id.x0 + r;
      const bool in = gi < nx && gj < ny;  // (ny % 4 == 0: a quad is in or out)
      // unweighted lam^{m+1} at the 4 cells
      float c1x[4], c1y[4];
      const float4 cx4 = *reinterpret_cast<const float4*>(hb + (r + 1) * kBW + j + 4);
      const float4 cy4 = *reinterpret_cast<const float4*>(hb + L::kBHa * kBW + (r + 1) * kBW + j + 4);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        c1x[q] = g4(cx4, q);
        c1y[q] = g4(cy4, q);
      }
      const size_t o = (size_t)gi * ny + gj;
      float vx[4], vy[4];
      leap4(ks, st, c1x, c1y, pv[q2][0], pv[q2][1], vx, vy);
      if (in) {
        if (a.frame >= 0 && a.record == kRecordFields) {
          const size_t go = ((size_t)id.shot * a.nt_out + a.frame) * N + o;
          const float4 gx = *reinterpret_cast<const float4*>(a.g_x + go);
          const float4 gy = *reinterpret_cast<const float4*>(a.g_y + go);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            vx[q] += gs * g4(gx, q);
            vy[q] += gs * g4(gy, q);
          }
        }
        *reinterpret_cast<float4*>(out + o) = make_float4(vx[0], vx[1], vx[2], vx[3]);
        *reinterpret_cast<float4*>(out + N + o) = make_float4(vy[0], vy[1], vy[2], vy[3]);
      }
      if (has_u) {
        win(ub, r + 2, j, vx_[2]);
        win(ub + L::kBHa * kBW, r + 2, j, vy_[2]);
        Sums4 su;
        sums4(vx_, vy_, su);
        if (in) {
          float* ga = a.gacc + (size_t)id.shot * N + o;
          float4 g = *reinterpret_cast<const float4*>(ga);
          float gv[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float Lx, Ly;
            apply(ks, su, q, Lx, Ly);
            gv[q] += c1x[q] * Lx + c1y[q] * Ly;
          }
          *reinterpret_cast<float4*>(ga) = make_float4(gv[0], gv[1], gv[2], gv[3]);
        }
        shift(vx_);
        shift(vy_);
      }
      shift(wx);
      shift(wy);
    }
    if (tile_inject) {
      // adjoint source at receiver cells, added to the stored lam^m (several
      // receivers may share a cell); the block's own stores are visible
      // after the barrier
      __syncthreads();
      for (int rr = tid; rr < a.nrec; rr += kThreads) {
        const int32_t idx = a.rec_idx[(size_t)id.shot * a.nrec + rr];
        if (idx < 0 || (size_t)idx >= N) continue;
        const int gi = idx / ny, gjj = idx - gi * ny;
        if (gi >= id.x0 && gi < id.x0 + L::kTR && gjj >= id.y0 && gjj < id.y0 + kTY) {
          const size_t go = ((size_t)id.shot * a.nt_out + a.frame) * a.nrec + rr;
          atomicAdd(out + idx, gs * a.g_x[go]);
          atomicAdd(out + N + idx, gs * a.g_y[go]);
        }
      }
    }
    release_stage(done, stage, [&] { issue(k + NS); });
  }
  if (tid == 0 && pipe_failed(&guard)) pipe_drain(bar, NS, &guard);
}

// ------------------------------------------------------ wait self-test
// One thread waits on an mbarrier that nothing arrives at (no copy is in
// flight towards this CTA), through the same bounded wait as the tile loop.
__global__ void wait_selftest_kernel(int* status) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    bar_init(&bar);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    bar_wait(&bar, 0u, status);
  }
}

__device__ int g_selftest_status;

// Receiver table of the tiled adjoint: flags[(shot, tile)] = 1 where the
// shot has a receiver in the tile.
__global__ void tile_flags_kernel(const int32_t* __restrict__ rec_idx, int S, int nrec, int nx, int ny,
                                  int tile_rows, int tiles_x, int tiles_y, uint8_t* __restrict__ flags) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= S * nrec) return;
  const int s = e / nrec;
  const int32_t idx = rec_idx[e];
  if (idx < 0 || (int64_t)idx >= (int64_t)nx * ny) return;  // ignored, as in the kernels
  const int gi = idx / ny, gj = idx - gi * ny;
  flags[(size_t)s * tiles_x * tiles_y + (size_t)(gi / tile_rows) * tiles_y + gj / kTY] = 1;
}

// ----------------------------------------------------------------- host
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
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

// Tensor map over S shots of [comp][nx][ny] floats: dims (ny, nx, 2 S).
bool make_map(CUtensorMap* m, const float* base, int nx, int ny, int S, int bw, int bh) {
  auto fn = encode_fn();
  if (fn == nullptr || base == nullptr) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)ny, (cuuint64_t)nx, (cuuint64_t)2 * S};
  const cuuint64_t strides[2] = {(cuuint64_t)ny * 4, (cuuint64_t)nx * ny * 4};
  const cuuint32_t box[3] = {(cuuint32_t)bw, (cuuint32_t)bh, 2};
  const cuuint32_t estr[3] = {1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tensor map over the degradation plane [nx][ny]: dims (ny, nx).
bool make_map2(CUtensorMap* m, const float* base, int nx, int ny, int bw, int bh) {
  auto fn = encode_fn();
  if (fn == nullptr || base == nullptr) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)ny, (cuuint64_t)nx};
  const cuuint64_t strides[1] = {(cuuint64_t)ny * 4};
  const cuuint32_t box[2] = {(cuuint32_t)bw, (cuuint32_t)bh};
  const cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr size_t kFwdSmem = 2 * (size_t)FwdLayout::kStage * 4 + 16 + 128;
constexpr size_t kAdjSmem = (size_t)AdjLayout::kStages * AdjLayout::kStage * 4 + 8 * AdjLayout::kStages + 128;

cudaError_t set_smem() {
  static OncePerDevice once;
  return once([] {
    const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
    const cudaError_t e = cudaFuncSetAttribute(tma_fwd_kernel, at, (int)kFwdSmem);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(tma_adj_kernel, at, (int)kAdjSmem);
  });
}

}  // namespace

cudaError_t wait_selftest(int* status_host, cudaStream_t st) {
  const int zero = 0;
  cudaError_t e = cudaMemcpyToSymbolAsync(g_selftest_status, &zero, sizeof(int), 0,
                                          cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return e;
  int* dev_status = nullptr;
  if ((e = cudaGetSymbolAddress(reinterpret_cast<void**>(&dev_status), g_selftest_status)) != cudaSuccess)
    return e;
  if ((e = tracked_launch(kProfOther, st, [&] { wait_selftest_kernel<<<1, 32, 0, st>>>(dev_status); })) !=
      cudaSuccess)
    return e;
  if ((e = cudaMemcpyFromSymbolAsync(status_host, g_selftest_status, sizeof(int), 0,
                                     cudaMemcpyDeviceToHost, st)) != cudaSuccess)
    return e;
  return cudaStreamSynchronize(st);
}

cudaError_t launch_tile_flags(const int32_t* rec_idx, int S, int nrec, int nx, int ny, uint8_t* flags,
                              cudaStream_t st) {
  const int tr = AdjLayout::kTR;
  const int tiles_x = (nx + tr - 1) / tr, tiles_y = (ny + kTY - 1) / kTY;
  cudaError_t e = cudaMemsetAsync(flags, 0, tma_tiles(nx, ny, S), st);
  if (e != cudaSuccess) return e;
  const int n = S * nrec;
  return tracked_launch(kProfOther, st, [&] {
    tile_flags_kernel<<<(n + 255) / 256, 256, 0, st>>>(rec_idx, S, nrec, nx, ny, tr, tiles_x, tiles_y,
                                                         flags);
  });
}

bool tma_eligible(int mode, int ny) { return mode == kModeDField && ny % 4 == 0 && encode_fn() != nullptr; }

size_t tma_tiles(int nx, int ny, int S) {
  return (size_t)S * ((nx + AdjLayout::kTR - 1) / AdjLayout::kTR) * ((ny + kTY - 1) / kTY);
}

namespace {
inline bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// CTAs of a persistent launch over `ntiles` tiles with room for `slots`
// resident CTAs: every slot.  (Spreading the tiles evenly over the fewest
// CTAs of the same number of waves measured slower, damage512 81.7 -> 88.8
// ms and multi64 734 -> 737 ms: the memory-bound kernels lose more to the
// fewer CTAs in flight than the last partial wave costs.)
inline int persistent_grid(int ntiles, int slots) { return ntiles < slots ? ntiles : slots; }
}  // namespace

// Steps the tiled kernels cannot take (u^i == 0 at the first step, buffers
// not on 16-byte boundaries) run on the plain per-step kernels instead.
// The launches are not chained: their grids fill every SM (one CTA per
// resident slot), and chaining the adjoint measured slower (8 x 512^2: 82.0
// against 88.6 ms per iteration).
cudaError_t launch_tma_fwd(const FwdStep& a, int* err, cudaStream_t st) {
  using F = FwdLayout;
  const bool ok = al16(a.field) && a.cur != nullptr && a.ny % 4 == 0 && al16(a.cur) && al16(a.prev) && al16(a.out) &&
                  al16(a.copy0) && al16(a.copy1) && (a.frame < 0 || (al16(a.hist_x) && al16(a.hist_y)));
  CUtensorMap cur_map, prev_map;
  if (!ok || !make_map(&cur_map, a.cur, a.nx, a.ny, a.S, kBW, F::kBHa) ||
      !make_map(&prev_map, a.prev ? a.prev : a.cur, a.nx, a.ny, a.S, kTY, F::kTR))
    return launch_fwd_step(kModeDField, a, st);
  cudaError_t e = set_smem();
  if (e != cudaSuccess) return e;
  const int tiles_x = (a.nx + F::kTR - 1) / F::kTR, tiles_y = (a.ny + kTY - 1) / kTY;
  const int grid = persistent_grid(a.S * tiles_x * tiles_y, device_info().sms * F::kCtasPerSm);
  return tracked_launch(kProfForward, st, [&] {
    launch_step_kernel(tma_fwd_kernel, dim3(grid), dim3(kThreads), kFwdSmem, st, false, a, cur_map, prev_map, tiles_x,
                       tiles_y, a.prev ? 1 : 0, err);
  }, (double)a.S * a.nx * a.ny * alg_bytes_forward(kModeDField));
}

cudaError_t launch_tma_adj(const AdjStep& a, int* err, cudaStream_t st) {
  using L = AdjLayout;
  const bool ok = al16(a.field) && al16(a.gacc) && a.ny % 4 == 0 && a.cur != nullptr && a.prev != nullptr &&
                  al16(a.cur) && al16(a.prev) && al16(a.out) && al16(a.u) &&
                  (a.record != kRecordFields || (al16(a.g_x) && al16(a.g_y)));
  CUtensorMap cur_map, u_map, d_map;
  if (!ok || !make_map(&cur_map, a.cur, a.nx, a.ny, a.S, kBW, L::kBHa) ||
      !make_map(&u_map, a.u ? a.u : a.cur, a.nx, a.ny, a.S, kBW, L::kBHa) ||
      !make_map2(&d_map, a.field, a.nx, a.ny, kBW, L::kBHa))
    return launch_adj_step(kModeDField, a, st);
  cudaError_t e = set_smem();
  if (e != cudaSuccess) return e;
  const int tiles_x = (a.nx + L::kTR - 1) / L::kTR, tiles_y = (a.ny + kTY - 1) / kTY;
  const int grid = persistent_grid(a.S * tiles_x * tiles_y, device_info().sms * L::kCtasPerSm);
  return tracked_launch(kProfAdjoint, st, [&] {
    launch_step_kernel(tma_adj_kernel, dim3(grid), dim3(kThreads), kAdjSmem, st, false, a, cur_map, u_map, d_map,
                       tiles_x, tiles_y, a.u ? 1 : 0, err);
  }, (double)a.S * a.nx * a.ny * alg_bytes_adjoint(kModeDField));
}

}  // namespace ernn
