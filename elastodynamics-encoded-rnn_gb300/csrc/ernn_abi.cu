// C ABI entry points of libernn_gb300.so (declared in include/ernn.h) and the
// host-side time-loop driver: step schedule, checkpoint/recompute plan,
// workspace layout.  Every launch goes on the caller's stream; nothing here
// synchronises the host or allocates device memory.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstddef>
#include <cstring>

#include "ernn.h"
#include "ernn_block.h"
#include "ernn_launch.h"
#include "ernn_resident.h"
#include "ernn_tma.h"

namespace ernn {
namespace {

constexpr size_t kAlign = 256;
constexpr double kPi = 3.14159265358979323846;
// segment length of the resident reverse pass when the tape keeps every state
constexpr int kResStoreAllSegment = 128;
constexpr int kBlockMinCols = 40;
constexpr double kBlockMaxFields = 1e6;
inline size_t align_up(size_t v) { return (v + kAlign - 1) / kAlign * kAlign; }

// Workspace plan of one problem.
struct Plan {
  int S, nx, ny, nt, k, nseg, nt_out, nblocks, npart, kres;
  int ncoef;  // coefficient blocks: nshots with ERNN_FLAG_SHOT_CONSTANTS, else 1
  bool store_all;
  size_t N, state_bytes;
  // tape
  size_t t_coef, t_A, t_B, t_store, t_total_tape, t_total_notape;
  // adjoint scratch
  size_t s_coef, s_LA, s_LB, s_seg, s_lbuf, s_gacc, s_part, s_tflags, s_total;
  // instances on a canvas: tile table (tape and scratch)
  bool inst;
  size_t inst_bytes, t_inst, s_inst;
  // time-blocked tile kernels: the problem is theirs (given aligned buffers),
  // floats between rows of a state, two more working levels in the tape and
  // the scratch
  bool block;
  int pitch, geo;
  size_t t_C, t_D, t_rec, t_flag, s_LC, s_LD, s_rec, s_flag;
};

// Grids that the plain per-step kernels took before the time-blocked ones:
// odd rows, or a step of fewer than four 64 x 32 tiles per SM of this part's
// 152.  From sizes alone: the workspace plan and the choice of the tiled
// per-step kernels (use_tiled), whose tables the plan makes room for, use the
// same line on every device.
constexpr size_t kTiledMinTiles = 4 * 152;
inline bool plain_size(const ErnnProblem& p) {
  return p.path == ERNN_PATH_AUTO && !(p.flags & ERNN_FLAG_INSTANCES) &&
         (p.ny % 4 != 0 || tma_tiles(p.nx, p.ny, p.nshots) < kTiledMinTiles);
}

inline bool cluster_fits(const ErnnProblem& p) {
  return resident_fits(p.mode, p.nx, p.ny, p.record == kRecordReceivers ? p.nrec : 0);
}

// Estimates of the time that the per-cell modes take a step, us: here by waves
// of tiles, in the plain kernels by the cells of their blocks (columns to 32,
// rows to 8).  Fitted to some 50 grids of each mode, 17 thousand to 1.8 million
// cells, 9 to 20000 rows; us there -> here on either side of the line:
//   constant planes, every state kept: 1 x 3000x240 34.0 -> 18.5, 16 x 250^2
//     39.3 -> 37.0, 20 x 130^2 19.1 -> 18.9; 300 x 50^2 41.6 -> 47.0, 120 x 64^2
//     22.1 -> 25.5; checkpoints (every 13 steps: the forward counts twice, and
//     segments end launches early) 8 x 301^2 46.2 -> 32.4; 16 x 250^2 50.3 ->
//     54.9; forward alone 8 x 301^2 9.6 -> 7.9; 16 x 250^2 10.6 -> 13.0
//   degradation map: 7 x 301^2 20.1 -> 14.8, 1 x 700x701 14.9 -> 14.1; 10 x
//     200x201 14.3 -> 14.7, 8 x 500x121 16.1 -> 18.6, 7 x 563x51 10.2 -> 14.5
//     (the same line with checkpoints, within 2 %)
enum class Pass { kForward, kBoth };
bool per_cell_tiles(const ErnnProblem& p, Pass pass) {
  const bool small = step_rows(p.nx, p.ny, p.nshots) == 8;  // blocks of the plain kernels
  const double rows = (p.nx + 7) / 8 * 8.0, cols = (p.ny + 31) / 32 * 32.0;
  double M = 1e-6 * p.nshots * rows * cols;
  if (p.mode == kModeDField) {
    const int geo = blk_geometry(p.mode, p.nx, p.ny, p.nshots);
    const double w = std::ceil(p.nshots * (double)blk_tiles(geo, p.nx, p.ny) / (geo == kBlkTall ? 304.0 : 152.0));
    return 1.0 + (geo == kBlkTall ? 17.0 : geo == kBlkShort ? 6.8 : 4.1) * w <=
           (small ? 6.3 + 17.0 * M : 6.5 + 18.4 * M);
  }
  const double tiles = p.nshots * (double)blk_tiles(kBlkFlat, p.nx, p.ny);
  if (tiles <= 152.0) return true;  // a run: half the time of the plain kernels
  // (a twentieth of a wave is lost in the wave before it)
  const double w = std::ceil(tiles / 152.0 - 0.05);
  double fwd = 0.9 + 1.07 * w, adj = 0.4 + 2.25 * w;
  if (p.ny <= 48 && p.nx > 64) fwd *= 0.94, adj *= 0.88;  // (half the sectors of a row)
  if (!small) M *= 0.5 + 0.5 * ((p.ny + 7) / 8 * 8.0) / cols;  // (a block's idle columns cost half)
  const double fwd_plain = small ? 2.1 + 9.0 * M : 2.0 + 8.4 * M, adj_plain = small ? 4.2 + 20.0 * M : 14.0 + 15.6 * M;
  if (pass == Pass::kForward) return fwd <= fwd_plain;
  if (p.ckpt_k >= p.nt) return fwd + adj <= fwd_plain + adj_plain;
  const double whole = std::ceil(p.ckpt_k / (double)kBlkSteps) * kBlkSteps / p.ckpt_k;
  return (2.0 * fwd + adj) * (0.5 + 0.5 * whole) <= 2.0 * fwd_plain + adj_plain;
}

// Problems of the time-blocked tile kernels, from sizes alone (the workspace
// queries, the forward and the adjoint agree).
//  - Instances, and scalar constants on the tiled path: all of them.
//  - ERNN_PATH_AUTO takes rows of any length from kBlockMinCols up (16 x
//    941x41, 200 steps, time-blocked tiles against plain kernels: 4.98 and
//    5.11 ms; 5 x 1000x41: 2.52 and 3.05), shorter ones from the size at which
//    one-step tiles used to take them (64 x 4000x36, 40 steps: 5.29 ms, 15.7
//    with the plain kernels, 7.63 with those tiles; 4 x 5000x32: 0.75, 1.02
//    and 1.25); states of odd rows are padded to 16-byte rows.
//    Where the cluster-resident path fits it comes first (on a device that
//    cannot schedule its clusters such a problem takes the plain kernels).
//    Larger receiver arrays, and grids that no cluster size can hold, come
//    here (us per iteration, plain -> here: 24 x 256^2 with 2000 receivers,
//    60 steps, 3980 -> 1616; 64 x 128^2 with 1100, 100 steps, 3631 -> 2308).
//  - A degradation map: grids of the plain kernels' size.  On larger ones the
//    TMA-fed kernels of one step are faster (8 x 512^2: 29 against 33 us per
//    forward and adjoint step): the map, u's rows and the running gradient
//    are read at every step either way, here from L2 by the threads.
//  - Six constant planes: up to kBlockMaxFields cells.
//    Both per-cell modes where a forward and an adjoint step take less here
//    than with the plain kernels (per_cell_tiles); a forward without a tape of
//    constant planes asks for its own time (forward_impl).
bool block_rule(const ErnnProblem& p) {
  if (p.flags & ERNN_FLAG_INSTANCES) return true;
  if (p.path == ERNN_PATH_TILED) return p.mode == kModeScalar && p.ny % 4 == 0;
  if (p.path != ERNN_PATH_AUTO) return false;
  if (p.mode == kModeScalar) return (p.ny >= kBlockMinCols || !plain_size(p)) && !cluster_fits(p);
  if (p.ny < kBlockMinCols) return false;
  if (p.mode == kModeFields ? (double)p.nshots * p.nx * p.ny > kBlockMaxFields : !plain_size(p)) return false;
  return per_cell_tiles(p, Pass::kBoth);
}

// Upper bound of the tile-table entries of any placement of S instances on
// an nx x ny canvas (each instance's tiling has at most one partial tile row
// and column; tiles of whole rows are fewer).
inline size_t inst_table_bound(int nx, int ny, int S) {
  const BlkShape g = blk_shape(kBlkTall);
  return ((size_t)(nx + g.rows - 1) / g.rows + S) * ((size_t)(ny + g.cols - 1) / g.cols + S);
}

Plan make_plan(const ErnnProblem& p) {
  Plan pl{};
  pl.S = p.nshots; pl.nx = p.nx; pl.ny = p.ny; pl.nt = p.nt;
  pl.k = p.ckpt_k < p.nt ? p.ckpt_k : p.nt;
  pl.nseg = (p.nt + pl.k - 1) / pl.k;
  pl.store_all = (pl.nseg == 1);
  pl.nt_out = (p.nt + p.stride - 1) / p.stride;
  pl.N = (size_t)p.nx * p.ny;
  pl.inst = (p.flags & ERNN_FLAG_INSTANCES) != 0;
  // instances share the canvas's one state plane
  pl.block = block_rule(p);
  pl.geo = pl.inst ? kBlkTall : p.mode == kModeFields ? kBlkFlat : blk_geometry(p.mode, p.nx, p.ny, p.nshots);
  pl.pitch = pl.block ? (p.ny + 3) / 4 * 4 : p.ny;
  pl.state_bytes = align_up((size_t)(pl.inst ? 1 : p.nshots) * 2 * p.nx * pl.pitch * sizeof(float));
  const dim3 g = step_grid(p.nx, p.ny, pl.inst ? 1 : p.nshots);
  pl.nblocks = (int)(g.x * g.y * g.z);
  pl.ncoef = (p.flags & (ERNN_FLAG_SHOT_CONSTANTS | ERNN_FLAG_INSTANCES)) ? p.nshots : 1;
  pl.inst_bytes = pl.inst ? align_up(inst_table_bound(p.nx, p.ny, p.nshots) * sizeof(int4)) +
                                align_up((size_t)2 * p.nshots * sizeof(int4))
                          : 0;
  size_t off = 0;
  pl.t_coef = off; off += align_up((size_t)pl.ncoef * sizeof(Coef));
  pl.t_inst = off; off += pl.inst_bytes;
  pl.t_A = off; off += pl.state_bytes;
  pl.t_B = off; off += pl.state_bytes;
  pl.t_C = off; if (pl.block) off += pl.state_bytes;
  pl.t_D = off; if (pl.block) off += pl.state_bytes;
  // receivers of the tiles
  const size_t rec_bytes =
      pl.block && p.record == kRecordReceivers
          ? align_up(blk_rec_bytes(pl.inst ? inst_table_bound(p.nx, p.ny, p.nshots)
                                           : (size_t)p.nshots * blk_tiles(pl.geo, p.nx, p.ny), p.nshots, p.nrec))
          : 0;
  pl.t_rec = off; off += rec_bytes;
  // pass counters of the tiles (runs)
  const size_t flag_bytes =
      pl.block && !pl.inst ? align_up((size_t)p.nshots * blk_tiles(pl.geo, p.nx, p.ny) * sizeof(int)) : 0;
  pl.t_flag = off; off += flag_bytes;
  pl.t_total_notape = off;
  pl.t_store = off;
  if (pl.store_all) off += (size_t)p.nt * pl.state_bytes;           // u^1..u^nt
  else off += (size_t)(pl.nseg - 1) * 2 * pl.state_bytes;          // (u^{jk}, u^{jk-1})
  pl.t_total_tape = off;
  off = 0;
  pl.s_coef = off; off += align_up((size_t)pl.ncoef * sizeof(Coef));
  pl.s_inst = off; off += pl.inst_bytes;
  pl.s_LA = off; off += pl.state_bytes;
  pl.s_LB = off; off += pl.state_bytes;
  pl.s_LC = off; if (pl.block) off += pl.state_bytes;
  pl.s_LD = off; if (pl.block) off += pl.state_bytes;
  pl.s_rec = off; off += rec_bytes;
  pl.s_flag = off; off += flag_bytes;
  // two recompute segments: the cluster-resident path recomputes segment j-1
  // while the adjoint consumes segment j
  // (one segment where that path cannot run)
  const bool res = cluster_fits(p) && !pl.inst;
  pl.s_seg = off; if (!pl.store_all) off += (size_t)(pl.block && !res ? 1 : 2) * pl.k * pl.state_bytes;
  // lam buffers of the resident reverse pass: two segments of kres steps,
  // only where that path can run
  pl.kres = pl.store_all ? (p.nt < kResStoreAllSegment ? p.nt : kResStoreAllSegment) : pl.k;
  if (!res) pl.kres = 0;
  pl.s_lbuf = off; off += (size_t)2 * pl.kres * pl.state_bytes;
  pl.s_gacc = off;
  if (p.mode == kModeDField) off += align_up((size_t)p.nshots * pl.N * sizeof(float));
  if (p.mode == kModeFields) off += align_up((size_t)p.nshots * 6 * pl.N * sizeof(float));
  pl.s_part = off;
  // partial-sum rows: plain per-step path one per block; resident path one
  // per imaging CTA (at most 8 clusters of 16 per shot); tiled path one per
  // CTA, kTiledRowsPerShot per shot with per-shot constants
  pl.npart = pl.nblocks > p.nshots * 16 * 8 ? pl.nblocks : p.nshots * 16 * 8;
  if (pl.ncoef > 1 && pl.npart < p.nshots * kTiledRowsPerShot) pl.npart = p.nshots * kTiledRowsPerShot;
  if (p.mode == kModeScalar) off += align_up((size_t)pl.npart * 8 * sizeof(double));
  // receiver table of the tiled per-step adjoint: one byte per (shot, tile)
  pl.s_tflags = off;
  if (p.record == kRecordReceivers && !pl.block) off += align_up(tma_tiles(p.nx, p.ny, p.nshots));
  if (pl.block) off += 16;  // the scratch starts at its first 16-byte boundary
  pl.s_total = off;
  return pl;
}

int validate(const ErnnProblem* p) {
  if (p == nullptr) return ERNN_ERR_INVALID;
  if (p->nshots < 1 || p->nshots > 65535 || p->nx < 1 || p->ny < 1 || p->nt < 1 ||
      p->stride < 1 || p->ckpt_k < 1)
    return ERNN_ERR_INVALID;
  if ((int64_t)p->nx * p->ny >= ((int64_t)1 << 31) || p->nx > 2000000) return ERNN_ERR_INVALID;
  if (p->mode < kModeScalar || p->mode > kModeFields) return ERNN_ERR_INVALID;
  if (p->record != kRecordFields && p->record != kRecordReceivers) return ERNN_ERR_INVALID;
  if (p->record == kRecordReceivers && p->nrec < 1) return ERNN_ERR_INVALID;
  if (p->src_comp != 0 && p->src_comp != 1) return ERNN_ERR_INVALID;
  if (p->src_bx < 0 || p->src_by < 0) return ERNN_ERR_INVALID;
  if (p->path < ERNN_PATH_AUTO || p->path > ERNN_PATH_TILED) return ERNN_ERR_INVALID;
  if ((p->flags & ~(ERNN_FLAG_SHOT_CONSTANTS | ERNN_FLAG_INSTANCES | ERNN_FLAG_TALL_TILES)) != 0)
    return ERNN_ERR_INVALID;
  if ((p->flags & ERNN_FLAG_SHOT_CONSTANTS) && p->mode != kModeScalar) return ERNN_ERR_INVALID;
  if ((p->flags & ERNN_FLAG_INSTANCES) &&
      (p->mode != kModeScalar || p->record != kRecordReceivers || p->nshots > kMaxInstances ||
       p->nx >= 65536 || p->ny >= 65536))
    return ERNN_ERR_INVALID;
  if (!(p->h > 0.0) || !(p->dt > 0.0) || !std::isfinite(p->h) || !std::isfinite(p->dt))
    return ERNN_ERR_INVALID;
  // Sizes that the plan forms in 64-bit (states of the tape and scratch: at
  // most nt + 2 ckpt_k + 2 resident segments + a few) and in 32-bit (blocks
  // of one plain step launch) must not wrap: such a problem is refused
  // instead of being given a workspace size that is too small.
  const double state_bytes =
      (double)((p->flags & ERNN_FLAG_INSTANCES) ? 1 : p->nshots) * 2.0 * (double)p->nx * p->ny * 4.0;
  if (state_bytes * (3.0 * (double)p->nt + 16.0) >= 4.0e18) return ERNN_ERR_INVALID;
  if ((double)p->nshots * ((p->nx + 7) / 8) * ((p->ny + 31) / 32) >= 2.0e9) return ERNN_ERR_INVALID;
  return ERNN_OK;
}

int validate_inputs(const ErnnProblem* p, const ErnnInputs* in) {
  if (in == nullptr || in->C == nullptr || in->rho == nullptr || in->src_signal == nullptr)
    return ERNN_ERR_INVALID;
  if (p->mode == kModeDField && in->D == nullptr) return ERNN_ERR_INVALID;
  if ((size_t)p->src_bx * p->src_by > 0 && (in->src_map == nullptr || in->src_origin == nullptr))
    return ERNN_ERR_INVALID;
  if (p->record == kRecordReceivers && in->rec_idx == nullptr) return ERNN_ERR_INVALID;
  return ERNN_OK;
}

inline bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
// The scratch of a time-blocked problem is used from its first 16-byte
// boundary (states that TMA reads).
inline void* scratch_base(const Plan& pl, void* scratch) {
  const uintptr_t v = reinterpret_cast<uintptr_t>(scratch);
  return pl.block ? reinterpret_cast<void*>((v + 15u) & ~(uintptr_t)15u) : scratch;
}

inline char* at(void* base, size_t off) { return static_cast<char*>(base) + off; }
inline float* fat(void* base, size_t off) { return reinterpret_cast<float*>(at(base, off)); }

#define ERNN_CUDA(expr)                      \
  do {                                       \
    if ((expr) != cudaSuccess) return ERNN_ERR_CUDA; \
  } while (0)

FwdStep base_fwd(const ErnnProblem& p, const ErnnInputs& in, const Coef* coef, int nt_out) {
  FwdStep a;
  std::memset(&a, 0, sizeof(a));
  a.nx = p.nx; a.ny = p.ny; a.S = p.nshots; a.nt = p.nt;
  a.frame = -1; a.gframe = -1; a.nt_out = nt_out;
  a.coef = coef;
  // one coefficient block per shot (per-shot constants) or per instance
  a.coef_stride = (p.flags & (ERNN_FLAG_SHOT_CONSTANTS | ERNN_FLAG_INSTANCES)) ? 1 : 0;
  a.field = (p.mode == kModeFields) ? in.C : in.D;
  a.src_signal = in.src_signal;
  a.src_map = in.src_map;
  a.src_origin = in.src_origin;
  a.bx = p.src_bx; a.by = p.src_by; a.src_comp = p.src_comp;
  a.rec_idx = in.rec_idx;
  a.nrec = p.nrec;
  return a;
}

std::atomic<int32_t> g_last_path{ERNN_PATH_AUTO};

// Tiled per-step kernels (degradation maps): requested (ERNN_PATH_TILED, an
// error when the problem is not eligible) or chosen by ERNN_PATH_AUTO when
// eligible and no plain_size grid.  They are persistent (2-3 CTAs of 72-111
// KB shared memory per SM, each streaming several tiles).  Scalar problems get
// here with a tape that is not on a 16-byte boundary, with few rows below
// kBlockMinCols cells, or on a device that cannot schedule the clusters of the
// resident path: the plain kernels take those.
int use_tiled(const ErnnProblem& p, int* tiled) {
  *tiled = 0;
  if (p.path == ERNN_PATH_STEP) return ERNN_OK;
  const bool ok = tma_eligible(p.mode, p.ny);
  if (p.path == ERNN_PATH_TILED) {
    *tiled = ok;
    return ok || (p.mode == kModeScalar && p.ny % 4 == 0 && blk_available()) ? ERNN_OK : ERNN_ERR_UNSUPPORTED;
  }
  *tiled = ok && !plain_size(p);
  return ERNN_OK;
}

// Cluster-resident configuration: CL CTAs of R rows each.  Returns false when
// the problem does not fit the path (mode, alignment, receivers, memory).
bool pick_resident(const ErnnProblem& p, const ErnnInputs& in, Coef* coef, ResCommon& rc) {
  if (!cluster_fits(p)) return false;  // (the plan reserved no lam buffers)
  rc.nx = p.nx; rc.ny = p.ny; rc.S = p.nshots; rc.nt = p.nt; rc.stride = p.stride;
  rc.nt_out = (p.nt + p.stride - 1) / p.stride;
  rc.coef = coef;
  rc.coef_stride = (p.flags & ERNN_FLAG_SHOT_CONSTANTS) ? 1 : 0;
  rc.src_signal = in.src_signal; rc.src_map = in.src_map; rc.src_origin = in.src_origin;
  rc.bx = p.src_bx; rc.by = p.src_by; rc.src_comp = p.src_comp;
  rc.rec_idx = (p.record == kRecordReceivers) ? in.rec_idx : nullptr;
  rc.nrec = (p.record == kRecordReceivers) ? p.nrec : 0;
  rc.err = &coef->err;
  for (int CL = 16; CL >= 1; CL /= 2) {
    rc.CL = CL;
    rc.R = resident_rows(p.nx, CL);
    if (rc.R > 0 && resident_feasible(rc, p.record == kRecordFields)) return true;
  }
  return false;
}

int resident_forward(const ErnnProblem& p, const Plan& pl, ResCommon& rc, float* out_ux,
                     float* out_uy, void* tape, int with_tape, cudaStream_t st) {
  ResFwd f;
  std::memset(&f, 0, sizeof(f));
  f.i0 = 0; f.i1 = p.nt;
  f.state_stride = pl.state_bytes / sizeof(float);
  if (with_tape && pl.store_all) f.states = fat(tape, pl.t_store);
  if (with_tape && !pl.store_all) {
    f.ckpt = fat(tape, pl.t_store);
    f.ck_k = pl.k;
    f.ck_nseg = pl.nseg;
  }
  const bool dense = (p.record == kRecordFields);
  if (dense) { f.hist_x = out_ux; f.hist_y = out_uy; }
  else { f.tr_x = out_ux; f.tr_y = out_uy; }
  ResLam a;
  std::memset(&a, 0, sizeof(a));
  ResImg g;
  std::memset(&g, 0, sizeof(g));
  ERNN_CUDA(launch_resident(rc, f, a, g, true, false, false, dense, st));
  return ERNN_OK;
}

// Reverse pass of the resident path, in segments of ks steps, one launch per
// segment j (from the last): LAM runs the adjoint over segment j and stores
// every lam into lbuf[j & 1]; FWD recomputes segment j from its checkpoint
// into ubuf[j & 1] (not needed when the tape holds every state); IMG forms the
// imaging sums of segment j + 1 from the buffers of the previous launch.
int resident_adjoint(const ErnnProblem& p, const Plan& pl, ResCommon& rc, const float* g_ux,
                     const float* g_uy, void* tape, void* scratch, double* partials,
                     int* img_rows, cudaStream_t st) {
  const size_t ss = pl.state_bytes / sizeof(float);
  const bool dense = (p.record == kRecordFields);
  const int ks = pl.kres;
  const int nseg = (p.nt + ks - 1) / ks;
  auto lbuf = [&](int j) { return fat(scratch, pl.s_lbuf + (size_t)(j & 1) * ks * pl.state_bytes); };
  auto ubuf = [&](int j) -> float* {
    if (pl.store_all) return fat(tape, pl.t_store + (size_t)j * ks * pl.state_bytes);  // u^{jk+1}..
    return fat(scratch, pl.s_seg + (size_t)(j & 1) * pl.k * pl.state_bytes);
  };
  auto ck = [&](int j, int lev) -> const float* {
    if (j == 0) return nullptr;
    if (lev == 1 && j * pl.k - 1 == 0) return nullptr;  // u^0 = 0 (k == 1)
    return fat(tape, pl.t_store + ((size_t)(j - 1) * 2 + lev) * pl.state_bytes);
  };
  ResLam a;
  std::memset(&a, 0, sizeof(a));
  a.lam_save = fat(scratch, pl.s_LA);
  a.save_stride = ss;  // LB follows LA
  a.g_x = g_ux; a.g_y = g_uy;
  a.state_stride = ss;
  ResFwd f;
  std::memset(&f, 0, sizeof(f));
  f.state_stride = ss;
  ResImg g;
  std::memset(&g, 0, sizeof(g));
  g.state_stride = ss;
  g.partials = partials;
  *img_rows = resident_img_clusters(rc) * rc.S * rc.CL;
  for (int j = nseg - 1; j >= -1; --j) {
    const bool run_lam = j >= 0;
    bool run_fwd = false;
    if (run_lam) {
      a.m_hi = (j + 1) * ks < p.nt ? (j + 1) * ks : p.nt;
      a.m_lo = j * ks;
      a.first = (j == nseg - 1) ? 1 : 0;
      a.lbuf = lbuf(j);
      a.slot_base = j * ks + 2;
      a.store_init = (a.m_hi <= p.nt - 1) ? 1 : 0;
      if (!pl.store_all) {  // recompute u^{jk+1} .. u^{min((j+1)k, nt-1)}
        f.i0 = j * pl.k;
        f.i1 = (j + 1) * pl.k < p.nt - 1 ? (j + 1) * pl.k : p.nt - 1;
        f.init_cur = ck(j, 0);
        f.init_prev = ck(j, 1);
        f.states = ubuf(j);
        run_fwd = f.i1 > f.i0;
      }
    }
    const int jj = j + 1;  // segment imaged in this launch
    g.n_lo = jj * ks + 1;
    g.n_hi = (jj + 1) * ks < p.nt - 1 ? (jj + 1) * ks : p.nt - 1;
    const bool run_img = jj <= nseg - 1 && g.n_hi >= g.n_lo;
    if (run_img) {
      g.lbuf = lbuf(jj);
      g.ubuf = ubuf(jj);
    }
    ERNN_CUDA(launch_resident(rc, f, a, g, run_fwd, run_lam, run_img, dense, st));
  }
  return ERNN_OK;
}

// Instances of a canvas problem (ERNN_FLAG_INSTANCES), checked and ordered
// by decreasing step count; upto[g] = tiles of the first g of that order.
struct InstPlan {
  InstDesc d;
  int geo;  // tiles: kBlkTall, or kBlkRow64 where every instance fits its columns
  int upto[kMaxInstances + 1];
  // tiles of forward (or recompute) step i: instances with nt > i
  int fwd_tiles(int i) const {
    int g = 0;
    while (g < d.count && d.nt[g] > i) ++g;
    return upto[g];
  }
  // tiles of adjoint step m: instances with nt >= m
  int adj_tiles(int m) const {
    int g = 0;
    while (g < d.count && d.nt[g] >= m) ++g;
    return upto[g];
  }
};

int plan_instances(const ErnnProblem& p, const ErnnInstances* in, InstPlan* ip) {
  if (!(p.flags & ERNN_FLAG_INSTANCES) || in == nullptr || in->count != p.nshots || in->x0 == nullptr ||
      in->y0 == nullptr || in->nx == nullptr || in->ny == nullptr || in->nt == nullptr)
    return ERNN_ERR_INVALID;
  const int S = in->count;
  for (int k = 0; k < S; ++k) {
    const int x0 = in->x0[k], y0 = in->y0[k], nx = in->nx[k], ny = in->ny[k], nt = in->nt[k];
    if (x0 < 0 || y0 < 0 || nx < 1 || ny < 4 || y0 % 4 != 0 || ny % 4 != 0 || (int64_t)x0 + nx > p.nx ||
        (int64_t)y0 + ny > p.ny || nt < 1 || nt > p.nt)  // (64-bit sums: no wrap past the canvas)
      return ERNN_ERR_INVALID;
  }
  // regions at least one cell apart: those cells stay zero, the instances'
  // ghost rings
  for (int a = 0; a < S; ++a)
    for (int b = a + 1; b < S; ++b) {
      const bool apart = in->x0[a] + in->nx[a] + 1 <= in->x0[b] || in->x0[b] + in->nx[b] + 1 <= in->x0[a] ||
                         in->y0[a] + in->ny[a] + 1 <= in->y0[b] || in->y0[b] + in->ny[b] + 1 <= in->y0[a];
      if (!apart) return ERNN_ERR_INVALID;
    }
  int order[kMaxInstances];
  for (int k = 0; k < S; ++k) order[k] = k;
  std::stable_sort(order, order + S, [&](int u, int v) { return in->nt[u] > in->nt[v]; });
  ip->d.count = S;
  // Tiles of whole rows where they save a wave of tiles (256 instances of 300 x
  // 32, 60 steps: 5.66 -> 3.52 ms).
  size_t tall = 0, rows = 0;
  bool narrow = true;
  for (int k = 0; k < S; ++k) {
    tall += blk_tiles(kBlkTall, in->nx[k], in->ny[k]);
    rows += blk_tiles(kBlkRow64, in->nx[k], in->ny[k]);
    narrow = narrow && in->ny[k] <= blk_shape(kBlkRow64).cols;
  }
  ip->geo = narrow && (rows + 303) / 304 < (tall + 303) / 304 ? kBlkRow64 : kBlkTall;
  ip->d.tile_rows = blk_shape(ip->geo).rows;
  ip->d.tile_cols = blk_shape(ip->geo).cols;
  ip->upto[0] = 0;
  for (int g = 0; g < S; ++g) {
    const int k = order[g];
    ip->d.id[g] = k;
    ip->d.x0[g] = in->x0[k];
    ip->d.y0[g] = in->y0[k];
    ip->d.nx[g] = in->nx[k];
    ip->d.ny[g] = in->ny[k];
    ip->d.nt[g] = in->nt[k];
    ip->d.base[g] = ip->upto[g];
    ip->upto[g + 1] = ip->upto[g] + (int)blk_tiles(ip->geo, in->nx[k], in->ny[k]);
  }
  return ERNN_OK;
}

// Steps of the next launch of a run of n: four at a time, the rest in
// launches of two or three (one only where the run has one step: a launch
// of one step leaves its older level behind in the buffer it read).
inline int block_steps(int n) { return n <= kBlkSteps ? n : (n == kBlkSteps + 1 ? kBlkSteps - 1 : kBlkSteps); }

// Of four working states, one that is neither x, y nor z.
inline float* free_state(float* const pool[4], const float* x, const float* y, const float* z) {
  for (int k = 0; k < 4; ++k)
    if (pool[k] != x && pool[k] != y && pool[k] != z) return pool[k];
  return nullptr;
}

BlkFwd base_blk_fwd(const ErnnProblem& p, const Plan& pl, const ErnnInputs& in, const InstPlan* ip, const Coef* coef,
                    const InstTiles& it) {
  BlkFwd a;
  std::memset(&a, 0, sizeof(a));
  a.geo = ip != nullptr ? ip->geo : pl.geo;
  a.plain_order = plain_size(p) ? 1 : 0;
  a.nx = p.nx; a.ny = p.ny; a.pitch = pl.pitch; a.S = p.nshots; a.nt = p.nt;
  a.nt_out = pl.nt_out; a.record = p.record; a.nrec = p.nrec;
  a.coef = coef; a.coef_stride = pl.ncoef > 1 ? 1 : 0;
  a.field = p.mode == kModeFields ? in.C : in.D;
  a.vec_field = p.ny % 4 == 0 && al16(a.field);
  a.src_signal = in.src_signal; a.src_map = in.src_map; a.src_origin = in.src_origin;
  a.bx = p.src_bx; a.by = p.src_by; a.src_comp = p.src_comp;
  a.inst = it;
  for (int t = 0; t <= kBlkSteps; ++t) a.frame[t] = -1;
  return a;
}

// Tiles of a time-blocked call.
size_t block_tiles(const ErnnProblem& p, const Plan& pl, const InstPlan* ip) {
  return ip != nullptr ? (size_t)ip->upto[ip->d.count] : (size_t)p.nshots * blk_tiles(pl.geo, p.nx, p.ny);
}

// Passes collected into runs (one cooperative launch each) where the tiles fit
// the chip, one per SM; otherwise every pass is a launch.  Measured, a launch
// per pass -> runs: 301^2 dense 4.69 -> 3.91 ms, 512^2 traces 5.23 -> 4.05,
// 301^2 constant planes 18.3 -> 17.1.  (52-row tiles for grids of up to 1 M
// cells, 12 warps of five rows: 3 x 501x389 8.27 -> 8.60 ms, left out.)
struct PassRunner {
  int mode;
  int* err;
  cudaStream_t st;
  bool on;
  int epoch = 0;
  bool chained = false;  // a launch of the loop precedes
  int* flags;
  FwdRun f;
  AdjRun r;
  const BlkFwd* fa = nullptr;
  const BlkAdj* ra = nullptr;

  PassRunner(const ErnnProblem& p, const Plan& pl, const InstPlan* ip, int* flags_, int* err_, cudaStream_t st_)
      : mode(p.mode), err(err_), st(st_), flags(flags_) {
    // (the setting alone: a profiled call makes the launches of an unprofiled one)
    on = ip == nullptr && launch_overlap_setting() && (p.mode != kModeScalar || plain_size(p)) &&
         blk_run_fits(p.mode, pl.geo, p.nx, p.ny, p.nshots);
    f.n = r.n = 0;
  }
  cudaError_t start(const ErnnProblem& p, const Plan& pl) {
    return on ? cudaMemsetAsync(flags, 0, (size_t)p.nshots * blk_tiles(pl.geo, p.nx, p.ny) * sizeof(int), st)
              : cudaSuccess;
  }
  cudaError_t add(BlkFwd& a) {
    if (!on) {
      a.chained = chained;
      chained = true;
      return launch_blk_fwd(mode, a, err, st);
    }
    FwdPass& q = f.p[f.n++];
    q.i = a.i; q.T = a.T; q.cur = a.cur; q.prev = a.prev;
    for (int t = 0; t <= kBlkSteps; ++t) { q.out[t] = a.out[t]; q.frame[t] = a.frame[t]; }
    fa = &a;
    return f.n == kRunPasses ? flush() : cudaSuccess;
  }
  cudaError_t add(BlkAdj& b) {
    if (!on) {
      b.chained = chained;
      chained = true;
      return launch_blk_adj(mode, b, err, st);
    }
    AdjPass& q = r.p[r.n++];
    q.m_hi = b.m_hi; q.T = b.T; q.cur = b.cur; q.prev = b.prev; q.out_last = b.out_last; q.out_before = b.out_before;
    ra = &b;
    return r.n == kRunPasses ? flush() : cudaSuccess;
  }
  cudaError_t flush() {
    cudaError_t e = cudaSuccess;
    if (f.n > 0) {
      f.epoch = epoch;
      f.flags = flags;
      epoch += f.n;
      e = launch_blk_fwd_run(mode, *fa, f, err, st);
      if (e == cudaErrorCooperativeLaunchTooLarge) {  // a context with fewer SMs: a launch per pass
        on = false;
        e = cudaSuccess;
        BlkFwd a = *fa;
        for (int k = 0; k < f.n && e == cudaSuccess; ++k) {
          const FwdPass& q = f.p[k];
          a.i = q.i; a.T = q.T; a.cur = q.cur; a.prev = q.prev;
          for (int t = 0; t <= kBlkSteps; ++t) { a.out[t] = q.out[t]; a.frame[t] = q.frame[t]; }
          e = add(a);
        }
      }
      f.n = 0;
    }
    if (e == cudaSuccess && r.n > 0) {
      r.epoch = epoch;
      r.flags = flags;
      epoch += r.n;
      e = launch_blk_adj_run(mode, *ra, r, err, st);
      if (e == cudaErrorCooperativeLaunchTooLarge) {
        on = false;
        e = cudaSuccess;
        BlkAdj b = *ra;
        for (int k = 0; k < r.n && e == cudaSuccess; ++k) {
          const AdjPass& q = r.p[k];
          b.m_hi = q.m_hi; b.T = q.T; b.cur = q.cur; b.prev = q.prev; b.out_last = q.out_last; b.out_before = q.out_before;
          e = add(b);
        }
      }
      r.n = 0;
    }
    return e;
  }
};

// Forward time loop on the time-blocked kernels: launches of up to four
// steps, ending at the checkpoints, whose pair of levels is what a launch
// leaves behind.
int block_forward(const ErnnProblem& p, const Plan& pl, const ErnnInputs& in, const InstPlan* ip, InstTiles itab,
                  Coef* coef, float* out_ux, float* out_uy, void* tape, int with_tape, cudaStream_t st) {
  BlkFwd a = base_blk_fwd(p, pl, in, ip, coef, itab);
  if (p.record == kRecordReceivers)
    ERNN_CUDA(launch_rec_tiles(a.geo, in.rec_idx, p.nshots, p.nrec, p.nx, p.ny, itab.box, block_tiles(p, pl, ip),
                               at(tape, pl.t_rec), &a.rec_tile, &a.rec_ent, out_ux, out_uy, pl.nt_out, st));
  a.rec_x = out_ux;
  a.rec_y = out_uy;
  a.vec = p.ny % 4 == 0 && al16(out_ux) && al16(out_uy);
  float* const pool[4] = {fat(tape, pl.t_A), fat(tape, pl.t_B), fat(tape, pl.t_C), fat(tape, pl.t_D)};
  const bool store_all = with_tape && pl.store_all;
  const int seg = with_tape && !pl.store_all ? pl.k : p.nt;
  const float *cur = nullptr, *prev = nullptr;
  PassRunner runner(p, pl, ip, reinterpret_cast<int*>(at(tape, pl.t_flag)), &coef->err, st);
  ERNN_CUDA(runner.start(p, pl));
  for (int i = 0; i < p.nt;) {
    const int end = (i / seg + 1) * seg < p.nt ? (i / seg + 1) * seg : p.nt;
    const int T = block_steps(end - i);
    a.i = i;
    a.T = T;
    a.cur = cur;
    a.prev = prev;
    for (int t = 0; t <= kBlkSteps; ++t) {
      a.out[t] = nullptr;
      a.frame[t] = t >= 1 && t <= T && (i + t - 1) % p.stride == 0 ? (i + t - 1) / p.stride : -1;
    }
    if (store_all) {
      for (int t = 1; t <= T; ++t) a.out[t] = fat(tape, pl.t_store + (size_t)(i + t - 1) * pl.state_bytes);
    } else {
      a.out[T] = free_state(pool, cur, prev, nullptr);
      if (T > 1) a.out[T - 1] = free_state(pool, cur, prev, a.out[T]);
      if (with_tape && end < p.nt && i + T == end) {  // checkpoint j: (u^{jk}, u^{jk-1})
        const int j = end / seg;
        a.out[T] = fat(tape, pl.t_store + (size_t)(j - 1) * 2 * pl.state_bytes);
        if (T > 1 || cur != nullptr) a.out[T - 1] = fat(tape, pl.t_store + ((size_t)(j - 1) * 2 + 1) * pl.state_bytes);
      }
    }
    if (ip != nullptr) a.inst.ntiles = ip->fwd_tiles(i);
    ERNN_CUDA(runner.add(a));
    prev = T > 1 ? a.out[T - 1] : cur;
    cur = a.out[T];
    i += T;
  }
  ERNN_CUDA(runner.flush());
  return ERNN_OK;
}

// Adjoint on the time-blocked kernels: per segment from the last, the
// recomputation of its states (when the tape does not hold them), then the
// reverse steps over it.
int block_adjoint(const ErnnProblem& p, const Plan& pl, const ErnnInputs& in, const InstPlan* ip, InstTiles itab,
                  Coef* coef, const float* g_ux, const float* g_uy, void* tape, void* scratch, double* partials,
                  cudaStream_t st) {
  BlkFwd a = base_blk_fwd(p, pl, in, ip, coef, itab);
  BlkAdj b;
  std::memset(&b, 0, sizeof(b));
  b.geo = a.geo;
  b.plain_order = a.plain_order;
  b.nx = p.nx; b.ny = p.ny; b.pitch = pl.pitch; b.S = p.nshots; b.nt = p.nt;
  b.u_stride = pl.state_bytes / sizeof(float);
  b.g_x = g_ux; b.g_y = g_uy;
  b.stride = p.stride; b.nt_out = pl.nt_out; b.record = p.record; b.nrec = p.nrec;
  if (p.record == kRecordReceivers)
    ERNN_CUDA(launch_rec_tiles(a.geo, in.rec_idx, p.nshots, p.nrec, p.nx, p.ny, itab.box, block_tiles(p, pl, ip),
                               at(scratch, pl.s_rec), &b.rec_tile, &b.rec_ent, nullptr, nullptr, 0, st));
  b.coef = coef;
  b.coef_stride = a.coef_stride;
  b.field = a.field;
  b.vec_field = a.vec_field;
  b.gacc = fat(scratch, pl.s_gacc);
  b.partials = partials;
  b.inst = itab;
  float* const pool[4] = {fat(scratch, pl.s_LA), fat(scratch, pl.s_LB), fat(scratch, pl.s_LC), fat(scratch, pl.s_LD)};
  PassRunner runner(p, pl, ip, reinterpret_cast<int*>(at(scratch, pl.s_flag)), &coef->err, st);
  ERNN_CUDA(runner.start(p, pl));
  const int seg = pl.store_all ? p.nt : pl.k, nseg = pl.store_all ? 1 : pl.nseg;
  for (int j = nseg - 1; j >= 0; --j) {
    const int i0 = j * seg, i1 = (j + 1) * seg < p.nt ? (j + 1) * seg : p.nt;
    if (pl.store_all) {
      b.u_base = fat(tape, pl.t_store);
    } else {
      // u^{i0+1} .. u^{i1} into the segment buffer (u^{nt} is never imaged)
      const int iend = i1 < p.nt ? i1 : p.nt - 1;
      const float* ck0 = j == 0 ? nullptr : fat(tape, pl.t_store + (size_t)(j - 1) * 2 * pl.state_bytes);
      const float* ck1 = j == 0 || j * pl.k - 1 == 0 ? nullptr  // u^0 = 0
                                                     : fat(tape, pl.t_store + ((size_t)(j - 1) * 2 + 1) * pl.state_bytes);
      auto slot = [&](int n) { return fat(scratch, pl.s_seg + (size_t)n * pl.state_bytes); };
      for (int i = i0; i < iend;) {
        const int T = block_steps(iend - i);
        a.i = i;
        a.T = T;
        a.cur = i == i0 ? ck0 : slot(i - i0 - 1);
        a.prev = i == i0 ? ck1 : (i == i0 + 1 ? ck0 : slot(i - i0 - 2));
        for (int t = 0; t <= kBlkSteps; ++t) a.out[t] = t >= 1 && t <= T ? slot(i - i0 + t - 1) : nullptr;
        if (ip != nullptr) a.inst.ntiles = ip->fwd_tiles(i);
        ERNN_CUDA(runner.add(a));
        i += T;
      }
      ERNN_CUDA(runner.flush());
      b.u_base = slot(0);
    }
    b.m_base = i0 + 1;
    for (int m = i1; m > i0;) {
      const int T = block_steps(m - i0);
      b.m_hi = m;
      b.T = T;
      b.out_last = free_state(pool, b.cur, b.prev, nullptr);
      b.out_before = T > 1 ? free_state(pool, b.cur, b.prev, b.out_last) : nullptr;
      if (ip != nullptr) b.inst.ntiles = ip->adj_tiles(m - T + 1);
      ERNN_CUDA(runner.add(b));
      b.prev = T > 1 ? b.out_before : b.cur;
      b.cur = b.out_last;
      m -= T;
    }
    ERNN_CUDA(runner.flush());
  }
  return ERNN_OK;
}

}  // namespace

void record_last_path(int32_t path) { g_last_path.store(path, std::memory_order_relaxed); }

}  // namespace ernn

using namespace ernn;

extern "C" {

int ernn_abi_version(void) { return ERNN_ABI_VERSION; }

const char* ernn_error_string(int code) {
  switch (code) {
    case ERNN_OK: return "ok";
    case ERNN_ERR_INVALID: return "invalid argument (null pointer, size or enum out of range)";
    case ERNN_ERR_WORKSPACE: return "workspace smaller than the size query returned";
    case ERNN_ERR_CUDA: return "CUDA runtime call failed";
    case ERNN_ERR_UNSTABLE: return "leapfrog stability bound violated for these constants";
    case ERNN_ERR_TIMEOUT: return "bounded device-side wait timed out";
    case ERNN_ERR_UNSUPPORTED: return "request not supported by this library";
    default: return "unknown error code";
  }
}

int ernn_validate(const ErnnProblem* p) { return validate(p); }

size_t ernn_tape_bytes(const ErnnProblem* p, int with_tape) {
  if (validate(p) != ERNN_OK) return 0;
  const Plan pl = make_plan(*p);
  return with_tape ? pl.t_total_tape : pl.t_total_notape;
}

size_t ernn_adjoint_scratch_bytes(const ErnnProblem* p) {
  if (validate(p) != ERNN_OK) return 0;
  return make_plan(*p).s_total;
}

int ernn_check_stability(const double* C, double rho, double h, double dt, double* courant) {
  if (C == nullptr || !(rho > 0.0) || !(h > 0.0) || !(dt > 0.0)) return ERNN_ERR_INVALID;
  // Symbol of -(h^2) A on the Fourier mode exp(i(tx*i + ty*j)):
  //   a = 4 sin^2(tx/2), b = 4 sin^2(ty/2), d = sin(tx) sin(ty)
  //   Mxx = C11 a + C66 b + 2 C16 d,  Myy = C66 a + C22 b + 2 C26 d,
  //   Mxy = C16 a + C26 b + (C12 + C66) d.
  // Leapfrog is stable when every eigenvalue of (dt^2 / (rho h^2)) M lies in [0, 4].
  const double q = dt * dt / (rho * h * h);
  const int n = 128;
  double worst = 0.0;
  bool indefinite = false;
  for (int u = 0; u <= n; ++u) {
    for (int v = 0; v <= n; ++v) {
      const double tx = kPi * u / n, ty = kPi * v / n;
      const double a = 4.0 * std::sin(tx / 2) * std::sin(tx / 2);
      const double b = 4.0 * std::sin(ty / 2) * std::sin(ty / 2);
      for (int sgn = -1; sgn <= 1; sgn += 2) {
        const double d = sgn * std::sin(tx) * std::sin(ty);
        const double mxx = C[0] * a + C[5] * b + 2 * C[3] * d;
        const double myy = C[5] * a + C[1] * b + 2 * C[4] * d;
        const double mxy = C[3] * a + C[4] * b + (C[2] + C[5]) * d;
        const double tr = mxx + myy, det = mxx * myy - mxy * mxy;
        const double disc = std::sqrt(std::fmax(tr * tr / 4 - det, 0.0));
        const double lmax = tr / 2 + disc, lmin = tr / 2 - disc;
        if (lmin < -1e-9 * std::fabs(lmax)) indefinite = true;
        if (q * lmax / 4.0 > worst) worst = q * lmax / 4.0;
      }
    }
  }
  if (courant) *courant = worst;
  return (worst > 1.0 || indefinite) ? ERNN_ERR_UNSTABLE : ERNN_OK;
}

int ernn_operator(int32_t nshots, int32_t nx, int32_t ny, int32_t mode, double h, const float* C,
                  const float* D, const float* rho, const float* ux, const float* uy,
                  const float* fx, const float* fy, float* Lux, float* Luy, void* stream) {
  if (nshots < 1 || nx < 1 || ny < 1 || mode < 0 || mode > 2 || !(h > 0.0)) return ERNN_ERR_INVALID;
  if (C == nullptr || rho == nullptr || ux == nullptr || uy == nullptr || Lux == nullptr ||
      Luy == nullptr || (mode == kModeDField && D == nullptr))
    return ERNN_ERR_INVALID;
  ERNN_CUDA(launch_operator(nshots, nx, ny, mode, h, C, D, rho, ux, uy, fx, fy, Lux, Luy,
                            (cudaStream_t)stream));
  return ERNN_OK;
}

// The forward time loop of ernn_forward and, with an instance plan `ip`, of
// ernn_forward_instances.
static int forward_impl(const ErnnProblem* p, const ErnnInputs* in, const InstPlan* ip, float* out_ux,
                        float* out_uy, void* tape, size_t tape_bytes, int with_tape, void* stream) {
  int rc = validate(p);
  if (rc) return rc;
  if ((rc = validate_inputs(p, in))) return rc;
  if (out_ux == nullptr || out_uy == nullptr || tape == nullptr) return ERNN_ERR_INVALID;
  if ((ip != nullptr) != ((p->flags & ERNN_FLAG_INSTANCES) != 0)) return ERNN_ERR_INVALID;
  const Plan pl = make_plan(*p);
  if (tape_bytes < (with_tape ? pl.t_total_tape : pl.t_total_notape)) return ERNN_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  Coef* coef = reinterpret_cast<Coef*>(at(tape, pl.t_coef));
  ERNN_CUDA(launch_coef(p->mode, in->C, in->rho, p->h, p->dt, coef, st, pl.ncoef));

  InstTiles itab{nullptr, nullptr, 0};
  const bool block = pl.block && al16(tape) && blk_available() &&
                     (with_tape != 0 || p->mode != kModeFields || per_cell_tiles(*p, Pass::kForward));
  if (ip != nullptr) {
    // instances: the time-blocked kernels over the tile table only, which
    // read and write a state inside the instances' regions alone; trace
    // frames past an instance's steps are zero
    if (p->path != ERNN_PATH_AUTO && p->path != ERNN_PATH_TILED) return ERNN_ERR_UNSUPPORTED;
    if (p->ny % 4 != 0) return ERNN_ERR_UNSUPPORTED;
    if (!block) return blk_available() ? ERNN_ERR_CUDA : ERNN_ERR_UNSUPPORTED;
    itab.tiles = reinterpret_cast<int4*>(at(tape, pl.t_inst));
    itab.box = reinterpret_cast<int4*>(at(tape, pl.t_inst + align_up(inst_table_bound(p->nx, p->ny, p->nshots) *
                                                                       sizeof(int4))));
    ERNN_CUDA(launch_inst_table(ip->d, const_cast<int4*>(itab.tiles), const_cast<int4*>(itab.box), st));
    const size_t tr_bytes = (size_t)p->nshots * pl.nt_out * p->nrec * sizeof(float);
    ERNN_CUDA(cudaMemsetAsync(out_ux, 0, tr_bytes, st));
    ERNN_CUDA(cudaMemsetAsync(out_uy, 0, tr_bytes, st));
  }

  if (ip == nullptr && (p->path == ERNN_PATH_AUTO || p->path == ERNN_PATH_RESIDENT)) {
    ResCommon res;
    if (pick_resident(*p, *in, coef, res)) {
      g_last_path.store(ERNN_PATH_RESIDENT, std::memory_order_relaxed);
      return resident_forward(*p, pl, res, out_ux, out_uy, tape, with_tape, st);
    }
    if (p->path == ERNN_PATH_RESIDENT) return ERNN_ERR_UNSUPPORTED;
  }
  if (block) {
    g_last_path.store(ERNN_PATH_TILED, std::memory_order_relaxed);
    return block_forward(*p, pl, *in, ip, itab, coef, out_ux, out_uy, tape, with_tape, st);
  }
  int tiled = 0;
  if ((rc = use_tiled(*p, &tiled))) return rc;
  g_last_path.store(tiled ? ERNN_PATH_TILED : ERNN_PATH_STEP, std::memory_order_relaxed);
  auto fwd_step = [&](const FwdStep& s) {
    return tiled ? launch_tma_fwd(s, &coef->err, st) : launch_fwd_step(p->mode, s, st);
  };

  const bool store_all = with_tape && pl.store_all;
  float* A = fat(tape, pl.t_A);
  float* B = fat(tape, pl.t_B);
  auto stored = [&](int n) { return fat(tape, pl.t_store + (size_t)(n - 1) * pl.state_bytes); };
  auto ck = [&](int j, int lev) {  // checkpoint j >= 1: lev 0 = u^{jk}, lev 1 = u^{jk-1}
    return fat(tape, pl.t_store + ((size_t)(j - 1) * 2 + lev) * pl.state_bytes);
  };
  const bool receivers = (p->record == kRecordReceivers);
  FwdStep a = base_fwd(*p, *in, coef, pl.nt_out);
  const float* last = nullptr;
  for (int i = 0; i < p->nt; ++i) {
    if (store_all) {
      a.out = stored(i + 1);
      a.cur = i >= 1 ? stored(i) : nullptr;
      a.prev = i >= 2 ? stored(i - 1) : nullptr;
    } else {
      a.out = (i % 2 == 0) ? A : B;
      a.cur = i == 0 ? nullptr : ((i % 2 == 0) ? B : A);
      a.prev = i <= 1 ? nullptr : a.out;
    }
    a.i = i;
    a.copy0 = a.copy1 = nullptr;
    if (with_tape && !pl.store_all) {
      if ((i + 1) % pl.k == 0 && (i + 1) / pl.k <= pl.nseg - 1) a.copy0 = ck((i + 1) / pl.k, 0);
      if ((i + 2) % pl.k == 0 && (i + 2) / pl.k <= pl.nseg - 1) a.copy1 = ck((i + 2) / pl.k, 1);
    }
    a.frame = -1;
    a.gframe = -1;
    if (!receivers) {
      if (i % p->stride == 0) { a.frame = i / p->stride; a.hist_x = out_ux; a.hist_y = out_uy; }
    } else if (i >= 1 && (i - 1) % p->stride == 0) {
      a.gframe = (i - 1) / p->stride; a.tr_x = out_ux; a.tr_y = out_uy;
    }
    a.chained = i > 0;  // step 0 follows the coefficient kernel
    ERNN_CUDA(fwd_step(a));
    last = a.out;
  }
  if (receivers && (p->nt - 1) % p->stride == 0) {
    ERNN_CUDA(launch_gather(last, p->nx, p->ny, p->nshots, in->rec_idx, p->nrec,
                            (p->nt - 1) / p->stride, pl.nt_out, out_ux, out_uy, st));
  }
  return ERNN_OK;
}

int ernn_forward(const ErnnProblem* p, const ErnnInputs* in, float* out_ux, float* out_uy,
                 void* tape, size_t tape_bytes, int with_tape, void* stream) {
  return forward_impl(p, in, nullptr, out_ux, out_uy, tape, tape_bytes, with_tape, stream);
}

int ernn_forward_instances(const ErnnProblem* p, const ErnnInputs* in, const ErnnInstances* inst,
                           float* out_ux, float* out_uy, void* tape, size_t tape_bytes, int with_tape,
                           void* stream) {
  int rc = validate(p);
  if (rc) return rc;
  InstPlan ip;
  if ((rc = plan_instances(*p, inst, &ip))) return rc;
  return forward_impl(p, in, &ip, out_ux, out_uy, tape, tape_bytes, with_tape, stream);
}

// The adjoint of ernn_adjoint and, with an instance plan `ip`, of
// ernn_adjoint_instances.
static int adjoint_impl(const ErnnProblem* p, const ErnnInputs* in, const InstPlan* ip, const float* g_ux,
                        const float* g_uy, const void* tape_c, size_t tape_bytes, void* scratch,
                        size_t scratch_bytes, double* grad_C, float* grad_field, void* stream) {
  int rc = validate(p);
  if (rc) return rc;
  if ((rc = validate_inputs(p, in))) return rc;
  if ((ip != nullptr) != ((p->flags & ERNN_FLAG_INSTANCES) != 0)) return ERNN_ERR_INVALID;
  if (g_ux == nullptr || g_uy == nullptr || tape_c == nullptr || scratch == nullptr)
    return ERNN_ERR_INVALID;
  if (p->mode == kModeScalar && grad_C == nullptr) return ERNN_ERR_INVALID;
  if (p->mode != kModeScalar && grad_field == nullptr) return ERNN_ERR_INVALID;
  const Plan pl = make_plan(*p);
  if (tape_bytes < pl.t_total_tape || scratch_bytes < pl.s_total) return ERNN_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  void* tape = const_cast<void*>(tape_c);  // read only below
  scratch = scratch_base(pl, scratch);
  const bool block = pl.block && al16(tape) && blk_available();

  Coef* coef = reinterpret_cast<Coef*>(at(scratch, pl.s_coef));
  ERNN_CUDA(launch_coef(p->mode, in->C, in->rho, p->h, p->dt, coef, st, pl.ncoef));
  const size_t gcount = (size_t)p->nshots * pl.nt_out *
                        (p->record == kRecordFields ? pl.N : (size_t)p->nrec);
  ERNN_CUDA(launch_gscale(g_ux, g_uy, gcount, coef, st, pl.ncoef));
  float* LA = fat(scratch, pl.s_LA);
  float* LB = fat(scratch, pl.s_LB);
  if (!block) ERNN_CUDA(cudaMemsetAsync(LA, 0, 2 * pl.state_bytes, st));  // LA and LB are adjacent
  float* gacc = fat(scratch, pl.s_gacc);
  double* partials = reinterpret_cast<double*>(at(scratch, pl.s_part));
  if (p->mode != kModeScalar) ERNN_CUDA(cudaMemsetAsync(gacc, 0, pl.s_part - pl.s_gacc, st));
  else ERNN_CUDA(cudaMemsetAsync(partials, 0, pl.s_tflags - pl.s_part, st));

  InstTiles itab{nullptr, nullptr, 0};
  if (ip != nullptr) {
    if (p->path != ERNN_PATH_AUTO && p->path != ERNN_PATH_TILED) return ERNN_ERR_UNSUPPORTED;
    if (p->ny % 4 != 0) return ERNN_ERR_UNSUPPORTED;
    if (!block) return blk_available() ? ERNN_ERR_CUDA : ERNN_ERR_UNSUPPORTED;
    itab.tiles = reinterpret_cast<int4*>(at(scratch, pl.s_inst));
    itab.box = reinterpret_cast<int4*>(at(scratch, pl.s_inst + align_up(inst_table_bound(p->nx, p->ny, p->nshots) *
                                                                          sizeof(int4))));
    ERNN_CUDA(launch_inst_table(ip->d, const_cast<int4*>(itab.tiles), const_cast<int4*>(itab.box), st));
  }

  if (ip == nullptr && (p->path == ERNN_PATH_AUTO || p->path == ERNN_PATH_RESIDENT)) {
    ResCommon res;
    if (pick_resident(*p, *in, coef, res)) {
      g_last_path.store(ERNN_PATH_RESIDENT, std::memory_order_relaxed);
      int img_rows = 0;
      if ((rc = resident_adjoint(*p, pl, res, g_ux, g_uy, tape, scratch, partials, &img_rows, st)))
        return rc;
      // imaging rows are grouped by shot
      if (pl.ncoef > 1) ERNN_CUDA(launch_finalize_scalar(partials, img_rows / p->nshots, coef, grad_C, st,
                                                         p->nshots, 1));
      else ERNN_CUDA(launch_finalize_scalar(partials, img_rows, coef, grad_C, st));
      return ERNN_OK;
    }
    if (p->path == ERNN_PATH_RESIDENT) return ERNN_ERR_UNSUPPORTED;
  }
  if (block) {
    g_last_path.store(ERNN_PATH_TILED, std::memory_order_relaxed);
    if ((rc = block_adjoint(*p, pl, *in, ip, itab, coef, g_ux, g_uy, tape, scratch, partials, st))) return rc;
    if (p->mode != kModeScalar) {
      ERNN_CUDA(launch_finalize_fields(p->mode, gacc, p->nshots, (int)pl.N, coef, grad_field, st));
      return ERNN_OK;
    }
    if (pl.ncoef > 1)
      ERNN_CUDA(launch_finalize_scalar(partials, kTiledRowsPerShot, coef, grad_C, st, p->nshots, 1));
    else
      ERNN_CUDA(launch_finalize_scalar(partials, pl.npart, coef, grad_C, st));
    return ERNN_OK;
  }
  int tiled = 0;
  if ((rc = use_tiled(*p, &tiled))) return rc;
  g_last_path.store(tiled ? ERNN_PATH_TILED : ERNN_PATH_STEP, std::memory_order_relaxed);

  auto stored = [&](int n) { return fat(tape, pl.t_store + (size_t)(n - 1) * pl.state_bytes); };
  auto ck = [&](int j, int lev) -> const float* {
    if (j == 0) return nullptr;
    if (lev == 1 && j * pl.k - 1 == 0) return nullptr;  // u^0 = 0 (k == 1)
    return fat(tape, pl.t_store + ((size_t)(j - 1) * 2 + lev) * pl.state_bytes);
  };
  auto seg = [&](int slot) { return fat(scratch, pl.s_seg + (size_t)slot * pl.state_bytes); };

  AdjStep b;
  std::memset(&b, 0, sizeof(b));
  b.nx = p->nx; b.ny = p->ny; b.S = p->nshots;
  b.coef = coef;
  b.field = (p->mode == kModeFields) ? in->C : in->D;
  b.g_x = g_ux; b.g_y = g_uy;
  b.nt_out = pl.nt_out; b.record = p->record; b.nrec = p->nrec; b.rec_idx = in->rec_idx;
  b.coef_stride = pl.ncoef > 1 ? 1 : 0;
  b.partials = partials;
  b.gacc = gacc;
  b.tile_flags = nullptr;
  if (tiled && p->record == kRecordReceivers) {
    uint8_t* flags = reinterpret_cast<uint8_t*>(at(scratch, pl.s_tflags));
    ERNN_CUDA(launch_tile_flags(in->rec_idx, p->nshots, p->nrec, p->nx, p->ny, flags, st));
    b.tile_flags = flags;
  }

  // every step launch after the first of the loop below follows a step kernel
  bool chained = false;
  auto adj_step = [&](int m, const float* um) -> int {
    const int idx = p->nt - m;
    b.m = m;
    b.out = (idx % 2 == 0) ? LA : LB;
    b.cur = (idx % 2 == 0) ? LB : LA;
    b.prev = b.out;
    b.u = (m <= p->nt - 1) ? um : nullptr;
    b.frame = ((m - 1) % p->stride == 0) ? (m - 1) / p->stride : -1;
    b.chained = chained ? 1 : 0;
    chained = true;
    const cudaError_t e = tiled ? launch_tma_adj(b, &coef->err, st) : launch_adj_step(p->mode, b, st);
    return e == cudaSuccess ? ERNN_OK : ERNN_ERR_CUDA;
  };

  if (pl.store_all) {
    for (int m = p->nt; m >= 1; --m)
      if ((rc = adj_step(m, stored(m)))) return rc;
  } else {
    FwdStep a = base_fwd(*p, *in, coef, pl.nt_out);
    for (int j = pl.nseg - 1; j >= 0; --j) {
      const int i0 = j * pl.k, i1 = (j + 1) * pl.k < p->nt ? (j + 1) * pl.k : p->nt;
      // recompute u^{i0+1} .. u^{i1} into the segment buffer; u^{nt} is never
      // imaged, so the last segment stops one step short
      const int iend = i1 < p->nt ? i1 : p->nt - 1;
      for (int i = i0; i < iend; ++i) {
        a.i = i;
        a.out = seg(i - i0);
        a.cur = (i == i0) ? ck(j, 0) : seg(i - i0 - 1);
        a.prev = (i == i0) ? ck(j, 1) : (i == i0 + 1 ? ck(j, 0) : seg(i - i0 - 2));
        a.chained = chained ? 1 : 0;
        chained = true;
        ERNN_CUDA(tiled ? launch_tma_fwd(a, &coef->err, st) : launch_fwd_step(p->mode, a, st));
      }
      for (int m = i1; m >= i0 + 1; --m)
        if ((rc = adj_step(m, seg(m - 1 - i0)))) return rc;
    }
  }
  if (p->mode == kModeScalar && pl.ncoef > 1) {
    // per-shot gradients: one row per block, blocks of a shot contiguous
    ERNN_CUDA(launch_finalize_scalar(partials, pl.nblocks / p->nshots, coef, grad_C, st, p->nshots, 1));
  } else if (p->mode == kModeScalar) {
    ERNN_CUDA(launch_finalize_scalar(partials, pl.nblocks, coef, grad_C, st));
  } else {
    ERNN_CUDA(launch_finalize_fields(p->mode, gacc, p->nshots, (int)pl.N, coef, grad_field, st));
  }
  return ERNN_OK;
}

int ernn_adjoint(const ErnnProblem* p, const ErnnInputs* in, const float* g_ux,
                 const float* g_uy, const void* tape_c, size_t tape_bytes, void* scratch,
                 size_t scratch_bytes, double* grad_C, float* grad_field, void* stream) {
  return adjoint_impl(p, in, nullptr, g_ux, g_uy, tape_c, tape_bytes, scratch, scratch_bytes, grad_C,
                      grad_field, stream);
}

int ernn_adjoint_instances(const ErnnProblem* p, const ErnnInputs* in, const ErnnInstances* inst,
                           const float* g_ux, const float* g_uy, const void* tape, size_t tape_bytes,
                           void* scratch, size_t scratch_bytes, double* grad_C, void* stream) {
  int rc = validate(p);
  if (rc) return rc;
  InstPlan ip;
  if ((rc = plan_instances(*p, inst, &ip))) return rc;
  return adjoint_impl(p, in, &ip, g_ux, g_uy, tape, tape_bytes, scratch, scratch_bytes, grad_C, nullptr,
                      stream);
}

uint64_t ernn_launch_count(void) { return launches(); }

int ernn_device_status(const ErnnProblem* p, const void* workspace, int is_scratch,
                       int32_t* status_host, void* stream) {
  int rc = validate(p);
  if (rc) return rc;
  if (workspace == nullptr || status_host == nullptr || (is_scratch != 0 && is_scratch != 1))
    return ERNN_ERR_INVALID;
  const Plan pl = make_plan(*p);
  const void* base = is_scratch ? scratch_base(pl, const_cast<void*>(workspace)) : workspace;
  const char* w = static_cast<const char*>(base) + (is_scratch ? pl.s_coef : pl.t_coef) + offsetof(Coef, err);
  ERNN_CUDA(cudaMemcpyAsync(status_host, w, sizeof(int32_t), cudaMemcpyDeviceToHost,
                            (cudaStream_t)stream));
  return ERNN_OK;
}

int ernn_wait_selftest(int32_t* status_host, void* stream) {
  if (status_host == nullptr) return ERNN_ERR_INVALID;
  int v = -1;
  ERNN_CUDA(wait_selftest(&v, (cudaStream_t)stream));
  *status_host = v;
  return ERNN_OK;
}

int32_t ernn_last_path(void) { return g_last_path.load(std::memory_order_relaxed); }

int ernn_set_launch_overlap(int on) {
  const int was = launch_overlap_setting() ? 1 : 0;
  set_launch_overlap(on != 0);
  return was;
}

int ernn_profile_enable(int enable) {
  profile_enable(enable != 0);
  return ERNN_OK;
}

int ernn_profile_read(double* ms3, uint64_t* launches3, double* alg_bytes3) {
  if (ms3 == nullptr || launches3 == nullptr) return ERNN_ERR_INVALID;
  return profile_read(ms3, launches3, alg_bytes3) == cudaSuccess ? ERNN_OK : ERNN_ERR_CUDA;
}

}  // extern "C"
