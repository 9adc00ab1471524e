// Time-blocked tile kernels (ernn_block.cu): up to four time steps per launch.
// Internal to the library.
#pragma once

#include "ernn_launch.h"
#include "ernn_tma.h"

namespace ernn {

constexpr int kBlkSteps = 4;       // most time steps of one launch (and halo rows / columns of a tile)
constexpr int kBlkCols = 120;      // columns of a tile (a warp's 128 less one quad each side)

// Instances on one canvas (ERNN_FLAG_INSTANCES): the kernels walk a tile
// table instead of the grid's tiling.  Entry t of the table is one tile's
// instance, origin and instance region (16-bit pairs); per instance k, box[2k] =
// (x0, y0, x1, y1) of its region and box[2k + 1] = (first table entry of its
// tiles, tiles per tile row, steps, 0).
struct InstTiles {
  const int4* tiles;   // the table, instances ordered by decreasing step count
  const int4* box;     // per instance (region, tiling and step count)
  int ntiles;          // entries of this launch: the prefix of running instances
};

// Forward: u^{i+1} .. u^{i+T} from (u^i, u^{i-1}).
struct BlkFwd {
  int geo;                         // tile geometry (blk_geometry)
  int plain_order;                 // SCALAR: rounding order of the plain kernels (oper), else the tiled ones'
  int nx, ny, pitch, S, nt, i, T;  // pitch: floats between rows of a state (ny rounded up to 4)
  const float* cur;                // u^i, nullptr: zero
  const float* prev;               // u^{i-1}, nullptr: zero
  float* out[kBlkSteps + 1];       // where u^{i+t} goes (t = 0: a copy of u^i), or nullptr
  // dense history or receiver traces: frame of u^{i+t} in frame[t], or -1
  float* rec_x;
  float* rec_y;
  int frame[kBlkSteps + 1];
  int nt_out, record, nrec;
  int vec;                         // dense history rows start on 16-byte boundaries
  const int2* rec_tile;            // receivers of every tile (launch_rec_tiles), or nullptr
  const int2* rec_ent;
  const Coef* coef;
  int coef_stride;
  const float* field;              // FIELDS: 6 planes of C; DFIELD: D plane (rows of ny floats)
  int vec_field;                   // the plane's rows start on 16-byte boundaries
  const float* src_signal;
  const float* src_map;
  const int32_t* src_origin;
  int bx, by, src_comp;
  int chained;
  InstTiles inst;
};

// Adjoint: lam^m, m = m_hi down to m_hi - T + 1, from (lam^{m_hi+1},
// lam^{m_hi+2}), and the imaging sums of the pairs (lam^{m+1}, u^m).
struct BlkAdj {
  int geo;
  int plain_order;      // as in BlkFwd
  int nx, ny, pitch, S, nt, m_hi, T;
  const float* cur;     // lam^{m_hi+1}, nullptr: zero
  const float* prev;    // lam^{m_hi+2}, nullptr: zero
  float* out_last;      // lam^{m_hi-T+1}
  float* out_before;    // lam^{m_hi-T+2} (T >= 2)
  // u^m = u_base + (m - m_base) u_stride floats; the pair of m == nt vanishes
  const float* u_base;
  size_t u_stride;
  int m_base;
  const float* g_x;
  const float* g_y;
  int stride, nt_out, record, nrec;
  const int2* rec_tile;
  const int2* rec_ent;
  const Coef* coef;
  int coef_stride;
  const float* field;   // as in BlkFwd (vec_field: gacc's rows too)
  int vec_field;
  float* gacc;          // DFIELD: [S][N]; FIELDS: [S][6][N] running sums
  double* partials;     // SCALAR
  int chained;
  InstTiles inst;
};

// A run: several passes (launches' worth of steps) in one cooperative launch,
// each over the state the one before left.  24 passes take 140 to 270 us, of
// which the launch is 3 to 4 (and their arguments 2 KB).
constexpr int kRunPasses = 24;
struct FwdPass {
  int i, T;
  const float* cur;
  const float* prev;
  float* out[kBlkSteps + 1];
  int frame[kBlkSteps + 1];
};
struct AdjPass {
  int m_hi, T;
  const float* cur;
  const float* prev;
  float* out_last;
  float* out_before;
};
struct FwdRun {
  int n, epoch;  // passes; passes that the flags have counted before
  int* flags;    // one per tile
  FwdPass p[kRunPasses];
};
struct AdjRun {
  int n, epoch;
  int* flags;
  AdjPass p[kRunPasses];
};
bool blk_run_fits(int mode, int geo, int nx, int ny, int S);
cudaError_t launch_blk_fwd_run(int mode, const BlkFwd& a, const FwdRun& r, int* err, cudaStream_t st);
cudaError_t launch_blk_adj_run(int mode, const BlkAdj& a, const AdjRun& r, int* err, cudaStream_t st);

// Tile geometry of a grid problem (instances: kBlkTall or kBlkRow64), tiles of
// an nx x ny grid.
constexpr int kBlkTall = 0, kBlkShort = 1, kBlkFlat = 2, kBlkTall5 = 3, kBlkTall4 = 4, kBlkRow128 = 5, kBlkRow64 = 6;
struct BlkShape {
  int rows, cols;  // that a tile stores
  int hy;          // halo columns on either side; 0: the tile holds whole rows
};
BlkShape blk_shape(int geo);
int blk_geometry(int mode, int nx, int ny, int S);
double blk_cost(int geo, int nx, int ny, int S);  // us of a launch of four steps (scalar constants)
size_t blk_tiles(int geo, int nx, int ny);
// Partial-sum rows reserved per shot with per-shot constants (an adjoint grid
// never exceeds this many CTAs).
constexpr int kTiledRowsPerShot = 1024;
// Instances on a canvas (ERNN_FLAG_INSTANCES), passed by value to the kernel
// that writes the tile table: in the order of decreasing step count, each
// with its caller-side index.
constexpr int kMaxInstances = 256;
struct InstDesc {
  int count, tile_rows, tile_cols;
  int id[kMaxInstances], x0[kMaxInstances], y0[kMaxInstances], nx[kMaxInstances];
  int ny[kMaxInstances], nt[kMaxInstances], base[kMaxInstances];
};
// Writes the tile table (in the order of d) and the per-instance boxes
// (2 x S int4) described in InstTiles.
cudaError_t launch_inst_table(const InstDesc& d, int4* tiles, int4* box, cudaStream_t st);
// Receivers of the tiles of a call: room for `ntiles` tiles, and the table
// (box: instances, else nullptr).  The traces of receivers outside the grid
// (tr_x, tr_y; nullptr: not recorded here) become zeros.
size_t blk_rec_bytes(size_t ntiles, int S, int nrec);
cudaError_t launch_rec_tiles(int geo, const int32_t* rec_idx, int S, int nrec, int nx, int ny, const int4* box,
                             size_t ntiles, void* ws, const int2** tile, const int2** ent, float* tr_x, float* tr_y,
                             int nt_out, cudaStream_t st);
bool blk_available();  // the driver exposes the tensor-map encoder
cudaError_t launch_blk_fwd(int mode, const BlkFwd& a, int* err, cudaStream_t st);
cudaError_t launch_blk_adj(int mode, const BlkAdj& a, int* err, cudaStream_t st);

}  // namespace ernn
