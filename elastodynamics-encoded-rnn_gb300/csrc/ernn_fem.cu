// FEM data generator step (sm_103a): the explicit time loop that produces
// the reference's training wavefields (Parameter_inversion/FEM_generate_data.py:
// mesh :117-185, lumped mass :330-342, element operator :345-457, central
// differences with fixed edges :474-499, 0.7-scaled frames :525-526, 901-930).
//
// The mesh is the structured triangular one of the generator: nodes on an
// nx x ny grid, each cell split along the diagonal n0-n2 when (ci + cj) is
// even and along n1-n3 when odd.  Its elements therefore come in four shapes
// with constant strain (one B matrix per shape), and every interior node
// sees the same 8 (node parity even) or 4 (odd) triangles.  Instead of
// gathering elements and scattering forces with atomics, one thread per node
// gathers the strains of its adjacent triangles from the 3 x 3 neighbourhood
// of displacements, forms their stresses and sums the node's share of each
// element force: one pass per step reading u^n (neighbourhood), u^{n-1}, the
// load, writing u^{n+1} and, on recording steps, the scaled frame.
// Edge nodes are fixed at zero (their forces are never needed).
//
// State layout: [i][j] with j (y) fastest, the layout of the saved frames
// (nt_out, nx, ny); node (i, j) is the generator's node j*nx + i.
#include <cmath>
#include <cstdint>
#include <cstring>

#include "ernn.h"
#include "ernn_launch.h"

namespace ernn {
namespace {

// Element shapes: 0 = even cell [n0, n1, n2], 1 = even [n0, n2, n3],
// 2 = odd [n0, n1, n3], 3 = odd [n1, n2, n3]; corners n0 = (0, 0),
// n1 = (1, 0), n2 = (1, 1), n3 = (0, 1) in (i, j) offsets within the cell.
struct FemConsts {
  float bx[4][3], by[4][3];  // dN/dx, dN/dy of the three nodes of each shape
  float fh;                  // |det J| x (3 Gauss points x weight 1/6)
  float C11, C22, C12, C16, C26, C66;
  float m_even, m_odd;       // lumped mass of interior nodes (8 or 4 triangles)
  float dt2, rho_inv, scale;
};

struct FemStep {
  int nx, ny, n;
  const float* cur_x; const float* cur_y;
  const float* prev_x; const float* prev_y;
  float* out_x; float* out_y;
  const float* load;    // (nx, ny)
  const float* signal;  // (nt)
  const float* cf;      // per-node constants, 6 planes (nx, ny), or nullptr
  float* frame_x;       // (nx, ny) slice of the frames, or nullptr
  float* frame_y;
};

// Contribution of one triangle of shape T, in the cell whose corner (0, 0)
// sits at offset (oi, oj) from the node, to the node's force; the node is
// the triangle's vertex `a`.  u[1 + di][1 + dj] is the neighbourhood.
// FIELDS: the element's constants are those of the grid node nearest its
// centroid (Damage_inversion/FEM_generate_data.py:1002-1017): centroids sit
// at (2/3, 1/3), (1/3, 2/3), (1/3, 1/3), (2/3, 2/3) of the cell for shapes
// 0..3, so that node is the cell corner (1, 0), (0, 1), (0, 0), (1, 1).
template <bool FIELDS, int T, int OI, int OJ, int A>
__device__ __forceinline__ void tri(const FemConsts& k, const FemStep& s, size_t o,
                                    const float ux[3][3], const float uy[3][3], float& fx, float& fy) {
  constexpr int vi[4][3] = {{0, 1, 1}, {0, 1, 0}, {0, 1, 0}, {1, 1, 0}};
  constexpr int vj[4][3] = {{0, 0, 1}, {0, 1, 1}, {0, 0, 1}, {0, 1, 1}};
  constexpr int ci[4] = {1, 0, 0, 1}, cj[4] = {0, 1, 0, 1};
  float C11 = k.C11, C22 = k.C22, C12 = k.C12, C16 = k.C16, C26 = k.C26, C66 = k.C66;
  if (FIELDS) {
    const size_t N = (size_t)s.nx * s.ny;
    const size_t e = o + (size_t)((OI + ci[T]) * s.ny + (OJ + cj[T]));
    C11 = __ldg(s.cf + e);
    C22 = __ldg(s.cf + N + e);
    C12 = __ldg(s.cf + 2 * N + e);
    C16 = __ldg(s.cf + 3 * N + e);
    C26 = __ldg(s.cf + 4 * N + e);
    C66 = __ldg(s.cf + 5 * N + e);
  }
  float exx = 0.f, eyy = 0.f, gxy = 0.f;
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    const float vx = ux[1 + OI + vi[T][b]][1 + OJ + vj[T][b]];
    const float vy = uy[1 + OI + vi[T][b]][1 + OJ + vj[T][b]];
    exx += k.bx[T][b] * vx;
    eyy += k.by[T][b] * vy;
    gxy += k.by[T][b] * vx + k.bx[T][b] * vy;
  }
  const float sxx = C11 * exx + C12 * eyy + C16 * gxy;
  const float syy = C12 * exx + C22 * eyy + C26 * gxy;
  const float txy = C16 * exx + C26 * eyy + C66 * gxy;
  fx += k.fh * (k.bx[T][A] * sxx + k.by[T][A] * txy);
  fy += k.fh * (k.by[T][A] * syy + k.bx[T][A] * txy);
}

template <bool FIELDS>
__global__ void __launch_bounds__(256) fem_step_kernel(const FemStep s, const FemConsts k) {
  grid_dep_trigger();
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= s.nx || j >= s.ny) return;
  const int ny = s.ny;
  const size_t o = (size_t)i * ny + j;
  const bool interior = i > 0 && i < s.nx - 1 && j > 0 && j < ny - 1;
  // the load term needs no state: formed before the wait
  const float lf = interior ? s.signal[s.n] * s.load[o] * k.rho_inv : 0.f;
  grid_dep_wait();  // levels of the previous launch complete from here on
  float vx = 0.f, vy = 0.f;
  if (interior) {
    float ux[3][3], uy[3][3];
#pragma unroll
    for (int di = 0; di < 3; ++di)
#pragma unroll
      for (int dj = 0; dj < 3; ++dj) {
        const size_t q = o + (size_t)(di - 1) * ny + (dj - 1);
        ux[di][dj] = s.cur_x[q];
        uy[di][dj] = s.cur_y[q];
      }
    float fx = 0.f, fy = 0.f;
    float m;
    // cells around the node: A = (i-1, j-1) (node is its n2), B = (i, j-1)
    // (n3), C = (i-1, j) (n1), D = (i, j) (n0); A and D have the node's
    // parity, B and C the other
    if (((i + j) & 1) == 0) {
      tri<FIELDS, 0, -1, -1, 2>(k, s, o, ux, uy, fx, fy);
      tri<FIELDS, 1, -1, -1, 1>(k, s, o, ux, uy, fx, fy);
      tri<FIELDS, 2, 0, -1, 2>(k, s, o, ux, uy, fx, fy);
      tri<FIELDS, 3, 0, -1, 2>(k, s, o, ux, uy, fx, fy);
      tri<FIELDS, 2, -1, 0, 1>(k, s, o, ux, uy, fx, fy);
      tri<FIELDS, 3, -1, 0, 0>(k, s, o, ux, uy, fx, fy);
      tri<FIELDS, 0, 0, 0, 0>(k, s, o, ux, uy, fx, fy);
      tri<FIELDS, 1, 0, 0, 0>(k, s, o, ux, uy, fx, fy);
      m = k.m_even;
    } else {
      tri<FIELDS, 3, -1, -1, 1>(k, s, o, ux, uy, fx, fy);
      tri<FIELDS, 1, 0, -1, 2>(k, s, o, ux, uy, fx, fy);
      tri<FIELDS, 0, -1, 0, 1>(k, s, o, ux, uy, fx, fy);
      tri<FIELDS, 2, 0, 0, 0>(k, s, o, ux, uy, fx, fy);
      m = k.m_odd;
    }
    const float fext = lf * m;
    vx = 2.f * ux[1][1] - s.prev_x[o] - k.dt2 * fx / m;
    vy = 2.f * uy[1][1] - s.prev_y[o] + k.dt2 * (fext - fy) / m;
  }
  s.out_x[o] = vx;
  s.out_y[o] = vy;
  if (s.frame_x != nullptr) {
    s.frame_x[o] = k.scale * vx;
    s.frame_y[o] = k.scale * vy;
  }
}

FemConsts fem_consts(const ErnnFemProblem& p) {
  FemConsts k;
  std::memset(&k, 0, sizeof(k));
  // corner coordinates of the four shapes (units of dx, dy)
  const int vi[4][3] = {{0, 1, 1}, {0, 1, 0}, {0, 1, 0}, {1, 1, 0}};
  const int vj[4][3] = {{0, 0, 1}, {0, 1, 1}, {0, 0, 1}, {0, 1, 1}};
  const double dxi[3] = {-1.0, 1.0, 0.0}, deta[3] = {-1.0, 0.0, 1.0};
  double det = 0.0;
  for (int t = 0; t < 4; ++t) {
    const double J00 = (vi[t][1] - vi[t][0]) * p.dx, J01 = (vi[t][2] - vi[t][0]) * p.dx;
    const double J10 = (vj[t][1] - vj[t][0]) * p.dy, J11 = (vj[t][2] - vj[t][0]) * p.dy;
    det = J00 * J11 - J01 * J10;
    // J^-1, rounded to float as the generator moves it to float32
    const float i00 = (float)(J11 / det), i01 = (float)(-J01 / det);
    const float i10 = (float)(-J10 / det), i11 = (float)(J00 / det);
    for (int a = 0; a < 3; ++a) {
      k.bx[t][a] = i00 * (float)dxi[a] + i10 * (float)deta[a];
      k.by[t][a] = i01 * (float)dxi[a] + i11 * (float)deta[a];
    }
  }
  // every shape has |det J| = dx dy; three Gauss points of weight 1/6
  const float w = (float)(1.0 / 6.0);
  const float f1 = (float)std::fabs(det) * w;
  k.fh = f1 + f1 + f1;
  k.C11 = (float)p.C[0]; k.C22 = (float)p.C[1]; k.C12 = (float)p.C[2];
  k.C16 = (float)p.C[3]; k.C26 = (float)p.C[4]; k.C66 = (float)p.C[5];
  // lumped mass: rho * (dx dy / 2) / 3 added once per adjacent triangle, in float
  const float mnode = (float)(p.rho * (p.dx * p.dy / 2.0) / 3.0);
  float m = 0.f;
  for (int c = 0; c < 8; ++c) {
    m += mnode;
    if (c == 3) k.m_odd = m;
  }
  k.m_even = m;
  k.dt2 = (float)(p.dt * p.dt);
  k.rho_inv = (float)(1.0 / p.rho);
  k.scale = (float)p.out_scale;
  return k;
}

// ------------------------------------------- several levels per launch
// Uniform constants: the force on a node is one linear stencil per node
// parity, sum over its neighbours of K_b (u_b - u), with K summed over the
// node's triangles on the host in double (an odd node's triangles reach its
// four edge neighbours, an even one's all eight; the rows of K sum to zero, so
// the centre enters through the differences).  16 to 32 multiply-adds a node
// instead of 120 to 240 operations and two divisions of the element form, and
// no divergence: a warp holds a row of 128 nodes, a lane four columns, whose
// parities are the same in every lane.  With so little arithmetic a level is
// bound by its launch, so a launch advances a tile up to H levels, the state
// of a thread's nodes in registers, rows exchanged through shared memory (one
// CTA barrier per level), H outer rows and columns of the tile not stored.
// 2001 levels of 301^2 nodes: 10.2 ms with one level a launch, 2.4 ms here
// (4.8 us a launch of four levels; 16 rows with H = 4 against 24 with 8: 2.5
// ms, 24 with 4: 3.7, 14 with 3 and 20 with 4 slower).
//
// The state is u^n and its difference to u^{n-1}, not the two levels: a
// rounding of u then moves u once, where in 2 u^n - u^{n-1} it would enter
// every later level.  Error against 64 bits after 2001 levels: 1e-6 (the one-
// level kernel: 1e-5 on 301^2 nodes, 4e-5 on 61^2).
struct FemStencil {
  float e[8][4];  // even nodes: (-1,-1) (-1,0) (-1,1) (0,-1) (0,1) (1,-1) (1,0) (1,1); xx, xy, yx, yy
  float o[4][4];  // odd nodes: (-1,0) (0,-1) (0,1) (1,0)
  float dt2, rho_inv, scale;
};

struct FemBlock {
  int nx, ny, pitch, n, T;   // levels n + 1 .. n + T from u^n and its difference to u^{n-1}
  const float* cur;          // [2][nx][pitch], nullptr: zero
  const float* diff;         // u^n - u^{n-1}
  float* out;                // u^{n+T} and the difference to the level before it
  float* out_diff;
  const float* load;
  const float* signal;
  float* frames_x;
  float* frames_y;
  int stride;
};

template <int W, int H>
__global__ void __launch_bounds__(32 * W) fem_block_kernel(const FemBlock a, const FemStencil k) {
  constexpr int kCols = 128 - 8 * ((H + 3) / 4), kLeft = 4 * ((H + 3) / 4);  // stored columns, halo columns
  __shared__ float4 ex[2][2][W][32];  // [parity][component][row][quad]
  grid_dep_trigger();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int gi = (int)blockIdx.y * (W - 2 * H) + w - H;
  const int gj = (int)blockIdx.x * kCols - kLeft + 4 * lane;
  const int nx = a.nx, ny = a.ny;
  const size_t N = (size_t)nx * ny, Np = (size_t)nx * a.pitch;
  const bool row_in = gi >= 0 && gi < nx;
  const int nq = row_in && gj >= 0 ? max(0, min(4, ny - gj)) : 0;
  const bool stored = w >= H && w < W - H && 4 * lane >= kLeft && 4 * lane < kLeft + kCols && nq > 0;
  bool inside[4];  // nodes that move: the edges are fixed at zero
  float ld[4], cx[4], cy[4], dx_[4], dy_[4];  // u^n and u^n - u^{n-1}
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    inside[q] = gi > 0 && gi < nx - 1 && gj + q > 0 && gj + q < ny - 1;
    ld[q] = inside[q] ? a.load[(size_t)gi * ny + gj + q] : 0.f;  // (written by no launch: before the wait)
  }
  grid_dep_wait();  // levels of the previous launch complete from here on
  const ptrdiff_t off = (ptrdiff_t)gi * a.pitch + gj;
  auto load_level = [&](const float* s, float(&x)[4], float(&y)[4]) {
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool in = s != nullptr && nq > 0;
    const float4 vx = in ? __ldcg(reinterpret_cast<const float4*>(s + off)) : z;
    const float4 vy = in ? __ldcg(reinterpret_cast<const float4*>(s + off + Np)) : z;
    x[0] = vx.x; x[1] = vx.y; x[2] = vx.z; x[3] = vx.w;
    y[0] = vy.x; y[1] = vy.y; y[2] = vy.z; y[3] = vy.w;
  };
  load_level(a.cur, cx, cy);
  load_level(a.diff, dx_, dy_);
  const bool even_row = (gi & 1) == 0;  // node (gi, gj + q) has the parity of gi + q
  for (int t = 1; t <= a.T; ++t) {
    ex[t & 1][0][w][lane] = make_float4(cx[0], cx[1], cx[2], cx[3]);
    ex[t & 1][1][w][lane] = make_float4(cy[0], cy[1], cy[2], cy[3]);
    __syncthreads();
    if (row_in && w >= t && w < W - t) {
      // windows of rows gi - 1, gi, gi + 1: columns gj - 1 .. gj + 4
      float ux[3][6], uy[3][6];
      auto window = [&](const float4& v, float(&u)[6]) {
        u[0] = __shfl_up_sync(0xffffffffu, v.w, 1);
        u[1] = v.x; u[2] = v.y; u[3] = v.z; u[4] = v.w;
        u[5] = __shfl_down_sync(0xffffffffu, v.x, 1);
      };
      window(ex[t & 1][0][w - 1][lane], ux[0]);
      window(ex[t & 1][1][w - 1][lane], uy[0]);
      window(make_float4(cx[0], cx[1], cx[2], cx[3]), ux[1]);
      window(make_float4(cy[0], cy[1], cy[2], cy[3]), uy[1]);
      window(ex[t & 1][0][w + 1][lane], ux[2]);
      window(ex[t & 1][1][w + 1][lane], uy[2]);
      const int n = a.n + t - 1;  // this level makes u^{n+1}
      const float amp = a.signal[n];
      auto node = [&](int q, bool even) {
        const float x = cx[q], y = cy[q];
        float fx = 0.f, fy = 0.f;
        auto add = [&](const float(&c)[4], int di, int dj) {
          const float dx = ux[1 + di][q + 1 + dj] - x, dy = uy[1 + di][q + 1 + dj] - y;
          fx = fmaf(c[0], dx, fmaf(c[1], dy, fx));
          fy = fmaf(c[2], dx, fmaf(c[3], dy, fy));
        };
        if (even) {
          add(k.e[0], -1, -1); add(k.e[1], -1, 0); add(k.e[2], -1, 1); add(k.e[3], 0, -1);
          add(k.e[4], 0, 1);   add(k.e[5], 1, -1); add(k.e[6], 1, 0);  add(k.e[7], 1, 1);
        } else {
          add(k.o[0], -1, 0); add(k.o[1], 0, -1); add(k.o[2], 0, 1); add(k.o[3], 1, 0);
        }
        const float f = k.dt2 * (amp * ld[q] * k.rho_inv);
        dx_[q] = inside[q] ? dx_[q] - fx : 0.f;
        dy_[q] = inside[q] ? dy_[q] + (f - fy) : 0.f;
      };
      if (even_row) {
        node(0, true); node(1, false); node(2, true); node(3, false);
      } else {
        node(0, false); node(1, true); node(2, false); node(3, true);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        cx[q] += dx_[q];
        cy[q] += dy_[q];
      }
      if (stored && (n + 1) % a.stride == 0) {
        const size_t o = (size_t)((n + 1) / a.stride) * N + (size_t)gi * ny + gj;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (q < nq) {
            a.frames_x[o + q] = k.scale * cx[q];
            a.frames_y[o + q] = k.scale * cy[q];
          }
      }
    }
  }
  if (stored) {
    *reinterpret_cast<float4*>(a.out + off) = make_float4(cx[0], cx[1], cx[2], cx[3]);
    *reinterpret_cast<float4*>(a.out + off + Np) = make_float4(cy[0], cy[1], cy[2], cy[3]);
    *reinterpret_cast<float4*>(a.out_diff + off) = make_float4(dx_[0], dx_[1], dx_[2], dx_[3]);
    *reinterpret_cast<float4*>(a.out_diff + off + Np) = make_float4(dy_[0], dy_[1], dy_[2], dy_[3]);
  }
}

// The stencils of both parities: every triangle adjacent to the node adds
// |J| / 2 (B_a^T C B_b), scaled by dt^2 / m.
FemStencil fem_stencil(const ErnnFemProblem& p) {
  const int vi[4][3] = {{0, 1, 1}, {0, 1, 0}, {0, 1, 0}, {1, 1, 0}};
  const int vj[4][3] = {{0, 0, 1}, {0, 1, 1}, {0, 0, 1}, {0, 1, 1}};
  // (shape, cell offset, vertex) of the triangles around an even and an odd node
  const int even[8][4] = {{0, -1, -1, 2}, {1, -1, -1, 1}, {2, 0, -1, 2}, {3, 0, -1, 2},
                          {2, -1, 0, 1}, {3, -1, 0, 0}, {0, 0, 0, 0}, {1, 0, 0, 0}};
  const int odd[4][4] = {{3, -1, -1, 1}, {1, 0, -1, 2}, {0, -1, 0, 1}, {2, 0, 0, 0}};
  const double* C = p.C;  // C11, C22, C12, C16, C26, C66
  auto build = [&](const int (*tri)[4], int ntri, double K[3][3][4]) {
    std::memset(K, 0, sizeof(double) * 36);
    const double m = ntri * p.rho * (p.dx * p.dy / 2.0) / 3.0;
    for (int t = 0; t < ntri; ++t) {
      const int T = tri[t][0], A = tri[t][3];
      const double J00 = (vi[T][1] - vi[T][0]) * p.dx, J01 = (vi[T][2] - vi[T][0]) * p.dx;
      const double J10 = (vj[T][1] - vj[T][0]) * p.dy, J11 = (vj[T][2] - vj[T][0]) * p.dy;
      const double det = J00 * J11 - J01 * J10;
      const double dxi[3] = {-1.0, 1.0, 0.0}, deta[3] = {-1.0, 0.0, 1.0};
      double bx[3], by[3];
      for (int b = 0; b < 3; ++b) {
        bx[b] = (J11 * dxi[b] - J10 * deta[b]) / det;
        by[b] = (-J01 * dxi[b] + J00 * deta[b]) / det;
      }
      const double f = std::fabs(det) / 2.0 * p.dt * p.dt / m;
      for (int b = 0; b < 3; ++b) {
        // stresses of a unit x, y displacement of vertex b
        const double sx[3] = {C[0] * bx[b] + C[3] * by[b], C[2] * bx[b] + C[4] * by[b], C[3] * bx[b] + C[5] * by[b]};
        const double sy[3] = {C[2] * by[b] + C[3] * bx[b], C[1] * by[b] + C[4] * bx[b], C[4] * by[b] + C[5] * bx[b]};
        double* c = K[1 + tri[t][1] + vi[T][b]][1 + tri[t][2] + vj[T][b]];
        c[0] += f * (bx[A] * sx[0] + by[A] * sx[2]);
        c[1] += f * (bx[A] * sy[0] + by[A] * sy[2]);
        c[2] += f * (by[A] * sx[1] + bx[A] * sx[2]);
        c[3] += f * (by[A] * sy[1] + bx[A] * sy[2]);
      }
    }
  };
  FemStencil s;
  double K[3][3][4];
  build(even, 8, K);
  for (int n = 0, b = 0; n < 9; ++n) {
    if (n == 4) continue;
    for (int c = 0; c < 4; ++c) s.e[b][c] = (float)K[n / 3][n % 3][c];
    ++b;
  }
  build(odd, 4, K);
  const int at[4][2] = {{0, 1}, {1, 0}, {1, 2}, {2, 1}};
  for (int b = 0; b < 4; ++b)
    for (int c = 0; c < 4; ++c) s.o[b][c] = (float)K[at[b][0]][at[b][1]][c];
  s.dt2 = (float)(p.dt * p.dt);
  s.rho_inv = (float)(1.0 / p.rho);
  s.scale = (float)p.out_scale;
  return s;
}

// Which uniform runs take several levels per launch: those of up to seven
// levels per node across the grid's narrower side.  The one-level kernel's
// rounding noise grows with the crossings of the grid, about 1.5e-6 of the
// field per (levels / nodes across) (61^2, 120^2, 200^2, 301^2 nodes, 430 to
// 2001 levels), and the two kernels' frames part by as much: up to this line
// by 1.6e-5 at most in what was measured.  Longer runs on small grids keep the
// element form, and with it their frames, at three to five times the time
// (100^2 nodes, 700 and 701 levels: 0.84 and 2.36 ms; 200^2, 1400 and 1401:
// 1.67 and 8.35): the line is where the frames stay the same to 2e-5, not where
// the kernels cross.
constexpr int kFemCrossings = 7;
inline bool fem_block_rule(const ErnnFemProblem& p) {
  return p.nt <= (int64_t)kFemCrossings * (p.nx < p.ny ? p.nx : p.ny);
}

constexpr size_t kFemAlign = 256;
inline size_t fem_align(size_t v) { return (v + kFemAlign - 1) / kFemAlign * kFemAlign; }

}  // namespace
}  // namespace ernn

using namespace ernn;

extern "C" size_t ernn_fem_workspace_bytes(const ErnnFemProblem* p) {
  if (p == nullptr || p->nx < 2 || p->ny < 2) return 0;
  // four levels of both components with rows padded to 16 bytes (several
  // levels per launch), at least three unpadded ones
  return 8 * fem_align((size_t)p->nx * ((p->ny + 3) / 4 * 4) * sizeof(float));
}

extern "C" int ernn_fem_forward(const ErnnFemProblem* p, const float* load, const float* signal,
                                const float* C_fields, float* frames_x, float* frames_y,
                                void* workspace, size_t workspace_bytes, void* stream) {
  // (the per-level launch takes 8 node rows per block along grid y: at most 65535 blocks)
  if (p == nullptr || p->nx < 2 || p->ny < 2 || p->nt < 1 || p->stride < 1 ||
      (int64_t)p->nx * p->ny >= ((int64_t)1 << 31) || (p->nx + 7) / 8 > 65535)
    return ERNN_ERR_INVALID;
  if (!(p->dx > 0.0) || !(p->dy > 0.0) || !(p->dt > 0.0) || !(p->rho > 0.0) ||
      !std::isfinite(p->dx) || !std::isfinite(p->dy) || !std::isfinite(p->dt) ||
      !std::isfinite(p->out_scale))
    return ERNN_ERR_INVALID;
  if (load == nullptr || signal == nullptr || frames_x == nullptr || frames_y == nullptr ||
      workspace == nullptr)
    return ERNN_ERR_INVALID;
  if (workspace_bytes < ernn_fem_workspace_bytes(p)) return ERNN_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t N = (size_t)p->nx * p->ny;
  const int nt_out = (p->nt + p->stride - 1) / p->stride;
  // frames of the levels that are never computed (0, and 1 when stride is 1)
  for (int f = 0; f < nt_out && f * p->stride <= 1; ++f) {
    if (cudaMemsetAsync(frames_x + (size_t)f * N, 0, N * sizeof(float), st) != cudaSuccess ||
        cudaMemsetAsync(frames_y + (size_t)f * N, 0, N * sizeof(float), st) != cudaSuccess)
      return ERNN_ERR_CUDA;
  }
  if (C_fields == nullptr && fem_block_rule(*p) && (reinterpret_cast<uintptr_t>(workspace) & 15u) == 0) {
    // uniform constants: kH levels per launch, each from one pair of working
    // states into the other (levels 0 and 1 are zero)
    constexpr int kW = 16, kH = 4, kCols = 128 - 8 * ((kH + 3) / 4);
    const int pitch = (p->ny + 3) / 4 * 4;
    const size_t lev = fem_align((size_t)p->nx * pitch * sizeof(float)) / sizeof(float);
    float* w = static_cast<float*>(workspace);
    FemBlock a;
    std::memset(&a, 0, sizeof(a));
    a.nx = p->nx; a.ny = p->ny; a.pitch = pitch;
    a.load = load;
    a.signal = signal;
    a.frames_x = frames_x;
    a.frames_y = frames_y;
    a.stride = p->stride;
    const FemStencil k = fem_stencil(*p);
    const dim3 grid((p->ny + kCols - 1) / kCols, (p->nx + kW - 2 * kH - 1) / (kW - 2 * kH), 1);
    int pair = 0;
    for (int n = 1; n < p->nt - 1;) {
      const int left = p->nt - 1 - n;
      a.n = n;
      a.T = left < kH ? left : kH;
      a.out = w + (size_t)(4 * pair) * lev;
      a.out_diff = a.out + 2 * lev;
      const bool chained = n > 1;  // the previous launch is the previous levels'
      const cudaError_t e = tracked_launch(kProfForward, st, [&] {
        launch_step_kernel(fem_block_kernel<kW, kH>, grid, dim3(32 * kW), 0, st, chained, a, k);
      }, (double)N * 28.0 * a.T);
      if (e != cudaSuccess) return ERNN_ERR_CUDA;
      a.cur = a.out;
      a.diff = a.out_diff;
      pair ^= 1;
      n += a.T;
    }
    return ERNN_OK;
  }
  const size_t lev = fem_align(N * sizeof(float));
  char* w = static_cast<char*>(workspace);
  float* ux[3];
  float* uy[3];
  for (int l = 0; l < 3; ++l) {
    ux[l] = reinterpret_cast<float*>(w + (2 * l) * lev);
    uy[l] = reinterpret_cast<float*>(w + (2 * l + 1) * lev);
  }
  // levels 0 and 1 are zero (slot n % 3 holds u^n)
  if (cudaMemsetAsync(w, 0, 4 * lev, st) != cudaSuccess) return ERNN_ERR_CUDA;
  const FemConsts k = fem_consts(*p);
  const dim3 block(32, 8, 1);
  const dim3 grid((p->ny + 31) / 32, (p->nx + 7) / 8, 1);
  FemStep s;
  std::memset(&s, 0, sizeof(s));
  s.nx = p->nx; s.ny = p->ny;
  s.load = load;
  s.signal = signal;
  s.cf = C_fields;
  for (int n = 1; n < p->nt - 1; ++n) {
    s.n = n;
    s.cur_x = ux[n % 3]; s.cur_y = uy[n % 3];
    s.prev_x = ux[(n + 2) % 3]; s.prev_y = uy[(n + 2) % 3];
    s.out_x = ux[(n + 1) % 3]; s.out_y = uy[(n + 1) % 3];
    if ((n + 1) % p->stride == 0) {
      const size_t f = (size_t)((n + 1) / p->stride) * N;
      s.frame_x = frames_x + f;
      s.frame_y = frames_y + f;
    } else {
      s.frame_x = s.frame_y = nullptr;
    }
    const bool chained = n > 1;  // the previous launch is the previous level's
    const cudaError_t e = tracked_launch(kProfForward, st, [&] {
      if (C_fields != nullptr) launch_step_kernel(fem_step_kernel<true>, grid, block, 0, st, chained, s, k);
      else launch_step_kernel(fem_step_kernel<false>, grid, block, 0, st, chained, s, k);
    }, (double)N * (C_fields != nullptr ? 52.0 : 28.0));
    if (e != cudaSuccess) return ERNN_ERR_CUDA;
  }
  return ERNN_OK;
}
