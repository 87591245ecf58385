// Reference-exact vertex-centred FP64 multigrid (the "port-equivalent" path).
//
// These kernels reproduce gradient-domain/src/gradient_domain/multigrid.py
// operation by operation: red-black Gauss-Seidel with colour (i + j) % 2 == 0
// first (multigrid.py:147-165), full-weighting restriction (:169-174) and
// bilinear prolongation (:177-181) on the m -> (m - 1) // 2 hierarchy, and the
// coarsest-grid sweeps (:205-207).  Arithmetic uses explicit round-to-nearest
// intrinsics in the same order as the NumPy/SciPy expressions, so no FMA
// contraction changes the result; products by 0.5, 0.25 and 1.0 are exact.
// gd_ref_vcycle runs them one pass per operation: it is the all-FP64 GPU
// translation of the reference that the batched solver is measured against.
// gd_ref_vcycle_fused, behind v_cycle and the "multigrid" method, gives the same
// bits in two launches a level instead of twelve: tiles in shared memory with
// enough halo for every sweep, so that smoothing, residual and restriction are one
// kernel on the way down and prolongation and smoothing one on the way up.  A
// launch of these kernels takes 2-4 us on all but the largest levels, so their
// number is what a cycle costs (1023 x 1023, 2 + 2 sweeps: 150 us a cycle, 240 us one
// operation a launch).  (The streaming smoother of
// gd_smooth.cu is no help here: on a few hundred rows its row-by-row FP64 chain
// took 17 us a level.)

#include <algorithm>
#include <cmath>
#include <mutex>

#include "gd_internal.cuh"

namespace gd {
namespace {

__device__ __forceinline__ double at(const double *a, int i, int j, int m, int n) {
  return (i >= 0 && i < m && j >= 0 && j < n) ? a[(size_t)i * n + j] : 0.0;
}

// neighbours = up + down + left + right, evaluated left to right (operators.py:104-106).
__device__ __forceinline__ double nbr_sum(const double *u, int i, int j, int m, int n) {
  double s = __dadd_rn(at(u, i - 1, j, m, n), at(u, i + 1, j, m, n));
  s = __dadd_rn(s, at(u, i, j - 1, m, n));
  return __dadd_rn(s, at(u, i, j + 1, m, n));
}

// One colour of one RB-GS sweep: u = 0.25 * (neighbours - h^2 b) on parity cells.
__global__ void ref_rb_colour(double *__restrict__ u, const double *__restrict__ b, int m, int n,
                              double h2, int parity) {
  const int half = (n + 1) / 2;
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (long long)m * half) return;
  const int i = (int)(k / half);
  const int j = 2 * (int)(k % half) + ((parity + i) & 1);
  if (j >= n) return;
  const double s = nbr_sum(u, i, j, m, n);
  u[(size_t)i * n + j] = __dmul_rn(0.25, __dsub_rn(s, __dmul_rn(h2, b[(size_t)i * n + j])));
}

// r = b - (neighbours - 4 u) / h^2  (multigrid.py:210 with operators.py:107).
__global__ void ref_residual_kernel(double *__restrict__ r, const double *__restrict__ u,
                                    const double *__restrict__ b, int m, int n, double h2) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (long long)m * n) return;
  const int i = (int)(k / n), j = (int)(k % n);
  const double lap = __ddiv_rn(__dsub_rn(nbr_sum(u, i, j, m, n), __dmul_rn(4.0, u[k])), h2);
  r[k] = __dsub_rn(b[k], lap);
}

// rc = 0.25 * Rows^T r Cols: rows first (fine rows 2I, 2I+1, 2I+2 in order),
// then columns, as scipy's csc products accumulate them.
__global__ void ref_restrict_kernel(double *__restrict__ rc, const double *__restrict__ r, int m,
                                    int n, int mc, int nc) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (long long)mc * nc) return;
  const int I = (int)(k / nc), J = (int)(k % nc);
  double t[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int j = 2 * J + q;
    const double *c = r + j;
    double s = __dmul_rn(0.5, c[(size_t)(2 * I) * n]);
    s = __dadd_rn(s, c[(size_t)(2 * I + 1) * n]);
    t[q] = __dadd_rn(s, __dmul_rn(0.5, c[(size_t)(2 * I + 2) * n]));
  }
  double s = __dadd_rn(__dmul_rn(0.5, t[0]), t[1]);
  s = __dadd_rn(s, __dmul_rn(0.5, t[2]));
  rc[k] = __dmul_rn(s, 0.25);
}

// Division by h^2: where that is a power of two (spacing 1 and its doublings) the
// product with its reciprocal is the same number.
struct Square {
  double value, inverse;  // inverse: exact reciprocal, or 0
  explicit Square(double h2) : value(h2), inverse(0.0) {
    int e = 0;
    if (std::frexp(h2, &e) == 0.5 && e > -500 && e < 500) inverse = 1.0 / h2;
  }
  __device__ __forceinline__ double divide(double a) const {
    return inverse != 0.0 ? __dmul_rn(a, inverse) : __ddiv_rn(a, value);
  }
};

// Interpolate one fine index from the coarse axis: returns the count of
// contributing coarse indices (c0, c1) and their weight.
__device__ __forceinline__ int prolong_sources(int i, int nc, int *c0, int *c1, double *w) {
  if (i & 1) {
    const int s = (i - 1) >> 1;
    *c0 = s;
    *w = 1.0;
    return (s >= 0 && s < nc) ? 1 : 0;
  }
  int cnt = 0;
  const int a = (i >> 1) - 1, b = i >> 1;
  *w = 0.5;
  if (a >= 0 && a < nc) { *c0 = a; cnt = 1; }
  if (b >= 0 && b < nc) {
    if (cnt == 0) *c0 = b; else *c1 = b;
    ++cnt;
  }
  return cnt;
}

// (Rows e Cols^T)(i, j): inner sum over coarse rows, then coarse columns.
__device__ __forceinline__ double prolonged(const double *__restrict__ e, int i, int j, int mc,
                                            int nc) {
  int ri0 = 0, ri1 = 0, cj0 = 0, cj1 = 0;
  double wi, wj;
  const int ni = prolong_sources(i, mc, &ri0, &ri1, &wi);
  const int nj = prolong_sources(j, nc, &cj0, &cj1, &wj);
  double total = 0.0;
  if (ni > 0 && nj > 0) {
    double col[2];
    const int cj[2] = {cj0, cj1};
    for (int q = 0; q < nj; ++q) {
      double s = __dmul_rn(wi, e[(size_t)ri0 * nc + cj[q]]);
      if (ni == 2) s = __dadd_rn(s, __dmul_rn(wi, e[(size_t)ri1 * nc + cj[q]]));
      col[q] = s;
    }
    total = __dmul_rn(wj, col[0]);
    if (nj == 2) total = __dadd_rn(total, __dmul_rn(wj, col[1]));
  }
  return total;
}

__global__ void ref_prolong_add_kernel(double *__restrict__ u, const double *__restrict__ e, int m,
                                       int n, int mc, int nc) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (long long)m * n) return;
  u[k] = __dadd_rn(u[k], prolonged(e, (int)(k / n), (int)(k % n), mc, nc));
}

// Coarsest grid: `sweeps` RB-GS sweeps by one CTA (multigrid.py:205-207).
// Uses shared memory when the grid fits, global memory otherwise.
constexpr int kCoarseThreads = 1024;
constexpr int kCoarseSmemCells = 2560;  // 2 arrays x 8 B x 2560 = 40 KB

__global__ void __launch_bounds__(kCoarseThreads)
ref_coarse_kernel(double *__restrict__ u_g, const double *__restrict__ b_g, int m, int n,
                  double h2, int sweeps) {
  __shared__ double su[kCoarseSmemCells], sb[kCoarseSmemCells];
  const int cells = m * n;
  const bool in_smem = cells <= kCoarseSmemCells;
  double *u = in_smem ? su : u_g;
  const double *b = in_smem ? sb : b_g;
  if (in_smem) {
    for (int k = threadIdx.x; k < cells; k += blockDim.x) {
      su[k] = u_g[k];
      sb[k] = b_g[k];
    }
  }
  __syncthreads();
  const int half = (n + 1) / 2;
  for (int s = 0; s < sweeps; ++s) {
    for (int parity = 0; parity < 2; ++parity) {
      for (int k = threadIdx.x; k < m * half; k += blockDim.x) {
        const int i = k / half;
        const int j = 2 * (k % half) + ((parity + i) & 1);
        if (j < n) {
          const double nb = nbr_sum(u, i, j, m, n);
          u[i * n + j] = __dmul_rn(0.25, __dsub_rn(nb, __dmul_rn(h2, b[i * n + j])));
        }
      }
      __syncthreads();
      if (!in_smem) __threadfence_block();
    }
  }
  if (in_smem)
    for (int k = threadIdx.x; k < cells; k += blockDim.x) u_g[k] = su[k];
}

// The same sweeps where a thread can own one cell of each colour and the grid fits
// in shared memory with a ring of zeros (the values outside the array): the
// thread's indices and h^2 b stay in registers, and a grid of at most 32 cells a
// colour needs one warp and no block barrier (7 x 7, 60 sweeps: 37 us
// with 1024 threads and bounds tests, 10 us).
constexpr int kSmallCells = 2816;  // padded cells: 22 KB

__global__ void __launch_bounds__(kCoarseThreads)
ref_coarse_small_kernel(double *__restrict__ u_g, const double *__restrict__ b_g, int m, int n,
                        double h2, int sweeps, int zero) {
  __shared__ double u[kSmallCells];
  const int pn = n + 2, half = (n + 1) / 2;
  for (int k = threadIdx.x; k < (m + 2) * pn; k += blockDim.x) {
    const int i = k / pn - 1, j = k % pn - 1;
    u[k] = zero ? 0.0 : at(u_g, i, j, m, n);
  }
  const int i = threadIdx.x / half, jj = 2 * (threadIdx.x % half);
  int c[2];
  double hb[2];
  bool on[2];
#pragma unroll
  for (int parity = 0; parity < 2; ++parity) {
    const int j = jj + ((parity + i) & 1);
    on[parity] = i < m && j < n;
    c[parity] = on[parity] ? (i + 1) * pn + j + 1 : 0;
    hb[parity] = on[parity] ? __dmul_rn(h2, b_g[i * n + j]) : 0.0;
  }
  const bool one_warp = blockDim.x <= 32;
  __syncthreads();
  for (int s = 0; s < sweeps; ++s) {
#pragma unroll
    for (int parity = 0; parity < 2; ++parity) {
      if (on[parity]) {
        const int q = c[parity];
        double v = __dadd_rn(u[q - pn], u[q + pn]);
        v = __dadd_rn(v, u[q - 1]);
        v = __dadd_rn(v, u[q + 1]);
        u[q] = __dmul_rn(0.25, __dsub_rn(v, hb[parity]));
      }
      if (one_warp) __syncwarp();
      else __syncthreads();
    }
  }
#pragma unroll
  for (int parity = 0; parity < 2; ++parity)
    if (on[parity]) u_g[(c[parity] / pn - 1) * n + c[parity] % pn - 1] = u[c[parity]];
}

// ---------------------------------------------------------------------------
// One level in shared memory: 32 x 32 tiles, a warp per row, a lane per pair of
// columns.  A half sweep leaves the outermost ring that is still exact one cell
// further in, so `sweeps` sweeps need 2 sweeps halo cells (the way down two more,
// for the residual's neighbours and the restriction's reach); cells outside the
// grid stay zero.  The halo is recomputed by every tile that needs it, and a level
// is read from one buffer and written to another, so tiles do not depend on each
// other.
constexpr int kTile = 32, kTileThreads = 512, kTileWarps = kTileThreads / 32;
constexpr int kTileSweeps = 4;  // most sweeps of one launch

inline int tile_halo_down(int sweeps) { return 2 * sweeps + 2; }
inline int tile_halo_up(int sweeps) { return 2 * sweeps; }
inline size_t tile_smem(int halo) {
  return (size_t)2 * (kTile + 2 * halo) * (kTile + 2 * halo) * sizeof(double);
}
static_assert(kTile + 2 * (2 * kTileSweeps + 2) <= 64, "a lane per pair of columns");

// `sweeps` sweeps on the tile (RX x RX cells, corner at gy0, gx0, whose parity is even).
__device__ __forceinline__ void tile_sweeps(double *u, const double *b, int RX, int gy0, int gx0,
                                            int m, int n, double h2, int sweeps) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int half = 0; half < 2 * sweeps; ++half) {
    for (int ry = 1 + warp; ry < RX - 1; ry += kTileWarps) {
      const int rx = 2 * lane + ((half + ry) & 1);
      const int i = gy0 + ry, j = gx0 + rx;
      if (rx >= 1 && rx < RX - 1 && i >= 0 && i < m && j >= 0 && j < n) {
        const int q = ry * RX + rx;
        double s = __dadd_rn(u[q - RX], u[q + RX]);
        s = __dadd_rn(s, u[q - 1]);
        s = __dadd_rn(s, u[q + 1]);
        u[q] = __dmul_rn(0.25, __dsub_rn(s, __dmul_rn(h2, b[q])));
      }
    }
    __syncthreads();
  }
}

// Pre-sweeps, the smoothed iterate to `out`, and the restricted residual to bc.
// `zero`: the iterate starts from zero (u_g is not read).
__global__ void __launch_bounds__(kTileThreads)
ref_down_kernel(double *__restrict__ out, double *__restrict__ bc, const double *__restrict__ u_g,
                const double *__restrict__ b_g, int m, int n, int mc, int nc, double h2, Square hd,
                int sweeps, int zero) {
  extern __shared__ double tile[];
  const int H = 2 * sweeps + 2, RX = kTile + 2 * H;
  double *u = tile, *b = tile + RX * RX;
  const int y0 = blockIdx.y * kTile, x0 = blockIdx.x * kTile;
  const int gy0 = y0 - H, gx0 = x0 - H;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int ry = warp; ry < RX; ry += kTileWarps)
    for (int rx = lane; rx < RX; rx += 32) {
      u[ry * RX + rx] = zero ? 0.0 : at(u_g, gy0 + ry, gx0 + rx, m, n);
      b[ry * RX + rx] = at(b_g, gy0 + ry, gx0 + rx, m, n);
    }
  __syncthreads();
  tile_sweeps(u, b, RX, gy0, gx0, m, n, h2, sweeps);
  for (int ry = H + warp; ry < H + kTile; ry += kTileWarps) {
    const int i = gy0 + ry, j = x0 + lane;
    if (i < m && j < n) out[(size_t)i * n + j] = u[ry * RX + H + lane];
  }
  // residual of the rows and columns the tile's coarse cells reach, in place of b
  for (int ry = H + warp; ry <= H + kTile; ry += kTileWarps)
    for (int rx = H + lane; rx <= H + kTile; rx += 32) {
      const int q = ry * RX + rx;
      double s = __dadd_rn(u[q - RX], u[q + RX]);
      s = __dadd_rn(s, u[q - 1]);
      s = __dadd_rn(s, u[q + 1]);
      b[q] = __dsub_rn(b[q], hd.divide(__dsub_rn(s, __dmul_rn(4.0, u[q]))));
    }
  __syncthreads();
  constexpr int kC = kTile / 2;
  if (threadIdx.x < kC * kC) {
    const int qi = threadIdx.x / kC, qj = threadIdx.x % kC;
    const int I = y0 / 2 + qi, J = x0 / 2 + qj;
    if (I < mc && J < nc) {
      double t[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const double *c = b + (H + 2 * qi) * RX + H + 2 * qj + q;
        double s = __dmul_rn(0.5, c[0]);
        s = __dadd_rn(s, c[RX]);
        t[q] = __dadd_rn(s, __dmul_rn(0.5, c[2 * RX]));
      }
      double s = __dadd_rn(__dmul_rn(0.5, t[0]), t[1]);
      s = __dadd_rn(s, __dmul_rn(0.5, t[2]));
      bc[(size_t)I * nc + J] = __dmul_rn(s, 0.25);
    }
  }
}

// The prolonged correction added, then post-sweeps: in -> out.
__global__ void __launch_bounds__(kTileThreads)
ref_up_kernel(double *__restrict__ out, const double *__restrict__ in,
              const double *__restrict__ b_g, const double *__restrict__ e, int m, int n, int mc,
              int nc, double h2, int sweeps) {
  extern __shared__ double tile[];
  const int H = 2 * sweeps, RX = kTile + 2 * H;
  double *u = tile, *b = tile + RX * RX;
  const int y0 = blockIdx.y * kTile, x0 = blockIdx.x * kTile;
  const int gy0 = y0 - H, gx0 = x0 - H;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int ry = warp; ry < RX; ry += kTileWarps)
    for (int rx = lane; rx < RX; rx += 32) {
      const int i = gy0 + ry, j = gx0 + rx;
      const bool inside = i >= 0 && i < m && j >= 0 && j < n;
      const size_t g = (size_t)i * n + j;
      u[ry * RX + rx] = inside ? __dadd_rn(in[g], prolonged(e, i, j, mc, nc)) : 0.0;
      b[ry * RX + rx] = inside ? b_g[g] : 0.0;
    }
  __syncthreads();
  tile_sweeps(u, b, RX, gy0, gx0, m, n, h2, sweeps);
  for (int ry = H + warp; ry < H + kTile; ry += kTileWarps) {
    const int i = gy0 + ry, j = x0 + lane;
    if (i < m && j < n) out[(size_t)i * n + j] = u[ry * RX + H + lane];
  }
}

constexpr int kReduceThreads = 256;
constexpr int kReduceBlocks = 592;  // 4 x 148 SMs

__global__ void __launch_bounds__(kReduceThreads)
ref_dot_partial(double *__restrict__ part, const double *__restrict__ a,
                const double *__restrict__ b, long long count) {
  double s = 0.0;
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < count;
       k += (long long)gridDim.x * blockDim.x)
    s += a[k] * b[k];
  s = block_sum<kReduceThreads>(s);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

__global__ void __launch_bounds__(kReduceThreads)
ref_dot_final(double *__restrict__ out, const double *__restrict__ part, int nparts) {
  double s = 0.0;
  for (int k = threadIdx.x; k < nparts; k += blockDim.x) s += part[k];
  s = block_sum<kReduceThreads>(s);
  if (threadIdx.x == 0) out[0] = s;
}

__global__ void ref_axpby_kernel(double *__restrict__ y, const double *__restrict__ x, double alpha,
                                 double beta, long long count) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < count) y[k] = __dadd_rn(__dmul_rn(alpha, x[k]), __dmul_rn(beta, y[k]));
}

inline unsigned blocks_for(long long work, int threads) {
  return (unsigned)((work + threads - 1) / threads);
}

struct RefLevel {
  int m, n;
  size_t u_off, b_off, r_off;  // byte offsets in the workspace (levels >= 1 use u, b)
};

// Level list of the reference recursion: stops at the first grid that is
// coarsest (min side <= coarsest_size or coarse side < 2).
int ref_levels(int m, int n, int coarsest_size, RefLevel *lv, int max_levels, size_t *bytes) {
  size_t off = 0;
  int count = 0;
  while (true) {
    if (count >= max_levels) return -1;
    RefLevel &L = lv[count++];
    L.m = m;
    L.n = n;
    const size_t cells = (size_t)m * n * sizeof(double);
    L.r_off = off;
    off = align_up(off + cells, 256);
    if (count > 1) {
      L.u_off = off;
      off = align_up(off + cells, 256);
      L.b_off = off;
      off = align_up(off + cells, 256);
    } else {
      L.u_off = L.b_off = 0;
    }
    const int mc = (m - 1) / 2, nc = (n - 1) / 2;
    if (m <= coarsest_size || n <= coarsest_size || mc < 2 || nc < 2) break;
    m = mc;
    n = nc;
  }
  *bytes = off + 1024 * sizeof(double);  // + dot partials
  return count;
}

int ref_vcycle_rec(RefLevel *lv, int nlev, int l, double *u, const double *b, double h,
                   int pre, int post, int sweeps, char *ws, cudaStream_t st) {
  const RefLevel &L = lv[l];
  const int m = L.m, n = L.n, T = 256;
  const double h2 = h * h;
  if (l == nlev - 1) {
    ref_coarse_kernel<<<1, kCoarseThreads, 0, st>>>(u, b, m, n, h2, sweeps);
    GD_CHECK_LAUNCH();
    return GD_OK;
  }
  const unsigned g_col = blocks_for((long long)m * ((n + 1) / 2), T);
  for (int s = 0; s < pre; ++s)
    for (int p = 0; p < 2; ++p) ref_rb_colour<<<g_col, T, 0, st>>>(u, b, m, n, h2, p);
  double *r = (double *)(ws + L.r_off);
  ref_residual_kernel<<<blocks_for((long long)m * n, T), T, 0, st>>>(r, u, b, m, n, h2);
  const RefLevel &C = lv[l + 1];
  double *uc = (double *)(ws + C.u_off);
  double *bc = (double *)(ws + C.b_off);
  ref_restrict_kernel<<<blocks_for((long long)C.m * C.n, T), T, 0, st>>>(bc, r, m, n, C.m, C.n);
  GD_CHECK_LAUNCH();
  GD_CHECK_CUDA(cudaMemsetAsync(uc, 0, (size_t)C.m * C.n * sizeof(double), st));
  int rc = ref_vcycle_rec(lv, nlev, l + 1, uc, bc, 2.0 * h, pre, post, sweeps, ws, st);
  if (rc != GD_OK) return rc;
  ref_prolong_add_kernel<<<blocks_for((long long)m * n, T), T, 0, st>>>(u, uc, m, n, C.m, C.n);
  for (int s = 0; s < post; ++s)
    for (int p = 0; p < 2; ++p) ref_rb_colour<<<g_col, T, 0, st>>>(u, b, m, n, h2, p);
  GD_CHECK_LAUNCH();
  return GD_OK;
}

// `sweeps` sweeps in place, one colour a launch.
void ref_colour_sweeps(double *u, const double *b, int m, int n, double h2, int sweeps,
                       cudaStream_t st) {
  for (int s = 0; s < sweeps; ++s)
    for (int p = 0; p < 2; ++p)
      ref_rb_colour<<<blocks_for((long long)m * ((n + 1) / 2), 256), 256, 0, st>>>(u, b, m, n, h2,
                                                                                   p);
}

// ref_vcycle_rec in two launches a level; a level's residual array holds the smoothed
// iterate between them.  `zero`: u starts from zero and is only written.  Sweeps
// beyond kTileSweeps run one colour a launch.
int ref_vcycle_fused_rec(RefLevel *lv, int nlev, int l, double *u, const double *b, double h,
                         int pre, int post, int sweeps, int zero, char *ws, cudaStream_t st) {
  const RefLevel &L = lv[l];
  const int m = L.m, n = L.n;
  const double h2 = h * h;
  const size_t bytes = (size_t)m * n * sizeof(double);
  if (l == nlev - 1) {
    const int owners = m * ((n + 1) / 2);
    if ((long long)(m + 2) * (n + 2) <= kSmallCells && owners <= kCoarseThreads) {
      ref_coarse_small_kernel<<<1, (owners + 31) / 32 * 32, 0, st>>>(u, b, m, n, h2, sweeps, zero);
    } else {
      if (zero) GD_CHECK_CUDA(cudaMemsetAsync(u, 0, bytes, st));
      ref_coarse_kernel<<<1, kCoarseThreads, 0, st>>>(u, b, m, n, h2, sweeps);
    }
    GD_CHECK_LAUNCH();
    return GD_OK;
  }
  const RefLevel &C = lv[l + 1];
  double *tmp = (double *)(ws + L.r_off), *uc = (double *)(ws + C.u_off);
  double *bc = (double *)(ws + C.b_off);
  const dim3 grid(ceil_div(n, kTile), ceil_div(m, kTile));
  const int early = std::max(pre - kTileSweeps, 0), late = std::max(post - kTileSweeps, 0);
  if (early > 0) {
    if (zero) GD_CHECK_CUDA(cudaMemsetAsync(u, 0, bytes, st));
    ref_colour_sweeps(u, b, m, n, h2, early, st);
    zero = 0;
  }
  ref_down_kernel<<<grid, kTileThreads, tile_smem(tile_halo_down(pre - early)), st>>>(
      tmp, bc, u, b, m, n, C.m, C.n, h2, Square(h2), pre - early, zero);
  GD_CHECK_LAUNCH();
  const int rc = ref_vcycle_fused_rec(lv, nlev, l + 1, uc, bc, 2.0 * h, pre, post, sweeps, 1, ws,
                                      st);
  if (rc != GD_OK) return rc;
  ref_up_kernel<<<grid, kTileThreads, tile_smem(tile_halo_up(post - late)), st>>>(
      u, tmp, b, uc, m, n, C.m, C.n, h2, post - late);
  ref_colour_sweeps(u, b, m, n, h2, late, st);
  GD_CHECK_LAUNCH();
  return GD_OK;
}

// Partial sums of r^2 for r = b - laplacian(u) (ref_residual_kernel's expression);
// ref_dot_final adds them.
__global__ void __launch_bounds__(kReduceThreads)
ref_residual_norm_partial(double *__restrict__ part, const double *__restrict__ u,
                          const double *__restrict__ b, int m, int n, Square h2) {
  double s = 0.0;
  for (int i = blockIdx.y; i < m; i += gridDim.y)
    for (int j = blockIdx.x * kReduceThreads + threadIdx.x; j < n; j += gridDim.x * kReduceThreads) {
      const size_t g = (size_t)i * n + j;
      const double lap = h2.divide(__dsub_rn(nbr_sum(u, i, j, m, n), __dmul_rn(4.0, u[g])));
      const double r = __dsub_rn(b[g], lap);
      s += r * r;
    }
  s = block_sum<kReduceThreads>(s);
  if (threadIdx.x == 0) part[blockIdx.y * gridDim.x + blockIdx.x] = s;
}

}  // namespace
}  // namespace gd

using namespace gd;

extern "C" size_t gd_ref_workspace_bytes(int32_t m, int32_t n, int32_t coarsest_size) {
  RefLevel lv[64];
  size_t bytes = 0;
  if (m <= 0 || n <= 0) return 0;
  if (ref_levels(m, n, coarsest_size, lv, 64, &bytes) < 0) return 0;
  return bytes;
}

extern "C" int gd_ref_vcycle(double *u, const double *b, int32_t m, int32_t n, double spacing,
                             int32_t pre, int32_t post, int32_t coarsest_size,
                             int32_t coarsest_sweeps, void *ws, size_t bytes, cudaStream_t st) {
  GD_REQUIRE(u && b && m > 0 && n > 0 && pre >= 0 && post >= 0 && coarsest_sweeps >= 0,
             GD_ERR_ARG, "gd_ref_vcycle: bad arguments");
  RefLevel lv[64];
  size_t need = 0;
  const int nlev = ref_levels(m, n, coarsest_size, lv, 64, &need);
  GD_REQUIRE(nlev > 0, GD_ERR_ARG, "gd_ref_vcycle: hierarchy too deep");
  GD_REQUIRE(ws != nullptr && bytes >= need, GD_ERR_ARG,
             "gd_ref_vcycle: workspace of %zu bytes, need %zu", bytes, need);
  return ref_vcycle_rec(lv, nlev, 0, u, b, spacing, pre, post, coarsest_sweeps, (char *)ws, st);
}

extern "C" int gd_ref_vcycle_fused(double *u, const double *b, int32_t m, int32_t n,
                                   double spacing, int32_t pre, int32_t post,
                                   int32_t coarsest_size, int32_t coarsest_sweeps, void *ws,
                                   size_t bytes, cudaStream_t st) {
  GD_REQUIRE(u && b && m > 0 && n > 0 && pre >= 0 && post >= 0 && coarsest_sweeps >= 0,
             GD_ERR_ARG, "gd_ref_vcycle_fused: bad arguments");
  RefLevel lv[64];
  size_t need = 0;
  const int nlev = ref_levels(m, n, coarsest_size, lv, 64, &need);
  GD_REQUIRE(nlev > 0, GD_ERR_ARG, "gd_ref_vcycle_fused: hierarchy too deep");
  GD_REQUIRE(ws != nullptr && bytes >= need, GD_ERR_ARG,
             "gd_ref_vcycle_fused: workspace of %zu bytes, need %zu", bytes, need);
  if (ceil_div(m, kTile) > 65535)  // more tile rows than a grid has: operation by operation
    return ref_vcycle_rec(lv, nlev, 0, u, b, spacing, pre, post, coarsest_sweeps, (char *)ws, st);
  return ref_vcycle_fused_rec(lv, nlev, 0, u, b, spacing, pre, post, coarsest_sweeps, 0,
                              (char *)ws, st);
}

extern "C" int gd_ref_residual_norm2(double *out, const double *u, const double *b, int32_t m,
                                     int32_t n, double spacing, void *ws, size_t bytes,
                                     cudaStream_t st) {
  GD_REQUIRE(out && u && b && m > 0 && n > 0, GD_ERR_ARG, "gd_ref_residual_norm2: bad arguments");
  GD_REQUIRE(ws && bytes >= kReduceBlocks * sizeof(double), GD_ERR_ARG,
             "gd_ref_residual_norm2: workspace needs %zu bytes",
             (size_t)kReduceBlocks * sizeof(double));
  double *part = (double *)ws;
  const int gx = std::min(ceil_div(n, kReduceThreads), kReduceBlocks);
  const dim3 grid(gx, std::max(1, std::min(m, kReduceBlocks / gx)));
  ref_residual_norm_partial<<<grid, kReduceThreads, 0, st>>>(part, u, b, m, n,
                                                             Square(spacing * spacing));
  ref_dot_final<<<1, kReduceThreads, 0, st>>>(out, part, (int)(grid.x * grid.y));
  GD_CHECK_LAUNCH();
  return GD_OK;
}

extern "C" int gd_ref_residual(double *r, const double *u, const double *b, int32_t m, int32_t n,
                               double spacing, cudaStream_t st) {
  GD_REQUIRE(r && u && b && m > 0 && n > 0, GD_ERR_ARG, "gd_ref_residual: bad arguments");
  ref_residual_kernel<<<blocks_for((long long)m * n, 256), 256, 0, st>>>(r, u, b, m, n,
                                                                         spacing * spacing);
  GD_CHECK_LAUNCH();
  return GD_OK;
}

extern "C" int gd_ref_dot(double *out, const double *a, const double *b, int64_t count, void *ws,
                          size_t bytes, cudaStream_t st) {
  GD_REQUIRE(out && a && b && count >= 0, GD_ERR_ARG, "gd_ref_dot: bad arguments");
  GD_REQUIRE(ws && bytes >= kReduceBlocks * sizeof(double), GD_ERR_ARG,
             "gd_ref_dot: workspace needs %zu bytes", (size_t)kReduceBlocks * sizeof(double));
  double *part = (double *)ws;
  ref_dot_partial<<<kReduceBlocks, kReduceThreads, 0, st>>>(part, a, b, count);
  ref_dot_final<<<1, kReduceThreads, 0, st>>>(out, part, kReduceBlocks);
  GD_CHECK_LAUNCH();
  return GD_OK;
}

extern "C" int gd_ref_axpby(double *y, const double *x, double alpha, double beta, int64_t count,
                            cudaStream_t st) {
  GD_REQUIRE(y && x && count >= 0, GD_ERR_ARG, "gd_ref_axpby: bad arguments");
  if (count == 0) return GD_OK;
  ref_axpby_kernel<<<blocks_for(count, 256), 256, 0, st>>>(y, x, alpha, beta, count);
  GD_CHECK_LAUNCH();
  return GD_OK;
}

extern "C" int gd_ref_restrict(double *rc, const double *r, int32_t m, int32_t n,
                               cudaStream_t st) {
  GD_REQUIRE(rc && r && m >= 3 && n >= 3, GD_ERR_ARG,
             "gd_ref_restrict: needs a fine grid of at least 3 x 3");
  const int mc = (m - 1) / 2, nc = (n - 1) / 2;
  ref_restrict_kernel<<<blocks_for((long long)mc * nc, 256), 256, 0, st>>>(rc, r, m, n, mc, nc);
  GD_CHECK_LAUNCH();
  return GD_OK;
}

extern "C" int gd_ref_prolong_add(double *u, const double *e, int32_t m, int32_t n, int32_t mc,
                                  int32_t nc, cudaStream_t st) {
  GD_REQUIRE(u && e && m > 0 && n > 0 && mc > 0 && nc > 0, GD_ERR_ARG,
             "gd_ref_prolong_add: bad arguments");
  ref_prolong_add_kernel<<<blocks_for((long long)m * n, 256), 256, 0, st>>>(u, e, m, n, mc, nc);
  GD_CHECK_LAUNCH();
  return GD_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free variant of gd_ref_vcycle.
//
// Some callers cannot allocate device memory when they need a V-cycle: code
// running while a CUDA stream is being captured into a graph (cudaMalloc is
// not permitted there), real-time loops that forbid allocation after start-up,
// and host applications that own the whole device memory budget and give
// plug-ins no allocator.  gd_ref_vcycle_static takes its coarse-level scratch
// from the file-scope array below instead of a caller workspace.  The array
// is GD_STATIC_SCRATCH_BYTES (4 MiB) on every GPU that loads this library and
// stays allocated until the process exits.  In host code `g_static_scratch`
// names a host-side stand-in, not device memory, so its device address is
// looked up with cudaGetSymbolAddress once per device and cached.
namespace gd {
namespace {

__device__ __align__(256) unsigned char g_static_scratch[GD_STATIC_SCRATCH_BYTES];

constexpr int kMaxStaticDevices = 64;
void *g_static_ptr[kMaxStaticDevices] = {};
std::mutex g_static_mu;

// Device address of g_static_scratch on the current device (looked up once).
int static_scratch(void **out) {
  int dev = 0;
  GD_CHECK_CUDA(cudaGetDevice(&dev));
  GD_REQUIRE(dev >= 0 && dev < kMaxStaticDevices, GD_ERR_UNSUPPORTED,
             "gd_ref_vcycle_static: device %d beyond the %d supported", dev, kMaxStaticDevices);
  std::lock_guard<std::mutex> hold(g_static_mu);
  if (g_static_ptr[dev] == nullptr) {
    void *p = nullptr;
    GD_CHECK_CUDA(cudaGetSymbolAddress(&p, g_static_scratch));
    g_static_ptr[dev] = p;
  }
  *out = g_static_ptr[dev];
  return GD_OK;
}

}  // namespace
}  // namespace gd

extern "C" int gd_ref_vcycle_static(double *u, const double *b, int32_t m, int32_t n,
                                    double spacing, int32_t pre, int32_t post,
                                    int32_t coarsest_size, int32_t coarsest_sweeps,
                                    cudaStream_t st) {
  GD_REQUIRE(u && b && m > 0 && n > 0 && pre >= 0 && post >= 0 && coarsest_sweeps >= 0,
             GD_ERR_ARG, "gd_ref_vcycle_static: bad arguments");
  RefLevel lv[64];
  size_t need = 0;
  const int nlev = ref_levels(m, n, coarsest_size, lv, 64, &need);
  GD_REQUIRE(nlev > 0, GD_ERR_ARG, "gd_ref_vcycle_static: hierarchy too deep");
  // a single-level hierarchy is the coarsest solve in place on u: no scratch at all
  void *ws = nullptr;
  if (nlev > 1) {
    GD_REQUIRE(need <= (size_t)GD_STATIC_SCRATCH_BYTES, GD_ERR_ARG,
               "gd_ref_vcycle_static: a %d x %d grid needs %zu bytes of scratch, more than "
               "the %zu-byte static array; use gd_ref_vcycle with a workspace",
               m, n, need, (size_t)GD_STATIC_SCRATCH_BYTES);
    const int rc = static_scratch(&ws);
    if (rc != GD_OK) return rc;
  }
  // ref_vcycle_rec zeroes every coarse iterate before use, so the contents left
  // by the previous call do not leak into this one.
  return ref_vcycle_rec(lv, nlev, 0, u, b, spacing, pre, post, coarsest_sweeps, (char *)ws, st);
}
