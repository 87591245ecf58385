// Right-hand-side assembly on the device, error reporting and version.
//
// gd_gradient follows operators.py:30-50 (forward differences, last column of
// gx and last row of gy zero), gd_divergence follows operators.py:53-83
// (backward differences with the
// edge rows/columns taken from the adjacent gradient), gd_fold_dirichlet
// follows operators.py:139-169 as solve_dirichlet calls it (poisson.py:131-143,
// spacing 1), and gd_masked_rhs follows the masked assembly of
// poisson.py:216-224.  All three keep the reference's order of additions.

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <type_traits>

#include "gd_internal.cuh"

namespace gd {

static thread_local char g_error[512] = "";

void set_error(const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_error, sizeof(g_error), fmt, ap);
  va_end(ap);
}

namespace {

__global__ void k_divergence(double *__restrict__ out, const double *__restrict__ gx,
                             const double *__restrict__ gy, int h, int w) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (long long)h * w) return;
  const int i = (int)(k / w), j = (int)(k % w);
  double dx = 0.0, dy = 0.0;
  if (w > 1) {
    if (j == 0) dx = gx[k];
    else if (j == w - 1) dx = -gx[k - 1];
    else dx = __dsub_rn(gx[k], gx[k - 1]);
  }
  if (h > 1) {
    if (i == 0) dy = gy[k];
    else if (i == h - 1) dy = -gy[k - w];
    else dy = __dsub_rn(gy[k], gy[k - w]);
  }
  out[k] = __dadd_rn(dx, dy);
}

__global__ void k_gradient(double *__restrict__ gx, double *__restrict__ gy,
                           const double *__restrict__ u, int h, int w) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (long long)h * w) return;
  const int i = (int)(k / w), j = (int)(k % w);
  gx[k] = j < w - 1 ? __dsub_rn(u[k + 1], u[k]) : 0.0;
  gy[k] = i < h - 1 ? __dsub_rn(u[k + w], u[k]) : 0.0;
}

__global__ void k_fold(double *__restrict__ f, const double *__restrict__ div,
                       const double *__restrict__ bnd, int h, int w, double scale) {
  const int m = h - 2, n = w - 2;
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (long long)m * n) return;
  const int i = (int)(k / n), j = (int)(k % n);
  double v = div[(long long)(i + 1) * w + (j + 1)];
  if (i == 0) v = __dsub_rn(v, bnd[j + 1]);
  if (i == m - 1) v = __dsub_rn(v, bnd[(long long)(h - 1) * w + j + 1]);
  if (j == 0) v = __dsub_rn(v, bnd[(long long)(i + 1) * w]);
  if (j == n - 1) v = __dsub_rn(v, bnd[(long long)(i + 1) * w + w - 1]);
  f[k] = __dmul_rn(scale, v);
}

// fold_boundary for any spacing and channel count (operators.py:139-169):
// rhs and out are (h-2, w-2, c), bnd is (h, w, c), channels interleaved.  The
// four ring subtractions run in the reference's order (first row, last row,
// first column, last column), each subtracting the rounded product
// weight * boundary, so a corner cell sees two of them in that order.
__global__ void k_fold_ring(double *out, const double *rhs, const double *__restrict__ bnd,
                            int h, int w, int c, double weight) {
  const int m = h - 2, n = w - 2;
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (long long)m * n * c) return;
  const int ch = (int)(k % c);
  const long long cell = k / c;
  const int i = (int)(cell / n), j = (int)(cell % n);
  auto ring = [&](int r, int col) { return bnd[((long long)r * w + col) * c + ch]; };
  double v = rhs[k];
  if (i == 0) v = __dsub_rn(v, __dmul_rn(weight, ring(0, j + 1)));
  if (i == m - 1) v = __dsub_rn(v, __dmul_rn(weight, ring(h - 1, j + 1)));
  if (j == 0) v = __dsub_rn(v, __dmul_rn(weight, ring(i + 1, 0)));
  if (j == n - 1) v = __dsub_rn(v, __dmul_rn(weight, ring(i + 1, w - 1)));
  out[k] = v;
}

__global__ void k_masked_rhs(double *__restrict__ f, const double *__restrict__ div,
                             const double *__restrict__ img, const unsigned char *__restrict__ unk,
                             int h, int w, double scale) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (long long)h * w) return;
  const int i = (int)(k / w), j = (int)(k % w);
  if (!unk[k]) {
    f[k] = 0.0;
    return;
  }
  double v = div[k];
  const int di[4] = {-1, 1, 0, 0}, dj[4] = {0, 0, -1, 1};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int y = i + di[q], x = j + dj[q];
    if (y < 0 || y >= h || x < 0 || x >= w) continue;  // unknowns never touch the border
    const long long g = (long long)y * w + x;
    if (!unk[g]) v = __dsub_rn(v, img[g]);
  }
  f[k] = __dmul_rn(scale, v);
}

// Guidance fields built on the fly (poisson.py:52-92 and the field set-up of
// seamless_clone, texture_flatten and illumination_change, poisson.py:306-431):
// the forward-difference gradient of an interleaved (H, W, C) image channel,
// combined per cell as the field kind says.
struct FieldView {
  gd_field_desc d;
  __device__ __forceinline__ double at(const double *img, int y, int x) const {
    return img[((long long)y * d.width + x) * d.channels + d.channel];
  }
  // forward differences of one image (operators.py:30-50)
  __device__ __forceinline__ void grad(const double *img, int y, int x, double &gx,
                                       double &gy) const {
    const double c = at(img, y, x);
    gx = x < d.width - 1 ? __dsub_rn(at(img, y, x + 1), c) : 0.0;
    gy = y < d.height - 1 ? __dsub_rn(at(img, y + 1, x), c) : 0.0;
  }
  __device__ __forceinline__ void field(int y, int x, double &gx, double &gy) const {
    double tx, ty;
    grad(d.target, y, x, tx, ty);
    switch (d.kind) {
      case GD_FIELD_IMPORT:
      case GD_FIELD_MIXED:
      case GD_FIELD_AVERAGE: {
        if (!d.select[(long long)y * d.width + x]) {  // GuidanceField.select: target outside
          gx = tx;
          gy = ty;
          return;
        }
        double sx, sy;
        grad(d.source, y, x, sx, sy);
        if (d.kind == GD_FIELD_IMPORT) {
          gx = sx;
          gy = sy;
        } else if (d.kind == GD_FIELD_MIXED) {  // mix_by_magnitude: the larger, source on ties
          gx = fabs(sx) >= fabs(tx) ? sx : tx;
          gy = fabs(sy) >= fabs(ty) ? sy : ty;
        } else {
          gx = __dmul_rn(0.5, __dadd_rn(sx, tx));
          gy = __dmul_rn(0.5, __dadd_rn(sy, ty));
        }
        return;
      }
      case GD_FIELD_WEIGHTED: {  // texture_flatten: gradient times the edge weights
        const double w = d.weights[(long long)y * d.width + x];
        gx = __dmul_rn(tx, w);
        gy = __dmul_rn(ty, w);
        return;
      }
      default: {  // illumination_change: alpha^beta * max(|g|, eps)^(-beta)
        const double m = sqrt(__dadd_rn(__dmul_rn(tx, tx), __dmul_rn(ty, ty)));
        const double f = __dmul_rn(d.alpha_pow_beta, pow(fmax(m, d.epsilon), -d.beta));
        gx = __dmul_rn(tx, f);
        gy = __dmul_rn(ty, f);
        return;
      }
    }
  }
};

// Divergence (operators.py:53-83) of the field over a window whose corner is
// image cell (row0, col0).  Interior cells take the backward differences; the
// window's outer ring is written 0 (no consumer of a window reads it) or, with
// `edges`, follows operators.py's edge rules for the window as a whole image.
//
// Both kernels form a cell's field once; its left neighbour's comes from the lane beside,
// whose first column only serves that.
__device__ __forceinline__ double guide_value(int i, int j, int h, int w, bool edges, double gx,
                                              double gxl, double gy, double gy_up) {
  if (!edges && (i == 0 || j == 0 || i == h - 1 || j == w - 1)) return 0.0;
  double dx = 0.0, dy = 0.0;
  if (w > 1) dx = j == 0 ? gx : j == w - 1 ? -gxl : __dsub_rn(gx, gxl);
  if (h > 1) dy = i == 0 ? gy : i == h - 1 ? -gy_up : __dsub_rn(gy, gy_up);
  return __dadd_rn(dx, dy);
}

// k_guidance_tile: a CTA's threads are rows of LANES columns (32, or the few that hold a
// narrow window), its first row serving the one below through shared memory, so that all
// its cells are in flight at once.  64 x 64 weighted field 6 us where a walk of eight rows
// takes 10; mixed 512 x 512 8 and 13 us, 1440 x 2160 50 and 55.
constexpr int kGuideThreads = 288;
template <int LANES>
constexpr int kTileRows = kGuideThreads / LANES - 1;
template <int LANES>
__global__ void __launch_bounds__(kGuideThreads)
    k_guidance_tile(double *__restrict__ out, FieldView fv, int row0, int col0, int h, int w) {
  __shared__ double gy_of[kGuideThreads];
  const int r = threadIdx.x / LANES, c = threadIdx.x % LANES;
  const int j = blockIdx.x * (LANES - 1) + c - 1;
  constexpr int rows = kTileRows<LANES>;
  for (int i0 = blockIdx.y * rows; i0 < h; i0 += gridDim.y * rows) {
    const int i = i0 + r - 1;
    const bool inside = i >= 0 && i < h && j >= 0 && j < w;
    double gx = 0.0, gy = 0.0;
    if (inside) fv.field(row0 + i, col0 + j, gx, gy);
    const double gxl = __shfl_up_sync(0xffffffffu, gx, 1);
    gy_of[threadIdx.x] = gy;
    __syncthreads();
    if (inside && r > 0 && c > 0)
      out[(long long)i * w + j] =
          guide_value(i, j, h, w, fv.d.edges, gx, gxl, gy, gy_of[threadIdx.x - LANES]);
    __syncthreads();
  }
}

// k_guidance_walk: a warp walks kGuideRows rows of 31 columns, the row above in registers.
// For weighted fields (two loads a cell) of at least kGuideWalks such walks, where there are
// warps enough to hide a walk's chain and a CTA per eight rows costs more than it hides:
// 1500 x 1500 (9212 walks) 20 us, 21 in tiles; 1440 x 2160 26 and 31; 4096 x 4096 151 and
// 190; but 1200 x 1600 (7800 walks) 19 both, 1100 x 1300 17 and 15.
constexpr int kGuideRows = 8, kGuideCols = 31, kGuideWarps = 8, kGuideWalks = 8192;
__global__ void __launch_bounds__(32 * kGuideWarps)
    k_guidance_walk(double *__restrict__ out, FieldView fv, int row0, int col0, int h, int w) {
  const int lane = threadIdx.x & 31;
  const int j = (blockIdx.x * kGuideWarps + (threadIdx.x >> 5)) * kGuideCols + lane - 1;
  if (j - lane >= w - 1) return;  // whole warp beyond the window
  const bool inside = j >= 0 && j < w;
  const int x = col0 + j;
  for (int i0 = blockIdx.y * kGuideRows; i0 < h; i0 += gridDim.y * kGuideRows) {
    const int i1 = min(i0 + kGuideRows, h);
    double gy_up = 0.0;
    if (i0 > 0 && inside) {
      double unused;
      fv.field(row0 + i0 - 1, x, unused, gy_up);
    }
    for (int i = i0; i < i1; ++i) {
      double gx = 0.0, gy = 0.0;
      if (inside) fv.field(row0 + i, x, gx, gy);
      const double gxl = __shfl_up_sync(0xffffffffu, gx, 1);
      if (inside && lane > 0)
        out[(long long)i * w + j] = guide_value(i, j, h, w, fv.d.edges, gx, gxl, gy, gy_up);
      gy_up = gy;
    }
  }
}

inline unsigned blocks(long long work) { return (unsigned)((work + 255) / 256); }

}  // namespace
}  // namespace gd

using namespace gd;

extern "C" const char *gd_last_error(void) { return g_error; }

extern "C" const char *gd_version(void) { return "gd_poisson 0.1 sm_100a"; }

extern "C" int gd_divergence(double *out, const double *gx, const double *gy, int32_t h, int32_t w,
                             cudaStream_t st) {
  GD_REQUIRE(out && gx && gy && h > 0 && w > 0, GD_ERR_ARG, "gd_divergence: bad arguments");
  k_divergence<<<blocks((long long)h * w), 256, 0, st>>>(out, gx, gy, h, w);
  GD_CHECK_LAUNCH();
  return GD_OK;
}

extern "C" int gd_gradient(double *gx, double *gy, const double *u, int32_t h, int32_t w,
                           cudaStream_t st) {
  GD_REQUIRE(gx && gy && u && h > 0 && w > 0, GD_ERR_ARG, "gd_gradient: bad arguments");
  k_gradient<<<blocks((long long)h * w), 256, 0, st>>>(gx, gy, u, h, w);
  GD_CHECK_LAUNCH();
  return GD_OK;
}

extern "C" int gd_fold_dirichlet(double *f, const double *div, const double *bnd, int32_t h,
                                 int32_t w, double scale, cudaStream_t st) {
  GD_REQUIRE(f && div && bnd && h > 2 && w > 2, GD_ERR_ARG, "gd_fold_dirichlet: bad arguments");
  k_fold<<<blocks((long long)(h - 2) * (w - 2)), 256, 0, st>>>(f, div, bnd, h, w, scale);
  GD_CHECK_LAUNCH();
  return GD_OK;
}

extern "C" int gd_fold_boundary(double *out, const double *rhs, const double *bnd, int32_t h,
                                int32_t w, int32_t channels, double spacing, cudaStream_t st) {
  GD_REQUIRE(out && rhs && bnd && h > 2 && w > 2 && channels > 0, GD_ERR_ARG,
             "gd_fold_boundary: bad arguments");
  GD_REQUIRE(spacing != 0.0 && std::isfinite(spacing), GD_ERR_ARG,
             "gd_fold_boundary: spacing must be finite and nonzero");
  const double weight = 1.0 / (spacing * spacing);
  k_fold_ring<<<blocks((long long)(h - 2) * (w - 2) * channels), 256, 0, st>>>(
      out, rhs, bnd, h, w, channels, weight);
  GD_CHECK_LAUNCH();
  return GD_OK;
}

extern "C" int gd_guidance_divergence(double *div, const gd_field_desc *field, int32_t row0,
                                      int32_t col0, int32_t h, int32_t w, cudaStream_t st) {
  GD_REQUIRE(div && field && field->target && h > 0 && w > 0 && (field->edges || (h > 2 && w > 2)),
             GD_ERR_ARG, "gd_guidance_divergence: bad arguments");
  const gd_field_desc &d = *field;
  GD_REQUIRE(d.kind >= GD_FIELD_IMPORT && d.kind <= GD_FIELD_ILLUMINATION, GD_ERR_ARG,
             "gd_guidance_divergence: unknown field kind %d", d.kind);
  GD_REQUIRE(d.height > 0 && d.width > 0 && d.channels > 0 && d.channel >= 0 &&
                 d.channel < d.channels,
             GD_ERR_ARG, "gd_guidance_divergence: bad image geometry");
  GD_REQUIRE(row0 >= 0 && col0 >= 0 && row0 + h <= d.height && col0 + w <= d.width, GD_ERR_ARG,
             "gd_guidance_divergence: window outside the image");
  GD_REQUIRE(d.kind > GD_FIELD_AVERAGE || (d.source && d.select), GD_ERR_ARG,
             "gd_guidance_divergence: cloning fields need a source and a selection");
  GD_REQUIRE(d.kind != GD_FIELD_WEIGHTED || d.weights, GD_ERR_ARG,
             "gd_guidance_divergence: weighted fields need weights");
  if (d.kind == GD_FIELD_WEIGHTED &&
      (long long)ceil_div(w, kGuideCols) * ceil_div(h, kGuideRows) >= kGuideWalks) {
    const dim3 grid(ceil_div(w, kGuideCols * kGuideWarps),
                    std::min(ceil_div(h, kGuideRows), 65535));
    k_guidance_walk<<<grid, 32 * kGuideWarps, 0, st>>>(div, FieldView{d}, row0, col0, h, w);
  } else {
    auto tiles = [&](auto lanes) {
      constexpr int L = decltype(lanes)::value;
      const dim3 grid(ceil_div(w, L - 1), std::min(ceil_div(h, kTileRows<L>), 65535));
      k_guidance_tile<L><<<grid, kGuideThreads, 0, st>>>(div, FieldView{d}, row0, col0, h, w);
    };
    if (w <= 3) tiles(std::integral_constant<int, 4>{});
    else if (w <= 7) tiles(std::integral_constant<int, 8>{});
    else if (w <= 15) tiles(std::integral_constant<int, 16>{});
    else tiles(std::integral_constant<int, 32>{});
  }
  GD_CHECK_LAUNCH();
  return GD_OK;
}

extern "C" int gd_masked_rhs(double *f, const double *div, const double *img, const uint8_t *unk,
                             int32_t h, int32_t w, double scale, cudaStream_t st) {
  GD_REQUIRE(f && div && img && unk && h > 0 && w > 0, GD_ERR_ARG, "gd_masked_rhs: bad arguments");
  k_masked_rhs<<<blocks((long long)h * w), 256, 0, st>>>(f, div, img, unk, h, w, scale);
  GD_CHECK_LAUNCH();
  return GD_OK;
}
