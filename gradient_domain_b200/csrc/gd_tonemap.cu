// Gradient-domain tone mapping on the device: the steps of hdr.py:73-185
// around the Neumann solve.
//
//   gd_tm_log_luminance   luminance = max(radiance . (0.2126, 0.7152, 0.0722), tiny)
//                         and its logarithm (hdr.py:168-170)
//   gd_tm_downsample      5-tap binomial blur with edge replication, every other
//                         sample (hdr.py:73-80, `_downsample`)
//   gd_tm_level_factor    one level of the attenuation field: central-difference
//                         gradient magnitude, its mean, the local factor, times the
//                         bilinear upsampling of the coarser level's factor
//                         (hdr.py:83-134, `_upsample`, `_central_gradient`,
//                         `attenuation_field`)
//   gd_tm_compose         exp(c - max c), chromatic ratios to the saturation power,
//                         99.5th percentile (NumPy's linear method), normalise and
//                         clip (hdr.py:178-185)
//
// Element-wise arithmetic uses explicitly rounded FP64 operations in the
// reference's order, so the results differ from NumPy's only where a library
// function (log, exp, pow, sqrt) or a reduction order differs.  Reductions are
// fixed trees (deterministic).  The percentile is exact: a radix selection on
// the order-preserving bit patterns of the non-negative image values.
// Scratch memory is the caller's (gd_tm_scratch_bytes).
//
// The kernels are bound by FP64 arithmetic (logarithms and powers) or by the
// arrays they stream; every reduction's last step is done where its result is
// needed (each CTA of the consumer sums the partials) or by the last CTA to
// finish, never by a launch of its own.  1440 x 2160 photograph, 8 levels
// (without the transform solve): 440 us, of which the factors 117, magnitudes 64, image
// and first histogram 56, percentile 80 (ncu); 690 us with eight histogram passes over
// the image and one-thread sums.

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "gd_internal.cuh"

namespace gd {
namespace {

constexpr int kTmThreads = 256;
constexpr int kTmBlocks = 296;  // fixed grid of the reductions: 2 x 148 SMs

inline unsigned blocks_for(long long n) { return (unsigned)((n + kTmThreads - 1) / kTmThreads); }

__device__ __forceinline__ double block_reduce_sum(double v) {
  __shared__ double part[kTmThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_down_sync(0xffffffffu, v, o));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) part[warp] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int k = 0; k < kTmThreads / 32; ++k) s = __dadd_rn(s, part[k]);
  return s;
}

__device__ __forceinline__ double block_reduce_max(double v) {
  __shared__ double part[kTmThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) part[warp] = v;
  __syncthreads();
  double s = -INFINITY;
  if (threadIdx.x == 0)
    for (int k = 0; k < kTmThreads / 32; ++k) s = fmax(s, part[k]);
  return s;
}

// Sum / maximum of `count` partials by a whole CTA, the same in every thread.
__device__ __forceinline__ double total_sum(const double *part, int count) {
  __shared__ double total;
  double s = 0.0;
  for (int k = threadIdx.x; k < count; k += kTmThreads) s = __dadd_rn(s, part[k]);
  s = block_reduce_sum(s);
  if (threadIdx.x == 0) total = s;
  __syncthreads();
  return total;
}

__device__ __forceinline__ double total_max(const double *part, int count) {
  __shared__ double total;
  double s = -INFINITY;
  for (int k = threadIdx.x; k < count; k += kTmThreads) s = fmax(s, part[k]);
  s = block_reduce_max(s);
  if (threadIdx.x == 0) total = s;
  __syncthreads();
  return total;
}

// Columns (log2) of a CTA over an array of width w: kTmThreads, or on a narrow array the
// power of two that holds it, the threads then being several rows (attenuation of
// 20000 x 20: 112 us with a row a CTA, 50 so; 6000 x 17 50 and 30).
inline int cta_columns(int w) {
  int c = 5;
  while ((1 << c) < kTmThreads && (1 << c) < w) ++c;
  return c;
}

// Where a thread of such a CTA works: rows row, row + rows, ... of columns column,
// column + columns, ... with `lg` = cta_columns(w).
struct Walk {
  int row, rows, column, columns;
  __device__ __forceinline__ explicit Walk(int lg) {
    const int each = kTmThreads >> lg;
    row = blockIdx.y * each + (threadIdx.x >> lg);
    rows = gridDim.y * each;
    column = (blockIdx.x << lg) + (threadIdx.x & ((1 << lg) - 1));
    columns = gridDim.x << lg;
  }
};

// CTAs over an h x w array, about `ctas` in all.
inline dim3 grid_2d(int h, int w, int ctas) {
  const int cols = 1 << cta_columns(w), each = kTmThreads / cols;
  const int gx = std::min((w + cols - 1) / cols, ctas);
  return dim3(gx, std::max(1, std::min((h + each - 1) / each, ctas / gx)));
}

__global__ void k_tm_luminance(double *__restrict__ logl, double *__restrict__ lum,
                               const double *__restrict__ rad, long long n) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const double *p = rad + 3 * k;
  double l = __dadd_rn(__dadd_rn(__dmul_rn(p[0], 0.2126), __dmul_rn(p[1], 0.7152)),
                       __dmul_rn(p[2], 0.0722));
  l = fmax(l, 2.2250738585072014e-308);  // np.finfo(float).tiny
  lum[k] = l;
  logl[k] = log(l);
}

// Output (i, j) = vertical blur of the horizontally blurred rows 2i-2 .. 2i+2
// at column 2j, both with edge replication and the weights 1 4 6 4 1 / 16
// summed left to right from zero, as the reference's `sum(...)` does.
// A thread makes kDownRows outputs of one column, so that a horizontally
// blurred row is formed for both outputs at once (3.5 blurred rows an output instead
// of 5; taller walks leave too few threads).
constexpr int kDownRows = 2;
__global__ void __launch_bounds__(kTmThreads) k_tm_downsample(double *__restrict__ out,
                                                              const double *__restrict__ in, int h,
                                                              int w, int lg) {
  const int oh = (h + 1) / 2, ow = (w + 1) / 2;
  const Walk walk(lg);
  const int j = walk.column;
  if (j >= ow) return;
  const double wgt[5] = {1.0 / 16.0, 4.0 / 16.0, 6.0 / 16.0, 4.0 / 16.0, 1.0 / 16.0};
  int col[5];
#pragma unroll
  for (int b = 0; b < 5; ++b) col[b] = min(max(2 * j + b - 2, 0), w - 1);
  auto blurred = [&](int r) {
    const double *row = in + (long long)min(max(r, 0), h - 1) * w;
    double hb = 0.0;
#pragma unroll
    for (int b = 0; b < 5; ++b) hb = __dadd_rn(hb, __dmul_rn(wgt[b], row[col[b]]));
    return hb;
  };
  for (int i0 = walk.row * kDownRows; i0 < oh; i0 += walk.rows * kDownRows) {
    const int i1 = min(i0 + kDownRows, oh);
    double hb[5];
#pragma unroll
    for (int a = 0; a < 3; ++a) hb[a + 2] = blurred(2 * i0 + a - 2);
    for (int i = i0; i < i1; ++i) {
#pragma unroll
      for (int a = 0; a < 3; ++a) hb[a] = hb[a + 2];
      hb[3] = blurred(2 * i + 1);
      hb[4] = blurred(2 * i + 2);
      double acc = 0.0;
#pragma unroll
      for (int a = 0; a < 5; ++a) acc = __dadd_rn(acc, __dmul_rn(wgt[a], hb[a]));
      out[(long long)i * ow + j] = acc;
    }
  }
}

// Division by the pyramid's doubled spacing: a power of two in the pyramid, where
// the product with its reciprocal is the same number.
struct Spacing {
  double value, inverse;  // inverse: exact reciprocal, or 0
  explicit Spacing(double v) : value(v), inverse(0.0) {
    int e = 0;
    if (std::frexp(v, &e) == 0.5 && e > -500 && e < 500) inverse = 1.0 / v;
  }
  __device__ __forceinline__ double divide(double a) const {
    return inverse != 0.0 ? __dmul_rn(a, inverse) : a / value;
  }
};

// Central-difference gradient magnitude of one level at (i, j), edges replicated.
__device__ __forceinline__ double tm_magnitude(const double *a, int h, int w, int i, int j,
                                               const Spacing &sp) {
  const double *row = a + (long long)i * w;
  const double gx = sp.divide(__dsub_rn(row[min(j + 1, w - 1)], row[max(j - 1, 0)]));
  const double gy = sp.divide(__dsub_rn(a[(long long)min(i + 1, h - 1) * w + j],
                                        a[(long long)max(i - 1, 0) * w + j]));
  return sqrt(__dadd_rn(__dmul_rn(gx, gx), __dmul_rn(gy, gy)));
}

__global__ void __launch_bounds__(kTmThreads) k_tm_mag_partials(double *__restrict__ part,
                                                                const double *__restrict__ a,
                                                                int h, int w, int lg,
                                                                Spacing sp) {
  const Walk walk(lg);
  double s = 0.0;
  for (int j = walk.column; j < w; j += walk.columns)
    for (int i = walk.row; i < h; i += walk.rows)
      s = __dadd_rn(s, tm_magnitude(a, h, w, i, j, sp));
  s = block_reduce_sum(s);
  if (threadIdx.x == 0) part[blockIdx.y * gridDim.x + blockIdx.x] = s;
}

// np.linspace(0, n_coarse - 1, n_fine)[i] (hdr.py:85-86); step = (n_coarse - 1) / (n_fine - 1)
__device__ __forceinline__ double tm_linspace(int i, int n_coarse, int n_fine, double step) {
  if (n_fine <= 1) return 0.0;
  if (i == n_fine - 1) return (double)(n_coarse - 1);
  return __dmul_rn((double)i, step);
}

__global__ void __launch_bounds__(kTmThreads)
    k_tm_factor(double *__restrict__ factor, const double *__restrict__ a,
                const double *__restrict__ coarse, const double *__restrict__ part, int nparts,
                int h, int w, int lg, int ch, int cw, Spacing sp, double alpha, double beta,
                double eps, double step_y, double step_x) {
  const double mean = total_sum(part, nparts) / (double)((long long)h * w);
  const double scale = __dmul_rn(alpha, fmax(mean, eps));
  const Walk walk(lg);
  for (int j = walk.column; j < w; j += walk.columns) {
    int c0 = 0, c1 = 0;
    double wx = 0.0;
    if (coarse) {
      const double rx = tm_linspace(j, cw, w, step_x);
      c0 = (int)floor(rx);
      c1 = min(c0 + 1, cw - 1);
      wx = __dsub_rn(rx, (double)c0);
    }
    for (int i = walk.row; i < h; i += walk.rows) {
      const double m = fmax(tm_magnitude(a, h, w, i, j, sp), eps);
      const double local = __dmul_rn(scale / m, pow(m / scale, beta));
      const long long k = (long long)i * w + j;
      if (!coarse) {
        factor[k] = local;
        continue;
      }
      const double ry = tm_linspace(i, ch, h, step_y);
      const int r0 = (int)floor(ry), r1 = min(r0 + 1, ch - 1);
      const double wy = __dsub_rn(ry, (double)r0);
      const double *p0 = coarse + (long long)r0 * cw, *p1 = coarse + (long long)r1 * cw;
      const double top = __dadd_rn(__dmul_rn(p0[c0], __dsub_rn(1.0, wx)), __dmul_rn(p0[c1], wx));
      const double bot = __dadd_rn(__dmul_rn(p1[c0], __dsub_rn(1.0, wx)), __dmul_rn(p1[c1], wx));
      const double up = __dadd_rn(__dmul_rn(top, __dsub_rn(1.0, wy)), __dmul_rn(bot, wy));
      factor[k] = __dmul_rn(up, local);
    }
  }
}

// ---------------------------------------------------------------------------
// Radix selection of the element of rank `rank` among n non-negative doubles:
// their IEEE bit patterns order like the values.  Two histograms of twelve bits
// (the first formed while the image is written) leave about n / 10000 candidates,
// which one more pass over the values collects into a list for its last CTA to
// search.  Values that crowd into one slice of 2^-12 of an octave (a nearly flat
// image) overflow the list: unless they are all the same value, four more histograms
// (which return at once otherwise) fix the other forty bits, by the whole grid like
// the first two.  (gd_tm_compose at 1440 x 2160: 29 ms when the last CTA searched such an
// image alone, 0.45 so, 0.17 where the list suffices.)

constexpr int kBins = 4096;
// Longer lists go on with the histograms: the one CTA that searches a list takes about
// 2.6 us per thousand values (61440 of a flat 128 x 160 image: 160 us).
constexpr int kListMax = 1 << 14;

struct SelectState {
  unsigned long long prefix;     // the leading bits chosen so far
  unsigned long long rank;       // of the wanted element among those that share them
  unsigned long long below;      // elements below all of those
  unsigned long long least, most;  // of those, as seen by the collection
  unsigned long long above;      // the smallest element seen beyond them
  unsigned long long selected, count_le, next;  // results
  unsigned long long matched;    // elements that share the prefix
  unsigned count;                // places of the list given out
  unsigned ticket;
  int done;
};

struct TmScratch {
  double *part;       // partials
  SelectState *sel;
  unsigned *hist;     // kBins counters
  unsigned long long *list;
};

constexpr size_t kSelOffset = 4096, kHistOffset = 8192, kListOffset = kHistOffset + kBins * 4;
constexpr size_t kScratchBytes = kListOffset + (size_t)kListMax * 8;

TmScratch tm_scratch(void *base) {
  char *p = static_cast<char *>(base);
  TmScratch s;
  s.part = reinterpret_cast<double *>(p);
  s.sel = reinterpret_cast<SelectState *>(p + kSelOffset);
  s.hist = reinterpret_cast<unsigned *>(p + kHistOffset);
  s.list = reinterpret_cast<unsigned long long *>(p + kListOffset);
  return s;
}

// Called by every CTA of a launch; true in the last one to arrive.
__device__ __forceinline__ bool last_cta(SelectState *s) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned ctas = gridDim.x * gridDim.y;
    last = atomicAdd(&s->ticket, 1u) == ctas - 1u;
    if (last) s->ticket = 0u;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// This CTA's counts into the launch's.
__device__ __forceinline__ void add_hist(unsigned *hist, const unsigned *h) {
  __syncthreads();
  for (int b = threadIdx.x; b < kBins; b += kTmThreads)
    if (h[b]) atomicAdd(&hist[b], h[b]);
}

// Inclusive sum over the lanes up to this one.
__device__ __forceinline__ unsigned long long warp_scan(unsigned long long v) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long q = __shfl_up_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) >= o) v += q;
  }
  return v;
}

// By the last CTA: the bin of `width` bits that holds the wanted rank extends the prefix;
// the counters are cleared for the next histogram.  `last`: these are the key's lowest bits
// (at most four, so that thread 0 holds every bin), and the selection is finished.
__device__ void choose_bin(SelectState *s, unsigned *hist, int width, bool last) {
  constexpr int kEach = kBins / kTmThreads;
  __shared__ unsigned long long warp_sums[kTmThreads / 32];
  __shared__ int bin_of;
  __shared__ unsigned long long below_bin;
  unsigned c[kEach];
  unsigned long long mine = 0;
  const unsigned long long rank = s->rank;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < kEach; ++q) {
    c[q] = __ldcg(&hist[threadIdx.x * kEach + q]);
    mine += c[q];
  }
  if (threadIdx.x == 0) {
    bin_of = kBins - 1;
    below_bin = 0;
  }
  const unsigned long long upto = warp_scan(mine);
  if (lane == 31) warp_sums[warp] = upto;
  __syncthreads();
  unsigned long long below = upto - mine;
  for (int q = 0; q < warp; ++q) below += warp_sums[q];
  if (rank >= below && rank < below + mine) {
    int q = 0;
    while (rank >= below + c[q]) below += c[q++];
    bin_of = threadIdx.x * kEach + q;
    below_bin = below;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned long long outer = s->prefix << width;
    s->prefix = outer | (unsigned long long)bin_of;
    s->rank = rank - below_bin;
    s->below += below_bin;
    if (last) {
      unsigned long long next = __ldcg(&s->above);
      int q = bin_of + 1;
      while (q < kEach && !c[q]) ++q;
      if (q < kEach) next = outer | (unsigned long long)q;
      s->selected = s->prefix;
      s->count_le = s->below + c[bin_of];
      s->next = next;
      s->done = 1;
    }
  }
#pragma unroll
  for (int q = 0; q < kEach; ++q) hist[threadIdx.x * kEach + q] = 0u;
}

// Histogram of the `width` bits at `shift` of the values that share the prefix above them.
// LATE: a histogram after the collection, which also notes the smallest value beyond the
// prefix (a longer prefix leaves no fewer values beyond it, so the last one's minimum holds).
template <bool LATE>
__global__ void __launch_bounds__(kTmThreads) k_select_hist(unsigned *__restrict__ hist,
                                                            const double *__restrict__ v,
                                                            long long n, SelectState *s,
                                                            int shift, int width) {
  if (LATE && s->done) return;
  __shared__ unsigned h[kBins];
  for (int b = threadIdx.x; b < kBins; b += kTmThreads) h[b] = 0u;
  __syncthreads();
  const unsigned long long prefix = s->prefix;
  const unsigned mask = (1u << width) - 1u;
  unsigned long long above = ~0ull;
  const long long stride = (long long)gridDim.x * kTmThreads;
  for (long long k0 = (long long)blockIdx.x * kTmThreads + threadIdx.x; k0 < n; k0 += 4 * stride) {
    unsigned long long key[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long k = k0 + u * stride;
      key[u] = k < n ? (unsigned long long)__double_as_longlong(v[k]) : ~prefix << (shift + width);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const unsigned long long top = key[u] >> (shift + width);
      if (top == prefix) atomicAdd(&h[(unsigned)(key[u] >> shift) & mask], 1u);
      else if (LATE && k0 + u * stride < n && top > prefix && key[u] < above) above = key[u];
    }
  }
  if constexpr (LATE) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long q = __shfl_down_sync(0xffffffffu, above, o);
      above = q < above ? q : above;
    }
    if ((threadIdx.x & 31) == 0 && above != ~0ull) atomicMin(&s->above, above);
  }
  add_hist(hist, h);
  if (last_cta(s)) choose_bin(s, hist, width, shift == 0);
}

// The wanted element among the keys get(0) .. get(m - 1) that share the prefix above
// `bits`, by the whole CTA: eight bits a round; then its count and successor among them.
template <class Get>
__device__ void search(SelectState *s, long long m, int bits, Get get) {
  __shared__ unsigned h[256];
  __shared__ unsigned long long sh_prefix, sh_rank, sh_le, sh_next;
  unsigned long long prefix = s->prefix, rank = s->rank;
  const unsigned long long outer = prefix;
  const int outer_bits = bits;
  while (bits > 0) {
    const int take = bits < 8 ? bits : 8;
    for (int b = threadIdx.x; b < 256; b += kTmThreads) h[b] = 0u;
    __syncthreads();
    for (long long k = threadIdx.x; k < m; k += kTmThreads) {
      const unsigned long long key = get(k);
      if (key >> bits == prefix) atomicAdd(&h[(key >> (bits - take)) & ((1u << take) - 1u)], 1u);
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // eight bins a lane; the rank lies in one of them
      unsigned long long mine = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q) mine += h[threadIdx.x * 8 + q];
      const unsigned long long upto = warp_scan(mine);
      unsigned long long below = upto - mine;
      if (rank >= below && rank < upto) {
        int q = 0;
        while (rank >= below + h[threadIdx.x * 8 + q]) below += h[threadIdx.x * 8 + q++];
        sh_prefix = prefix << take | (unsigned long long)(threadIdx.x * 8 + q);
        sh_rank = rank - below;
      }
    }
    __syncthreads();
    prefix = sh_prefix;
    rank = sh_rank;
    bits -= take;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    sh_le = 0;
    sh_next = ~0ull;
  }
  __syncthreads();
  unsigned long long le = 0, next = ~0ull;
  for (long long k = threadIdx.x; k < m; k += kTmThreads) {
    const unsigned long long key = get(k);
    if (key >> outer_bits != outer) continue;
    if (key <= prefix) ++le;
    else if (key < next) next = key;
  }
  atomicAdd(&sh_le, le);
  atomicMin(&sh_next, next);
  __syncthreads();
  if (threadIdx.x == 0) {
    s->selected = prefix;
    s->count_le = s->below + sh_le;
    s->next = sh_next < s->above ? sh_next : s->above;
    s->done = 1;
  }
}

// The values that share the prefix above `bits` into the list, and the smallest beyond
// them; the last CTA finishes the selection when they fit or are one value.
__global__ void __launch_bounds__(kTmThreads) k_select_collect(const double *__restrict__ v,
                                                               long long n, SelectState *s,
                                                               unsigned long long *list,
                                                               int bits) {
  const unsigned long long prefix = s->prefix;
  unsigned long long least = ~0ull, most = 0ull, above = ~0ull, matched = 0ull;
  const long long stride = (long long)gridDim.x * kTmThreads;
  for (long long k0 = (long long)blockIdx.x * kTmThreads + threadIdx.x; k0 < n; k0 += 4 * stride) {
    unsigned long long key[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long k = k0 + u * stride;
      key[u] = k < n ? (unsigned long long)__double_as_longlong(v[k]) : 0ull;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (k0 + u * stride >= n) break;
      const unsigned long long top = key[u] >> bits;
      if (top == prefix) {
        least = key[u] < least ? key[u] : least;
        most = key[u] > most ? key[u] : most;
        ++matched;
        // places are given out until the list is full; a full one is of no use
        if (__ldcg(&s->count) <= (unsigned)kListMax) {
          const unsigned at = atomicAdd(&s->count, 1u);
          if (at < (unsigned)kListMax) list[at] = key[u];
        }
      } else if (top > prefix && key[u] < above) {
        above = key[u];
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long q = __shfl_down_sync(0xffffffffu, least, o);
    least = q < least ? q : least;
    q = __shfl_down_sync(0xffffffffu, most, o);
    most = q > most ? q : most;
    q = __shfl_down_sync(0xffffffffu, above, o);
    above = q < above ? q : above;
    matched += __shfl_down_sync(0xffffffffu, matched, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (matched) atomicAdd(&s->matched, matched);
    if (least != ~0ull) atomicMin(&s->least, least);
    if (most) atomicMax(&s->most, most);
    if (above != ~0ull) atomicMin(&s->above, above);
  }
  if (!last_cta(s)) return;
  const unsigned long long m = __ldcg(&s->matched);
  if (__ldcg(&s->least) == __ldcg(&s->most)) {  // one value, however often
    if (threadIdx.x == 0) {
      s->selected = s->least;
      s->count_le = s->below + m;
      s->next = s->above;
      s->done = 1;
    }
  } else if (m <= (unsigned long long)kListMax) {
    search(s, (long long)m, bits, [&](long long k) { return __ldcg(&list[k]); });
  }
}

// Partial maxima of c; also clears the selection state and the histogram for the
// kernels that follow.
__global__ void __launch_bounds__(kTmThreads) k_tm_max_partials(double *__restrict__ part,
                                                                const double *__restrict__ c,
                                                                long long n, SelectState *sel,
                                                                unsigned *hist,
                                                                unsigned long long rank) {
  if (blockIdx.x == 0) {
    for (int b = threadIdx.x; b < kBins; b += kTmThreads) hist[b] = 0u;
    if (threadIdx.x == 0) {
      SelectState z = {};
      z.rank = rank;
      z.least = z.above = ~0ull;
      *sel = z;
    }
  }
  double s = -INFINITY;
  const long long stride = (long long)gridDim.x * kTmThreads;
  for (long long k0 = (long long)blockIdx.x * kTmThreads + threadIdx.x; k0 < n; k0 += 4 * stride) {
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = k0 + u * stride < n ? c[k0 + u * stride] : -INFINITY;
#pragma unroll
    for (int u = 0; u < 4; ++u) s = fmax(s, v[u]);
  }
  s = block_reduce_max(s);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// x ** 0.5 as pow gives it (0 for -0, inf for -inf), by the correctly rounded root.
__device__ __forceinline__ double power_half(double x) {
  return x == -INFINITY ? INFINITY : __dadd_rn(sqrt(x), 0.0);
}

// image = (radiance / luminance) ** saturation * exp(c - max c)   (hdr.py:178-182), and
// the histogram of its leading twelve bits.  ROOT: saturation is 0.5, its default.
template <bool ROOT>
__global__ void __launch_bounds__(kTmThreads)
    k_tm_image(double *__restrict__ image, const double *__restrict__ rad,
               const double *__restrict__ lum, const double *__restrict__ comp,
               const double *__restrict__ part, int nparts, long long n, double saturation,
               SelectState *sel, unsigned *hist) {
  __shared__ unsigned h[kBins];
  for (int b = threadIdx.x; b < kBins; b += kTmThreads) h[b] = 0u;
  const double top = total_max(part, nparts);
  const long long stride = (long long)gridDim.x * kTmThreads;
  for (long long k = (long long)blockIdx.x * kTmThreads + threadIdx.x; k < n; k += stride) {
    const double l = lum[k], cv = comp[k];
    double r[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) r[c] = rad[3 * k + c];
    const double result = exp(__dsub_rn(cv, top));
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double q = r[c] / l;
      const double v = __dmul_rn(ROOT ? power_half(q) : pow(q, saturation), result);
      image[3 * k + c] = v;
      atomicAdd(&h[(unsigned long long)__double_as_longlong(v) >> 52], 1u);
    }
  }
  add_hist(hist, h);
  if (last_cta(sel)) choose_bin(sel, hist, 12, false);
}

// np.percentile(image, q) with the linear method, then clip(image / peak, 0, 1).
__global__ void __launch_bounds__(kTmThreads) k_tm_finish(double *__restrict__ out,
                                                          const double *__restrict__ image,
                                                          long long n,
                                                          const SelectState *__restrict__ s,
                                                          long long lo_rank, double t, int vec) {
  const double a = __longlong_as_double((long long)s->selected);
  // rank lo + 1 is the selected value again when it repeats, else the next one up
  const double b = (s->count_le > (unsigned long long)lo_rank + 1ull || t == 0.0)
                       ? a
                       : __longlong_as_double((long long)s->next);
  // NumPy's _lerp: a + (b - a) t, or b - (b - a)(1 - t) for t >= 0.5
  const double diff = __dsub_rn(b, a);
  const double peak = t >= 0.5 ? __dsub_rn(b, __dmul_rn(diff, __dsub_rn(1.0, t)))
                               : __dadd_rn(a, __dmul_rn(diff, t));
  const double den = fmax(peak, 1e-12);
  auto map = [&](double v) { return fmin(fmax(v / den, 0.0), 1.0); };
  const long long first = (long long)blockIdx.x * kTmThreads + threadIdx.x;
  const long long stride = (long long)gridDim.x * kTmThreads;
  if (vec) {
    const long long pairs = n / 2;
    const double2 *src = reinterpret_cast<const double2 *>(image);
    double2 *dst = reinterpret_cast<double2 *>(out);
    for (long long k0 = first; k0 < pairs; k0 += 2 * stride) {
      double2 v[2];
#pragma unroll
      for (int u = 0; u < 2; ++u)
        v[u] = k0 + u * stride < pairs ? src[k0 + u * stride] : make_double2(0.0, 0.0);
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (k0 + u * stride < pairs) dst[k0 + u * stride] = make_double2(map(v[u].x), map(v[u].y));
    }
    if (first == 0 && (n & 1)) out[n - 1] = map(image[n - 1]);
  } else {
    for (long long k = first; k < n; k += stride) out[k] = map(image[k]);
  }
}

}  // namespace
}  // namespace gd

using namespace gd;

extern "C" size_t gd_tm_scratch_bytes(void) { return kScratchBytes; }

extern "C" int gd_tm_log_luminance(double *logl, double *lum, const double *radiance, int32_t h,
                                   int32_t w, cudaStream_t st) {
  GD_REQUIRE(logl && lum && radiance && h > 0 && w > 0, GD_ERR_ARG,
             "gd_tm_log_luminance: bad arguments");
  const long long n = (long long)h * w;
  k_tm_luminance<<<blocks_for(n), kTmThreads, 0, st>>>(logl, lum, radiance, n);
  GD_CHECK_LAUNCH();
  return GD_OK;
}

extern "C" int gd_tm_downsample(double *out, const double *in, int32_t h, int32_t w,
                                cudaStream_t st) {
  GD_REQUIRE(out && in && h > 0 && w > 0, GD_ERR_ARG, "gd_tm_downsample: bad arguments");
  const int oh = (h + 1) / 2, ow = (w + 1) / 2, lg = cta_columns(ow), cols = 1 << lg;
  const int rows = kTmThreads / cols * kDownRows;  // outputs of a CTA
  const dim3 grid((ow + cols - 1) / cols, std::min((oh + rows - 1) / rows, 65535));
  k_tm_downsample<<<grid, kTmThreads, 0, st>>>(out, in, h, w, lg);
  GD_CHECK_LAUNCH();
  return GD_OK;
}

extern "C" int gd_tm_level_factor(double *factor, const double *level, const double *coarse,
                                  int32_t h, int32_t w, int32_t ch, int32_t cw, double spacing,
                                  double alpha, double beta, double epsilon, void *scratch,
                                  cudaStream_t st) {
  GD_REQUIRE(factor && level && scratch && h > 0 && w > 0 && spacing > 0.0, GD_ERR_ARG,
             "gd_tm_level_factor: bad arguments");
  GD_REQUIRE(!coarse || (ch > 0 && cw > 0), GD_ERR_ARG, "gd_tm_level_factor: bad coarse level");
  const TmScratch s = tm_scratch(scratch);
  const Spacing sp(2.0 * spacing);
  const dim3 gm = grid_2d(h, w, kTmBlocks), gf = grid_2d(h, w, 8 * kTmBlocks);
  const int lg = cta_columns(w);
  const double step_y = h > 1 ? (double)(ch - 1) / (double)(h - 1) : 0.0;
  const double step_x = w > 1 ? (double)(cw - 1) / (double)(w - 1) : 0.0;
  k_tm_mag_partials<<<gm, kTmThreads, 0, st>>>(s.part, level, h, w, lg, sp);
  k_tm_factor<<<gf, kTmThreads, 0, st>>>(factor, level, coarse, s.part, (int)(gm.x * gm.y), h, w,
                                         lg, ch, cw, sp, alpha, beta, epsilon, step_y, step_x);
  GD_CHECK_LAUNCH();
  return GD_OK;
}

extern "C" int gd_tm_compose(double *out, double *image, const double *radiance,
                             const double *lum, const double *compressed, int32_t h, int32_t w,
                             double saturation, double percentile, void *scratch,
                             cudaStream_t st) {
  GD_REQUIRE(out && image && radiance && lum && compressed && scratch && h > 0 && w > 0,
             GD_ERR_ARG, "gd_tm_compose: bad arguments");
  GD_REQUIRE(percentile >= 0.0 && percentile <= 100.0, GD_ERR_ARG,
             "gd_tm_compose: percentile outside [0, 100]");
  const TmScratch s = tm_scratch(scratch);
  const long long n = (long long)h * w, n3 = 3 * n;
  // NumPy's linear percentile: index q/100 (n - 1), neighbours floor and floor + 1
  const double index = percentile / 100.0 * (double)(n3 - 1);
  const long long lo = (long long)index;
  const double t = index - (double)lo;
  const int wide = 4 * kTmBlocks;
  k_tm_max_partials<<<kTmBlocks, kTmThreads, 0, st>>>(s.part, compressed, n, s.sel, s.hist,
                                                      (unsigned long long)lo);
  auto *const make_image = saturation == 0.5 ? k_tm_image<true> : k_tm_image<false>;
  make_image<<<wide, kTmThreads, 0, st>>>(image, radiance, lum, compressed, s.part, kTmBlocks, n,
                                          saturation, s.sel, s.hist);
  k_select_hist<false><<<wide, kTmThreads, 0, st>>>(s.hist, image, n3, s.sel, 40, 12);
  k_select_collect<<<wide, kTmThreads, 0, st>>>(image, n3, s.sel, s.list, 40);
  for (int shift : {28, 16, 4, 0})  // return at once where the list was enough
    k_select_hist<true><<<kTmBlocks, kTmThreads, 0, st>>>(s.hist, image, n3, s.sel, shift,
                                                          shift ? 12 : 4);
  const int vec = ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(image)) & 15) == 0;
  k_tm_finish<<<8 * kTmBlocks, kTmThreads, 0, st>>>(out, image, n3, s.sel, lo, t, vec);
  GD_CHECK_LAUNCH();
  return GD_OK;
}
