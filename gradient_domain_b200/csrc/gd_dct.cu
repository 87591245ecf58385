// Exact Neumann Poisson solve by the discrete cosine transform: the algorithm
// of solvers.py:224-262 (dctn type 2, division by the eigenvalues
// 2 cos(pi i / m) + 2 cos(pi j / n) - 4 with the constant mode dropped, idctn),
// on the device with this library's own FFT kernels.
//
// Three passes over HBM, each CTA working on two lines (rows or columns) at
// once as one complex sequence z = a + i b:
//   rows:    load two rows of b, DCT-II along x, write the coefficients to T;
//   columns: load two columns of T, DCT-II along y, divide by the
//            eigenvalues, inverse transform (DCT-III) along y, write back;
//   rows:    load two rows of T, DCT-III along x, write u.
//
// One DCT-II of length N is one complex FFT of length N (Makhoul's
// reordering v = (x0, x2, x4, ..., x5, x3, x1), X_k = Re(e^{-i pi k/2N} V_k));
// two real lines share one FFT and are separated from its output by the
// Hermitian symmetry of each.  The inverse forms
// W_k = e^{i pi k/2N} (X_k - i X_{N-k}) and takes an inverse FFT (scaled by
// 1/N) whose output, read back through the reordering, is the line.  The
// coefficients here are half those of scipy's unnormalised DCT-II; the
// forward / inverse pair is exact either way and the solve only divides by
// the eigenvalues in between.
//
// Layout of T.  T[c][p] is the pair of columns 2c, 2c + 1 of the row at place p
// of the reordering along y, 16 bytes, p fastest.  The column pass then reads
// and writes contiguous memory in exactly the order its FFT wants, and since a
// row CTA takes the rows at places 2p and 2p + 1, what it reads or writes for a
// column pair is one whole 32-byte sector.  (With T stored row by row the column
// pass used half of every sector: 284 us a channel at 4096 x 4096.)
//
// The FFTs are mixed-radix, forward passes decimating in frequency (natural
// order in, digit-reversed out), inverse passes in time (digit-reversed in,
// natural out).  What bounds them is FP64 arithmetic and shared-memory
// bandwidth, so passes are few and large (radices up to 16), the first forward
// pass takes its operands straight from global memory, and the last inverse one
// writes its results there.  Lengths 64 .. 8192 that are powers of two run
// kernels whose every index is known at compile time, one radix-16 butterfly per
// thread and pass, with the values in registers from the loads to the
// coefficients: 3 passes and 2 exchanges for 4096 where radix 8 with staging
// took 4 passes and 6.  Other lengths take the radices of the cheapest
// factorisation (choose_passes) at run time.  Measured a channel: 4096 x 4096 275 us
// (75 rows, 122 columns, 83 rows under ncu; 490 with row-major T, radix 8 and staging),
// 1080 x 1920 97 us (181).

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "gd_internal.cuh"

namespace gd {
namespace dct {

constexpr int kMaxLen = 8192;   // longest line (128 KB of complex values in shared memory)
constexpr int kMaxPasses = 14;
constexpr int kThreads = 256;   // most threads of the run-time kernels; the large-prime ones' size

// One pass of a run-time transform: radix r on sub-transforms of length r m;
// step = N / (r m); div = ceil(2^32 / m) divides butterfly numbers by m.
struct Pass {
  int r, m, step;
  unsigned div;
};

struct Radices {
  int n = 0, count = 0;
  Pass p[kMaxPasses] = {};
};

// FP64 instructions per point of one pass of radix r (butterfly and twiddles,
// counted from the code below), plus what a pass costs besides: its exchange
// through shared memory and its barrier, worth about eight instructions a point.
// A model, measured against two to four other factorisations each: its choice was the
// fastest for squares of 1000 (43.6 us a solve, the next 55.9), 1440 (84, 94), 2160
// (190, 203) and 3000 (350, 389), and at 1920 (12 x 16 x 10, 160 us) 8 % behind 16 x 15 x 8.
inline double pass_cost(int r) {
  switch (r) {
    case 2: return 8 + 4.0;
    case 3: return 8 + 9.0;
    case 4: return 8 + 9.0;
    case 5: return 8 + 13.0;
    case 6: return 8 + 11.0;
    case 7: return 8 + 17.0;
    case 8: return 8 + 13.0;
    case 9: return 8 + 16.0;
    case 10: return 8 + 15.0;
    case 11: return 8 + 24.0;
    case 12: return 8 + 14.0;
    case 13: return 8 + 28.0;
    case 14: return 8 + 19.0;
    case 15: return 8 + 18.0;
    case 16: return 8 + 17.0;
    default: return 16 + 2.0 * r;  // a prime above 13: symmetric sums
  }
}

// Composite radices up to `cap`.
inline bool usable(int r, int cap) { return r <= cap || r == 5 || r == 7 || r == 11 || r == 13; }

// Passes for `lines` lines of length n.  A short line's CTA is a warp or two, and a
// launch of few of them is as long as one thread's butterflies: radices up to kSmallCap
// then (360 x 240: 35.6 us a solve with radices up to 16, 25.3 so; 240 x 320 32.5 and 27.3;
// 480 x 480 29.3 and 27.3), 16 where there are
// enough CTAs, or threads in one, to keep the FP64 pipes busy.
constexpr int kShortLine = 512, kFewLines = 8 * 148, kSmallCap = 8;
constexpr int kMaxDivisors = 64;  // of a length up to kMaxLen (7560 has most)
inline bool power_of_two_kernels(int n) { return n >= 64 && (n & (n - 1)) == 0; }
inline Radices choose_passes(int n, int lines) {
  const int cap = n < kShortLine && lines <= kFewLines ? kSmallCap : 16;
  Radices f;
  f.n = n;
  if (power_of_two_kernels(n)) return f;  // their passes are fixed
  // the divisors of n in ascending order, with the cost of each one's cheapest
  // factorisation and its first radix; a divisor without a small radix takes its least prime
  constexpr int kRoot = 91;  // above the square root of kMaxLen
  int divisor[kMaxDivisors], first[kMaxDivisors], divisors = 0;
  double cost[kMaxDivisors];
  unsigned char low[kRoot], high[kRoot];  // where divisor d and divisor n / d are
  for (int d = 1; d * d <= n; ++d)
    if (n % d == 0) {
      low[d] = (unsigned char)divisors;
      divisor[divisors++] = d;
    }
  for (int i = divisors - 1; i >= 0; --i) {
    high[divisor[i]] = low[divisor[i]];
    if (divisor[i] * divisor[i] == n) continue;
    high[divisor[i]] = (unsigned char)divisors;
    divisor[divisors++] = n / divisor[i];
  }
  // where the divisor d is, `other` being n / d
  auto place = [&](int d, int other) { return d <= other ? low[d] : high[other]; };
  cost[0] = 0.0;
  for (int i = 1; i < divisors; ++i) {
    const int d = divisor[i], other = n / d;
    cost[i] = -1.0;
    auto consider = [&](int r) {
      const double c = pass_cost(r) + cost[place(d / r, other * r)];
      if (cost[i] < 0.0 || c < cost[i]) {
        cost[i] = c;
        first[i] = r;
      }
    };
    for (int r = 16; r >= 2; --r)
      if (d % r == 0 && usable(r, cap)) consider(r);
    if (cost[i] < 0.0) {
      int q = 17;
      while (q * q <= d && d % q) q += 2;
      consider(d % q ? d : q);
    }
  }
  int r[kMaxPasses], count = 0;
  for (int m = n; m > 1; m /= r[count - 1]) r[count++] = first[place(m, n / m)];
  std::sort(r, r + count, [](int a, int b) { return a > b; });
  int L = n;
  for (int s = 0; s < count; ++s) {
    const int m = L / r[s];
    f.p[s] = Pass{r[s], m, n / L, m > 1 ? (unsigned)((0x100000000ull + m - 1) / m) : 0u};
    L = m;
  }
  f.count = count;
  return f;
}

inline bool has_large_prime(const Radices &r) {
  for (int s = 0; s < r.count; ++s)
    if (r.p[s].r > 16) return true;
  return false;
}

// Threads of a run-time kernel: one butterfly each in the pass that has most.
inline int gen_threads(const Radices &r) {
  if (has_large_prime(r)) return kThreads;
  int most = 1;
  for (int s = 0; s < r.count; ++s) most = std::max(most, r.n / r.p[s].r);
  return std::min(kThreads, (most + 31) / 32 * 32);
}

// Per-axis tables: FFT twiddles e^{-2 pi i m / N}, the DCT twiddles
// e^{-i pi k / 2N}, the eigenvalue terms 2 cos(pi k / N) and the place of
// frequency k in the digit-reversed output (N entries each).  The eigenvalue of
// mode (i, j) is formed as (2 cos(pi i / m) + 2 cos(pi j / n)) - 4 with
// cos(pi k / N) evaluated from the rounded product pi k, as solvers.py:253-258
// does: the smallest eigenvalues cancel most of their digits in that sum, and
// the solution's smoothest modes carry that rounding, so the same expression
// keeps the result within rounding of the reference's.
struct Axis {
  Radices rad;
  const double2 *tw;
  const double2 *post;
  const double *eig;
  const unsigned short *rev;
};

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {  // a * conj(b)
  return make_double2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 csub(double2 a, double2 b) {
  return make_double2(a.x - b.x, a.y - b.y);
}
// multiply by -i (forward, SIGN = -1) or +i (inverse, SIGN = +1)
template <int SIGN>
__device__ __forceinline__ double2 rot90(double2 a) {
  return SIGN < 0 ? make_double2(a.y, -a.x) : make_double2(-a.y, a.x);
}
// multiply by c + SIGN i s
template <int SIGN>
__device__ __forceinline__ double2 rot(double2 a, double c, double s) {
  return make_double2(c * a.x - SIGN * s * a.y, c * a.y + SIGN * s * a.x);
}

// In-register DFTs y_q = sum_j x_j e^{SIGN 2 pi i j q / R}, natural order.
template <int SIGN>
__device__ __forceinline__ void dft2(double2 &a, double2 &b) {
  const double2 t = a;
  a = cadd(t, b);
  b = csub(t, b);
}

template <int SIGN>
__device__ __forceinline__ void dft4(double2 &x0, double2 &x1, double2 &x2, double2 &x3) {
  const double2 a0 = cadd(x0, x2), a1 = csub(x0, x2);
  const double2 b0 = cadd(x1, x3), b1 = rot90<SIGN>(csub(x1, x3));
  x0 = cadd(a0, b0);
  x2 = csub(a0, b0);
  x1 = cadd(a1, b1);
  x3 = csub(a1, b1);
}

template <int SIGN>
__device__ __forceinline__ void dft8(double2 (&x)[8]) {
  constexpr double h = 0.70710678118654752440;  // sqrt(1/2)
  // two DFT-4 of the even and odd samples, then the radix-2 combination
  dft4<SIGN>(x[0], x[2], x[4], x[6]);
  dft4<SIGN>(x[1], x[3], x[5], x[7]);
  const double2 e[4] = {x[0], x[2], x[4], x[6]};
  double2 o[4] = {x[1], x[3], x[5], x[7]};
  o[1] = make_double2(h * (o[1].x - SIGN * o[1].y), h * (o[1].y + SIGN * o[1].x));
  o[2] = rot90<SIGN>(o[2]);
  o[3] = make_double2(h * (-o[3].x - SIGN * o[3].y), h * (-o[3].y + SIGN * o[3].x));
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    x[q] = cadd(e[q], o[q]);
    x[q + 4] = csub(e[q], o[q]);
  }
}

// 4 x 4: DFT-4 over samples a, a + 4, a + 8, a + 12, twiddles e^{SIGN 2 pi i a b / 16},
// DFT-4 over a; output b + 4 c.
template <int SIGN>
__device__ __forceinline__ void dft16(double2 (&x)[16]) {
  constexpr double c1 = 0.9238795325112867, s1 = 0.3826834323650898, h = 0.70710678118654752440;
#pragma unroll
  for (int a = 0; a < 4; ++a) dft4<SIGN>(x[a], x[a + 4], x[a + 8], x[a + 12]);
  // x[a + 4 b] now holds G[a][b]
  x[5] = rot<SIGN>(x[5], c1, s1);
  x[9] = make_double2(h * (x[9].x - SIGN * x[9].y), h * (x[9].y + SIGN * x[9].x));
  x[13] = rot<SIGN>(x[13], s1, c1);
  x[6] = make_double2(h * (x[6].x - SIGN * x[6].y), h * (x[6].y + SIGN * x[6].x));
  x[10] = rot90<SIGN>(x[10]);
  x[14] = make_double2(h * (-x[14].x - SIGN * x[14].y), h * (-x[14].y + SIGN * x[14].x));
  x[7] = rot<SIGN>(x[7], s1, c1);
  x[11] = make_double2(h * (-x[11].x - SIGN * x[11].y), h * (-x[11].y + SIGN * x[11].x));
  x[15] = rot<SIGN>(x[15], -c1, -s1);
#pragma unroll
  for (int b = 0; b < 4; ++b) dft4<SIGN>(x[4 * b], x[4 * b + 1], x[4 * b + 2], x[4 * b + 3]);
  // x[4 b + c] holds output b + 4 c: transpose in registers
#pragma unroll
  for (int b = 0; b < 4; ++b)
#pragma unroll
    for (int c = b + 1; c < 4; ++c) {
      const double2 t = x[4 * b + c];
      x[4 * b + c] = x[4 * c + b];
      x[4 * c + b] = t;
    }
}

// Odd primes by the symmetric sums and differences of the samples j and P - j.
template <int P>
struct Roots;  // cos and sin of 2 pi j / P, j = 1 .. (P - 1) / 2
template <>
struct Roots<3> {
  static __device__ __forceinline__ double c(int) { return -0.5; }
  static __device__ __forceinline__ double s(int) { return 0.8660254037844386; }
};
template <>
struct Roots<5> {
  static __device__ __forceinline__ double c(int j) {
    return j == 1 ? 0.30901699437494745 : -0.8090169943749475;
  }
  static __device__ __forceinline__ double s(int j) {
    return j == 1 ? 0.9510565162951535 : 0.5877852522924731;
  }
};
template <>
struct Roots<7> {
  static __device__ __forceinline__ double c(int j) {
    return j == 1 ? 0.6234898018587335 : j == 2 ? -0.2225209339563144 : -0.9009688679024191;
  }
  static __device__ __forceinline__ double s(int j) {
    return j == 1 ? 0.7818314824680298 : j == 2 ? 0.9749279121818236 : 0.4338837391175581;
  }
};
template <>
struct Roots<11> {
  static __device__ __forceinline__ double c(int j) {
    return j == 1   ? 0.8412535328311812
           : j == 2 ? 0.41541501300188644
           : j == 3 ? -0.14231483827328514
           : j == 4 ? -0.6548607339452851
                    : -0.9594929736144974;
  }
  static __device__ __forceinline__ double s(int j) {
    return j == 1   ? 0.5406408174555976
           : j == 2 ? 0.9096319953545183
           : j == 3 ? 0.9898214418809327
           : j == 4 ? 0.7557495743542583
                    : 0.28173255684142967;
  }
};
template <>
struct Roots<13> {
  static __device__ __forceinline__ double c(int j) {
    return j == 1   ? 0.8854560256532099
           : j == 2 ? 0.5680647467311558
           : j == 3 ? 0.12053668025532305
           : j == 4 ? -0.3546048870425356
           : j == 5 ? -0.7485107481711011
                    : -0.970941817426052;
  }
  static __device__ __forceinline__ double s(int j) {
    return j == 1   ? 0.46472317204376856
           : j == 2 ? 0.8229838658936564
           : j == 3 ? 0.992708874098054
           : j == 4 ? 0.9350162426854148
           : j == 5 ? 0.6631226582407952
                    : 0.23931566428755777;
  }
};

template <int P, int SIGN>
__device__ __forceinline__ void dft_prime(double2 (&x)[P]) {
  constexpr int H = (P - 1) / 2;
  double2 t[H], d[H];
  double2 sum = x[0];
#pragma unroll
  for (int j = 0; j < H; ++j) {
    t[j] = cadd(x[j + 1], x[P - 1 - j]);
    d[j] = csub(x[j + 1], x[P - 1 - j]);
    sum = cadd(sum, t[j]);
  }
  const double2 x0 = x[0];
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    double2 a = x0, b = make_double2(0.0, 0.0);
#pragma unroll
    for (int j = 1; j <= H; ++j) {
      const int e = (j * k) % P;                  // e^{2 pi i e / P}
      const int f = e <= H ? e : P - e;           // table index
      const double c = Roots<P>::c(f), s = e <= H ? Roots<P>::s(f) : -Roots<P>::s(f);
      a.x += c * t[j - 1].x;
      a.y += c * t[j - 1].y;
      b.x += s * d[j - 1].x;
      b.y += s * d[j - 1].y;
    }
    // X_k = a + SIGN i b, X_{P-k} = a - SIGN i b
    x[k] = make_double2(a.x - SIGN * b.y, a.y + SIGN * b.x);
    x[P - k] = make_double2(a.x + SIGN * b.y, a.y - SIGN * b.x);
  }
  x[0] = sum;
}

template <int R, int SIGN>
__device__ __forceinline__ void dft(double2 (&x)[R]);

// A B with coprime factors (Good-Thomas): no twiddles between the two sets of DFTs.
template <int A, int B, int SIGN>
__device__ __forceinline__ void dft_coprime(double2 (&x)[A * B]) {
  constexpr int R = A * B;
  double2 g[A][B];
#pragma unroll
  for (int n1 = 0; n1 < A; ++n1) {
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) g[n1][n2] = x[(B * n1 + A * n2) % R];
    dft<B, SIGN>(g[n1]);
  }
  constexpr auto inverse = [](int a, int m) {  // a^-1 mod m
    for (int i = 1; i < m; ++i)
      if ((a * i) % m == 1) return i;
    return 1;
  };
  constexpr int ea = B * inverse(B % A, A), eb = A * inverse(A % B, B);
#pragma unroll
  for (int k2 = 0; k2 < B; ++k2) {
    double2 y[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) y[n1] = g[n1][k2];
    dft<A, SIGN>(y);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) x[(k1 * ea + k2 * eb) % R] = y[k1];
  }
}

template <int SIGN>
__device__ __forceinline__ void dft9(double2 (&x)[9]) {
  double2 g[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
#pragma unroll
    for (int b = 0; b < 3; ++b) g[a][b] = x[a + 3 * b];
    dft_prime<3, SIGN>(g[a]);
  }
  g[1][1] = rot<SIGN>(g[1][1], 0.766044443118978, 0.6427876096865394);
  g[1][2] = rot<SIGN>(g[1][2], 0.17364817766693036, 0.984807753012208);
  g[2][1] = rot<SIGN>(g[2][1], 0.17364817766693036, 0.984807753012208);
  g[2][2] = rot<SIGN>(g[2][2], -0.9396926207859084, 0.3420201433256687);
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    double2 y[3] = {g[0][b], g[1][b], g[2][b]};
    dft_prime<3, SIGN>(y);
#pragma unroll
    for (int c = 0; c < 3; ++c) x[b + 3 * c] = y[c];
  }
}

template <int R, int SIGN>
__device__ __forceinline__ void dft(double2 (&x)[R]) {
  if constexpr (R == 2) dft2<SIGN>(x[0], x[1]);
  else if constexpr (R == 4) dft4<SIGN>(x[0], x[1], x[2], x[3]);
  else if constexpr (R == 8) dft8<SIGN>(x);
  else if constexpr (R == 16) dft16<SIGN>(x);
  else if constexpr (R == 9) dft9<SIGN>(x);
  else if constexpr (R == 6) dft_coprime<2, 3, SIGN>(x);
  else if constexpr (R == 10) dft_coprime<2, 5, SIGN>(x);
  else if constexpr (R == 12) dft_coprime<4, 3, SIGN>(x);
  else if constexpr (R == 14) dft_coprime<2, 7, SIGN>(x);
  else if constexpr (R == 15) dft_coprime<3, 5, SIGN>(x);
  else if constexpr (R > 1) dft_prime<R, SIGN>(x);
}

// x[q] *= w^q (forward) or conj(w)^q (inverse), q < R, where power(q) gives w^q for
// q = 1, 2, 3, 4, 8, 12, from a table or at most one product; every other power is one
// product of two of these.  (Powers by repeated products from w alone carried up to eight
// roundings into the smoothest modes, whose small eigenvalues magnify them: error of a
// tone-mapping solve against 80-bit transforms, 720 x 1280 4.3e-13 then, 1.5e-13 so;
// 1024 x 1024 2.5e-13 then, 1.8e-13 so.)
template <int R, int SIGN, class Power>
__device__ __forceinline__ void twiddle(double2 (&x)[R], Power power) {
  auto mul = [](double2 a, double2 t) { return SIGN < 0 ? cmul(a, t) : cmulc(a, t); };
  const double2 w1 = power(1);
  x[1] = mul(x[1], w1);
  if constexpr (R > 2) {
    const double2 w2 = power(2);
    x[2] = mul(x[2], w2);
    if constexpr (R > 3) {
      const double2 w3 = power(3);
      x[3] = mul(x[3], w3);
#pragma unroll
      for (int b = 4; b < R; b += 4) {
        const double2 base = power(b);
        x[b] = mul(x[b], base);
        if (b + 1 < R) x[b + 1] = mul(x[b + 1], cmul(base, w1));
        if (b + 2 < R) x[b + 2] = mul(x[b + 2], cmul(base, w2));
        if (b + 3 < R) x[b + 3] = mul(x[b + 3], cmul(base, w3));
      }
    }
  }
}

// Shared-memory slot of element idx.  A warp's 16-byte accesses are served eight
// lanes at a time, without conflict when the eight hit different slots modulo
// eight; storing element idx at idx ^ (XOR of the octal digits above the lowest)
// gives that to any eight elements that differ in three consecutive index bits,
// so to every butterfly stride of a power-of-two length.  at(i ^ j) = at(i) ^ at(j).
__device__ __forceinline__ int fold(int idx) {
  const int x = idx >> 3;
  return (x ^ (x >> 3) ^ (x >> 6) ^ (x >> 9)) & 7;
}
__device__ __forceinline__ int at(int idx) { return idx ^ fold(idx); }

// Where sample j of a line sits in Makhoul's even/odd reordering, and the sample
// at place p.
__device__ __forceinline__ int mak_sample(int p, int n) {
  return p < (n + 1) / 2 ? 2 * p : 2 * (n - 1 - p) + 1;
}

// Forward DCT coefficients of the two lines packed in Z, at frequency k and
// its partner n - k (k in 1 .. n-1): X_a[k], X_b[k], X_a[n-k], X_b[n-k].
struct Coef4 {
  double ak, bk, an, bn;
};

// tk = e^{-i pi k / 2n}; its partner e^{-i pi (n-k) / 2n} is (-tk.y, -tk.x)
__device__ __forceinline__ Coef4 split(double2 zk, double2 zn, double2 tk) {
  // A_k = (Z_k + conj Z_{n-k}) / 2, B_k = (Z_k - conj Z_{n-k}) / 2i; A_{n-k} = conj A_k
  const double2 A = make_double2(0.5 * (zk.x + zn.x), 0.5 * (zk.y - zn.y));
  const double2 B = make_double2(0.5 * (zk.y + zn.y), 0.5 * (zn.x - zk.x));
  Coef4 c;
  c.ak = tk.x * A.x - tk.y * A.y;   // Re(t_k A_k)
  c.bk = tk.x * B.x - tk.y * B.y;
  c.an = -tk.y * A.x - tk.x * A.y;  // Re(t_{n-k} conj A_k)
  c.bn = -tk.y * B.x - tk.x * B.y;
  return c;
}

// W_k = conj(t_k) (X_k - i X_{n-k}) for both lines, packed as W_a + i W_b.
__device__ __forceinline__ double2 pack_inverse(double xa, double xan, double xb, double xbn,
                                                double2 tk) {
  // conj(t) (x - i y) = (c + i s)(x - i y) with t = c - i s
  const double c = tk.x, s = -tk.y;
  const double2 wa = make_double2(c * xa + s * xan, s * xa - c * xan);
  const double2 wb = make_double2(c * xb + s * xbn, s * xb - c * xbn);
  return make_double2(wa.x - wb.y, wa.y + wb.x);
}

// The two rows of a pair: places 2p and 2p + 1 of the reordering along y.
struct RowPair {
  int p0, ra, rb;
  bool two;
  __device__ __forceinline__ RowPair(int pair, int h) {
    p0 = 2 * pair;
    two = p0 + 1 < h;
    ra = mak_sample(p0, h);
    rb = two ? mak_sample(p0 + 1, h) : ra;
  }
};

constexpr int kPowers = 4;  // rows of a pass in a power-of-two length's twiddle table

// ---------------------------------------------------------------------------
// Powers of two, 64 .. 8192: N / 16 threads with sixteen values each, below 512 N / 8 with
// eight, as many pairs of lines in a CTA as a warp holds.  (A launch of few short lines is as
// long as one thread's chain: 64 x 64 and 256 x 256 took 25.2 and 27.5 us a solve by the
// run-time passes, 17.0 and 17.4 so; 8192 x 64 56 and 38 us.)
// Passes: radix V while the sub-transform allows, the last of radix 2^(LOG mod LV)
// (or V).  After the forward passes thread t of a pair holds the frequencies t + TP i.
template <int LOG>
struct P2 {
  static constexpr int LV = LOG < 9 ? 3 : 4, V = 1 << LV;
  static constexpr int N = 1 << LOG, TP = N / V;
  static constexpr int PB = TP < 32 ? 32 / TP : 1;  // pairs of lines in a CTA
  static constexpr int REM = LOG % LV ? LOG % LV : LV;
  static constexpr int LR = 1 << REM;               // radix of the last pass
  static constexpr int G = V / LR;                  // its butterflies per thread
  static constexpr int MID = (LOG - REM) / LV - 1;  // radix-V passes after the first
  static constexpr int threads = TP * PB;
  static constexpr size_t smem = (size_t)PB * N * sizeof(double2);

  // this thread's number in its pair of lines, the pair's number and its shared memory
  static __device__ __forceinline__ int lane() { return threadIdx.x & (TP - 1); }
  static __device__ __forceinline__ int pair() { return blockIdx.x * PB + threadIdx.x / TP; }
  static __device__ __forceinline__ double2 *line(double2 *smem) {
    return smem + threadIdx.x / TP * N;
  }
  static inline unsigned ctas(int pairs) { return (unsigned)((pairs + PB - 1) / PB); }

  // The table of the twiddled passes (k_dct_tables): for pass s, a row of its TP >> LV s
  // butterflies' e^{-2 pi i k q / L} for each of q = 1, 2, 4, 8, so that a warp reads whole
  // lines.  Rows for q = 3 and 12 too cost more than the products (4096 x 4096: 296 and
  // 280 us a solve) and gained no accuracy to speak of.
  template <int S>
  static constexpr int table_offset() {
    int o = 0;
    for (int s = 0; s < S; ++s) o += kPowers * (TP >> (LV * s));
    return o;
  }
  static constexpr int table_len = table_offset<MID + 1>();
  static_assert(table_len <= N, "the table takes the place of the plain twiddles");
  template <int SIGN, int S>
  static __device__ __forceinline__ void twiddle_pass(double2 (&x)[V], const double2 *tab) {
    constexpr int M = TP >> (LV * S);
    const double2 *p = tab + table_offset<S>() + (lane() & (M - 1));
    const double2 w1 = p[0], w2 = p[M], w4 = p[2 * M];
    double2 w8 = w4;
    if constexpr (V == 16) w8 = p[3 * M];
    twiddle<V, SIGN>(x, [&](int q) {
      return q == 1   ? w1
             : q == 2 ? w2
             : q == 3 ? cmul(w2, w1)
             : q == 4 ? w4
             : q == 8 ? w8
                      : cmul(w8, w4);
    });
  }
  // first element of this thread's butterfly in middle pass s (stride TP >> 4 s)
  template <int S>
  static __device__ __forceinline__ int mid_base() {
    constexpr int M = TP >> (LV * S);
    const int t = lane();
    return ((t & ~(M - 1)) << LV) | (t & (M - 1));
  }
  // place of frequency f (< N / LR) in the digit-reversed order
  static __device__ __forceinline__ int last_base(int f) {
    int pos = 0;
#pragma unroll
    for (int s = 0; s <= MID; ++s) pos |= ((f >> (LV * s)) & (V - 1)) << (LOG - LV * s - LV);
    return pos;
  }
  template <int SIGN, int S>
  static __device__ __forceinline__ void mid_pass(double2 *z, const double2 *tab) {
    constexpr int M = TP >> (LV * S);
    const int b = at(mid_base<S>());
    double2 x[V];
#pragma unroll
    for (int j = 0; j < V; ++j) x[j] = z[b ^ at(j * M)];
    if constexpr (SIGN > 0) twiddle_pass<1, S>(x, tab);
    dft<V, SIGN>(x);
    if constexpr (SIGN < 0) twiddle_pass<-1, S>(x, tab);
#pragma unroll
    for (int j = 0; j < V; ++j) z[b ^ at(j * M)] = x[j];
    __syncthreads();
  }
  // x[j] = v[t + TP j] -> x[i] = V[t + TP i]; the shared memory may be in use by
  // this thread's own columns (places = t mod TP) on entry
  static __device__ __forceinline__ void forward(double2 (&x)[V], double2 *z,
                                                 const double2 *tab) {
    const int b = at(lane());
    dft<V, -1>(x);
    twiddle_pass<-1, 0>(x, tab);
#pragma unroll
    for (int q = 0; q < V; ++q) z[b ^ at(q * TP)] = x[q];
    __syncthreads();
    if constexpr (MID >= 1) mid_pass<-1, 1>(z, tab);
    if constexpr (MID >= 2) mid_pass<-1, 2>(z, tab);
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int p = last_base(lane() + TP * g);
      double2 y[LR];
#pragma unroll
      for (int j = 0; j < LR; ++j) y[j] = z[at(p + j)];
      dft<LR, -1>(y);
#pragma unroll
      for (int q = 0; q < LR; ++q) x[g + G * q] = y[q];
    }
    __syncthreads();
  }
  // the inverse (unscaled); the shared memory is free on entry
  static __device__ __forceinline__ void inverse(double2 (&x)[V], double2 *z,
                                                 const double2 *tab) {
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int p = last_base(lane() + TP * g);
      double2 y[LR];
#pragma unroll
      for (int q = 0; q < LR; ++q) y[q] = x[g + G * q];
      dft<LR, 1>(y);
#pragma unroll
      for (int j = 0; j < LR; ++j) z[at(p + j)] = y[j];
    }
    __syncthreads();
    if constexpr (MID >= 2) mid_pass<1, 2>(z, tab);
    if constexpr (MID >= 1) mid_pass<1, 1>(z, tab);
    const int b = at(lane());
#pragma unroll
    for (int q = 0; q < V; ++q) x[q] = z[b ^ at(q * TP)];
    twiddle_pass<1, 0>(x, tab);
    dft<V, 1>(x);
  }
};

// e^{-i pi i / 32}, i = 0 .. 15: the DCT twiddle of frequency t + TP i is that of t times
// this of 16 i / V.
__device__ __forceinline__ double2 c32(int i) {
  constexpr double c[17] = {1.0, 0.9951847266721969, 0.9807852804032304, 0.9569403357322088,
                            0.9238795325112867, 0.881921264348355, 0.8314696123025452,
                            0.773010453362737, 0.7071067811865476, 0.6343932841636455,
                            0.5555702330196022, 0.47139673682599764, 0.3826834323650898,
                            0.2902846772544624, 0.19509032201612828, 0.0980171403295606, 0.0};
  return make_double2(c[i], -c[16 - i]);
}

// CTAs per SM for 128 registers a thread.
template <int LOG>
constexpr int kP2Ctas = P2<LOG>::threads >= 512 ? 1 : 512 / P2<LOG>::threads;

template <int LOG>
__global__ void __launch_bounds__(P2<LOG>::threads, kP2Ctas<LOG>)
    k_rows_p2(double2 *__restrict__ T, int hp, const double *__restrict__ bsrc, long long bpitch,
              int h, const double2 *__restrict__ tab, const double2 *__restrict__ post) {
  using F = P2<LOG>;
  constexpr int N = F::N, TP = F::TP, V = F::V;
  extern __shared__ double2 smem[];
  double2 *const z = F::line(smem);
  const int t = F::lane(), pairs = (h + 1) / 2;
  const bool live = F::PB == 1 || F::pair() < pairs;  // else the last pair again, not stored
  const RowPair rp(live ? F::pair() : pairs - 1, h);
  const double *ra = bsrc + rp.ra * bpitch, *rb = bsrc + rp.rb * bpitch;
  double2 x[V];
  double2 va[V / 2], vb[V / 2];
  if (((reinterpret_cast<uintptr_t>(ra) | reinterpret_cast<uintptr_t>(rb)) & 15) == 0) {
#pragma unroll
    for (int j = 0; j < V / 2; ++j) {
      va[j] = reinterpret_cast<const double2 *>(ra)[t + TP * j];
      vb[j] = reinterpret_cast<const double2 *>(rb)[t + TP * j];
    }
  } else {
#pragma unroll
    for (int j = 0; j < V / 2; ++j) {
      const int m = 2 * (t + TP * j);
      va[j] = make_double2(ra[m], ra[m + 1]);
      vb[j] = make_double2(rb[m], rb[m + 1]);
    }
  }
  // the even samples are this thread's, the odd ones belong to place N - 1 - m
#pragma unroll
  for (int j = 0; j < V / 2; ++j) {
    x[j] = make_double2(va[j].x, rp.two ? vb[j].x : 0.0);
    z[at(N - 1 - (t + TP * j))] = make_double2(va[j].y, rp.two ? vb[j].y : 0.0);
  }
  __syncthreads();
#pragma unroll
  for (int j = V / 2; j < V; ++j) x[j] = z[at(t + TP * j)];
  F::forward(x, z, tab);
#pragma unroll
  for (int i = 0; i < V; ++i) z[at(t + TP * i)] = x[i];
  __syncthreads();
  // lanes 2l and 2l + 1 hold one column pair: the even one takes row a, the odd one row b
  const int odd = t & 1;
  double2 *dst = T + (long long)(t >> 1) * hp + rp.p0 + odd;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const double2 zk = x[i], zn = z[at((N - (t + TP * i)) & (N - 1))];
    const Coef4 f = split(zk, zn, cmul(post[t], c32(16 / V * i)));
    const double xa = f.ak, xb = f.bk;
    const double got = __shfl_xor_sync(0xffffffffu, odd ? xa : xb, 1);
    const double2 v = odd ? make_double2(got, xb) : make_double2(xa, got);
    if (live && (!odd || rp.two)) dst[(long long)(TP / 2 * i) * hp] = v;
  }
}

template <int LOG>
__global__ void __launch_bounds__(P2<LOG>::threads, kP2Ctas<LOG>)
    k_cols_p2(double2 *__restrict__ T, int hp, int w, const double2 *__restrict__ tab,
              const double2 *__restrict__ post, const double *__restrict__ eig,
              const double *__restrict__ eig_w) {
  using F = P2<LOG>;
  constexpr int N = F::N, TP = F::TP, V = F::V;
  extern __shared__ double2 smem[];
  double2 *const z = F::line(smem);
  const int t = F::lane(), pairs = (w + 1) / 2;
  const bool live = F::PB == 1 || F::pair() < pairs;  // else zeros, not stored
  const int pair = live ? F::pair() : 0, c0 = 2 * pair;
  double2 *col = T + (long long)pair * hp;
  double2 x[V];
#pragma unroll
  for (int j = 0; j < V; ++j) x[j] = live ? col[t + TP * j] : make_double2(0.0, 0.0);
  const double ew_a = eig_w[c0], ew_b = c0 + 1 < w ? eig_w[c0 + 1] : 0.0;
  F::forward(x, z, tab);
  // pairs (k, N - k) with k = t + TP i, i < V / 2: the upper halves change hands
#pragma unroll
  for (int i = V / 2; i < V; ++i) z[at(t + TP * i)] = x[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < V / 2; ++i) {
    const int k = t + TP * i;
    const double ek = eig[k];
    if (k == 0) {
      // X_a[0] = Re Z_0, X_b[0] = Im Z_0, W_0 = X_0; mode (0, 0) is the constant: zero
      const double la = (ek + ew_a) - 4.0, lb = (ek + ew_b) - 4.0;
      x[0] = make_double2(c0 == 0 ? 0.0 : x[0].x / la, x[0].y / lb);
    } else {
      const int pn = at(N - k);
      const double en = eig[N - k];
      const double2 tk = cmul(post[t], c32(16 / V * i));
      Coef4 c = split(x[i], z[pn], tk);
      c.ak /= (ek + ew_a) - 4.0;
      c.bk /= (ek + ew_b) - 4.0;
      c.an /= (en + ew_a) - 4.0;
      c.bn /= (en + ew_b) - 4.0;
      x[i] = pack_inverse(c.ak, c.an, c.bk, c.bn, tk);
      z[pn] = pack_inverse(c.an, c.ak, c.bn, c.bk, make_double2(-tk.y, -tk.x));
    }
  }
  if (t == 0) {  // k = N / 2 is its own partner
    const double ek = eig[N / 2];
    const double2 tk = post[N / 2];
    Coef4 c = split(x[V / 2], x[V / 2], tk);
    c.ak /= (ek + ew_a) - 4.0;
    c.bk /= (ek + ew_b) - 4.0;
    z[at(N / 2)] = pack_inverse(c.ak, c.ak, c.bk, c.bk, tk);
  }
  __syncthreads();
#pragma unroll
  for (int i = V / 2; i < V; ++i) x[i] = z[at(t + TP * i)];
  __syncthreads();
  F::inverse(x, z, tab);
  constexpr double inv_n = 1.0 / (double)N;
#pragma unroll
  for (int j = 0; j < V; ++j)
    if (live) col[t + TP * j] = make_double2(x[j].x * inv_n, x[j].y * inv_n);
}

template <int LOG>
__global__ void __launch_bounds__(P2<LOG>::threads, kP2Ctas<LOG>)
    k_irows_p2(double *__restrict__ u, long long upitch, const double2 *__restrict__ T, int hp,
               int h, const double2 *__restrict__ tab, const double2 *__restrict__ post) {
  using F = P2<LOG>;
  constexpr int N = F::N, TP = F::TP, V = F::V;
  extern __shared__ double2 smem[];
  double2 *const z = F::line(smem);
  const int t = F::lane(), odd = t & 1, pairs = (h + 1) / 2;
  const bool live = F::PB == 1 || F::pair() < pairs;  // else the last pair again, not stored
  const RowPair rp(live ? F::pair() : pairs - 1, h);
  // the even lane of a column pair loads row a, the odd one row b
  const double2 *src = T + (long long)(t >> 1) * hp + rp.p0 + (rp.two ? odd : 0);
  double2 x[V];
#pragma unroll
  for (int i = 0; i < V; ++i) x[i] = src[(long long)(TP / 2 * i) * hp];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const double got = __shfl_xor_sync(0xffffffffu, odd ? x[i].x : x[i].y, 1);
    x[i] = odd ? make_double2(got, x[i].y) : make_double2(x[i].x, got);  // (X_a[k], X_b[k])
    if (!rp.two) x[i].y = 0.0;
    z[at(t + TP * i)] = x[i];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int k = t + TP * i;
    double2 xn = z[at((N - k) & (N - 1))];
    if (k == 0) xn = make_double2(0.0, 0.0);  // X_N = 0
    x[i] = pack_inverse(x[i].x, xn.x, x[i].y, xn.y, cmul(post[t], c32(16 / V * i)));
  }
  __syncthreads();
  F::inverse(x, z, tab);
  constexpr double inv_n = 1.0 / (double)N;
  // place N - 1 - m holds the odd sample of pair m
#pragma unroll
  for (int j = V / 2; j < V; ++j) z[at(t + TP * j)] = x[j];
  __syncthreads();
  if (!live) return;
  double *ua = u + rp.ra * upitch, *ub = u + rp.rb * upitch;
  const bool vec = ((reinterpret_cast<uintptr_t>(ua) | reinterpret_cast<uintptr_t>(ub)) & 15) == 0;
#pragma unroll
  for (int j = 0; j < V / 2; ++j) {
    const int m = t + TP * j;
    const double2 o = z[at(N - 1 - m)];
    const double2 a = make_double2(x[j].x * inv_n, o.x * inv_n);
    const double2 b = make_double2(x[j].y * inv_n, o.y * inv_n);
    if (vec) {
      reinterpret_cast<double2 *>(ua)[m] = a;
      if (rp.two) reinterpret_cast<double2 *>(ub)[m] = b;
    } else {
      ua[2 * m] = a.x;
      ua[2 * m + 1] = a.y;
      if (rp.two) {
        ub[2 * m] = b.x;
        ub[2 * m + 1] = b.y;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Any other length: the passes of choose_passes at run time, in place in shared
// memory.  PRIME: the length has a prime factor above 13 (a separate
// instantiation, so that the register buffer of prime_pass does not weigh on the
// common lengths).

// Butterfly t of a pass: its first element and its twiddle index within the sub-transform.
__device__ __forceinline__ int butterfly(const Pass &p, int t, int *k) {
  const int blk = p.div ? (int)__umulhi((unsigned)t, p.div) : t;
  *k = t - blk * p.m;
  return blk * p.r * p.m + *k;
}

// Decimation in frequency; src(i) gives element i (shared memory, or the line itself
// in the first pass).
template <int R, class Src>
__device__ __forceinline__ void dif_pass(double2 *z, int n, const Pass &p, const double2 *tw,
                                         Src src) {
  for (int t = threadIdx.x; t < n / R; t += blockDim.x) {
    int k;
    const int base = butterfly(p, t, &k);
    double2 x[R];
#pragma unroll
    for (int j = 0; j < R; ++j) x[j] = src(base + j * p.m);
    dft<R, -1>(x);
    if (p.m > 1) twiddle<R, -1>(x, [&](int q) { return tw[q * k * p.step]; });
#pragma unroll
    for (int j = 0; j < R; ++j) z[at(base + j * p.m)] = x[j];
  }
}

// Decimation in time; dst(i, v) takes element i.
template <int R, class Dst>
__device__ __forceinline__ void dit_pass(double2 *z, int n, const Pass &p, const double2 *tw,
                                         Dst dst) {
  for (int t = threadIdx.x; t < n / R; t += blockDim.x) {
    int k;
    const int base = butterfly(p, t, &k);
    double2 x[R];
#pragma unroll
    for (int j = 0; j < R; ++j) x[j] = z[at(base + j * p.m)];
    if (p.m > 1) twiddle<R, 1>(x, [&](int q) { return tw[q * k * p.step]; });
    dft<R, 1>(x);
#pragma unroll
    for (int j = 0; j < R; ++j) dst(base + j * p.m, x[j]);
  }
}

// A pass of a prime radix r above 13, in shared memory, by the symmetric sums and
// differences of the samples j and r - j (formed in place first): a thread computes
// the outputs k and r - k of a butterfly together, 4 multiply-adds per pair of
// samples where a direct transform takes 16, into registers, and they are written
// back after a barrier.  Neighbouring threads take neighbouring butterflies, so the
// roots are broadcast and the samples contiguous.
constexpr int kMaxPairs = (kMaxLen / 2 + kMaxLen / 34 + kThreads - 1) / kThreads;
template <int SIGN>
__device__ void prime_pass(double2 *z, int n, const Pass &p, const double2 *tw) {
  const int r = p.r, m = p.m, step = p.step, s = n / r, H = (r - 1) / 2;
  // s butterflies; butterfly b: first element, twiddle index k
  for (int i = threadIdx.x; i < s * H; i += kThreads) {
    const int j = i / s + 1, b = i - (j - 1) * s;
    int k;
    const int first = butterfly(p, b, &k);
    double2 x = z[at(first + j * m)], y = z[at(first + (r - j) * m)];
    if (SIGN > 0) {  // DIT: input twiddles
      x = cmulc(x, tw[j * k * step]);
      y = cmulc(y, tw[(r - j) * k * step]);
    }
    z[at(first + j * m)] = cadd(x, y);
    z[at(first + (r - j) * m)] = csub(x, y);
  }
  __syncthreads();
  double2 lo[kMaxPairs], hi[kMaxPairs];
#pragma unroll
  for (int c = 0; c < kMaxPairs; ++c) {
    const int i = threadIdx.x + c * kThreads;
    if (i < s * (H + 1)) {
      const int q = i / s, b = i - q * s;  // outputs q and r - q (q == 0: that one alone)
      int k;
      const int first = butterfly(p, b, &k);
      double2 u = z[at(first)], v = make_double2(0.0, 0.0);
      int e = 0;  // (j q) mod r
      for (int j = 1; j <= H; ++j) {
        e += q;
        if (e >= r) e -= r;
        const double2 t = z[at(first + j * m)], d = z[at(first + (r - j) * m)];
        const double2 w = tw[e * s];  // cos, -sin
        u.x += w.x * t.x;
        u.y += w.x * t.y;
        v.x -= w.y * d.x;
        v.y -= w.y * d.y;
      }
      double2 x = make_double2(u.x - SIGN * v.y, u.y + SIGN * v.x);
      double2 y = make_double2(u.x + SIGN * v.y, u.y - SIGN * v.x);
      if (SIGN < 0 && q) {  // DIF: output twiddles
        x = cmul(x, tw[q * k * step]);
        y = cmul(y, tw[(r - q) * k * step]);
      }
      lo[c] = x;
      hi[c] = y;
    }
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < kMaxPairs; ++c) {
    const int i = threadIdx.x + c * kThreads;
    if (i < s * (H + 1)) {
      const int q = i / s, b = i - q * s;
      int k;
      const int first = butterfly(p, b, &k);
      z[at(first + q * m)] = lo[c];
      if (q) z[at(first + (r - q) * m)] = hi[c];
    }
  }
}

#define GD_DCT_RADICES(X) \
  X(16) X(15) X(14) X(13) X(12) X(11) X(10) X(9) X(8) X(7) X(6) X(5) X(4) X(3) X(2)

template <bool PRIME, class Src>
__device__ __forceinline__ void forward_pass(double2 *z, const Axis &a, int s, Src src) {
  const Pass &p = a.rad.p[s];
  switch (p.r) {
#define X(R) case R: dif_pass<R>(z, a.rad.n, p, a.tw, src); break;
    GD_DCT_RADICES(X)
#undef X
    default:
      if constexpr (PRIME) prime_pass<-1>(z, a.rad.n, p, a.tw);
      break;
  }
}

template <bool PRIME, class Dst>
__device__ __forceinline__ void inverse_pass(double2 *z, const Axis &a, int s, Dst dst) {
  const Pass &p = a.rad.p[s];
  switch (p.r) {
#define X(R) case R: dit_pass<R>(z, a.rad.n, p, a.tw, dst); break;
    GD_DCT_RADICES(X)
#undef X
    default:
      if constexpr (PRIME) prime_pass<1>(z, a.rad.n, p, a.tw);
      break;
  }
}

// load(i): sample at place i of the reordered line; natural order in, digit-reversed
// out in z.  A large prime comes first and then works on staged values.
template <bool PRIME, class Load>
__device__ __forceinline__ void forward_fft(double2 *z, const Axis &a, Load load) {
  int s = 0;
  bool staged = false;
  if constexpr (PRIME) staged = a.rad.p[0].r > 16;
  if (staged) {
    for (int i = threadIdx.x; i < a.rad.n; i += blockDim.x) z[at(i)] = load(i);
  } else {
    forward_pass<false>(z, a, 0, load);
    s = 1;
  }
  __syncthreads();
  for (; s < a.rad.count; ++s) {
    forward_pass<PRIME>(z, a, s, [&](int i) { return z[at(i)]; });
    __syncthreads();
  }
}

// digit-reversed in z; store(i, v) takes the (unscaled) value at place i.
template <bool PRIME, class Store>
__device__ __forceinline__ void inverse_fft(double2 *z, const Axis &a, Store store) {
  for (int s = a.rad.count - 1; s >= 1; --s) {
    inverse_pass<PRIME>(z, a, s, [&](int i, double2 v) { z[at(i)] = v; });
    __syncthreads();
  }
  bool staged = false;
  if constexpr (PRIME) staged = a.rad.p[0].r > 16;
  if (staged) {
    inverse_pass<PRIME>(z, a, 0, [&](int i, double2 v) { z[at(i)] = v; });
    __syncthreads();
    for (int i = threadIdx.x; i < a.rad.n; i += blockDim.x) store(i, z[at(i)]);
  } else {
    inverse_pass<false>(z, a, 0, store);
  }
}

// Pass 1: two rows of b -> their DCT-II coefficients along x in T.
template <bool PRIME>
__global__ void __launch_bounds__(kThreads, PRIME ? 1 : 2)
    k_rows_gen(double2 *__restrict__ T, int hp, const double *__restrict__ b, long long bpitch,
               int h, Axis ax) {
  extern __shared__ double2 z[];
  const int n = ax.rad.n;
  const RowPair rp(blockIdx.x, h);
  const double *ra = b + rp.ra * bpitch, *rb = b + rp.rb * bpitch;
  forward_fft<PRIME>(z, ax, [&](int i) {
    const int j = mak_sample(i, n);
    return make_double2(ra[j], rp.two ? rb[j] : 0.0);
  });
  for (int c = threadIdx.x; 2 * c < n; c += blockDim.x) {
    double va[2] = {0.0, 0.0}, vb[2] = {0.0, 0.0};
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int k = 2 * c + q;
      if (k >= n) break;
      const Coef4 f = split(z[at(ax.rev[k])], z[at(ax.rev[k ? n - k : 0])], ax.post[k]);
      va[q] = f.ak;
      vb[q] = f.bk;
    }
    double2 *dst = T + (long long)c * hp + rp.p0;
    dst[0] = make_double2(va[0], va[1]);
    if (rp.two) dst[1] = make_double2(vb[0], vb[1]);
  }
}

// Pass 2: columns c0, c0 + 1 of T: DCT-II along y, division by the
// eigenvalues (the constant mode set to zero), DCT-III along y.
template <bool PRIME>
__global__ void __launch_bounds__(kThreads, PRIME ? 1 : 2)
    k_cols_gen(double2 *__restrict__ T, int hp, int w, Axis ay,
               const double *__restrict__ eig_w) {
  extern __shared__ double2 z[];
  const int n = ay.rad.n, c0 = 2 * blockIdx.x;
  double2 *col = T + (long long)blockIdx.x * hp;
  forward_fft<PRIME>(z, ay, [&](int i) { return col[i]; });
  const double ew_a = eig_w[c0], ew_b = c0 + 1 < w ? eig_w[c0 + 1] : 0.0;
  for (int k = threadIdx.x; k <= n / 2; k += blockDim.x) {
    const int pk = at(ay.rev[k]);
    const double ek = ay.eig[k];
    if (k == 0) {
      const double2 z0 = z[pk];  // X_a[0] = Re Z_0, X_b[0] = Im Z_0; W_0 = X_0
      const double la = (ek + ew_a) - 4.0, lb = (ek + ew_b) - 4.0;
      // mode (0, 0) is the constant: zero (the zero-mean solution)
      z[pk] = make_double2(c0 == 0 ? 0.0 : z0.x / la, z0.y / lb);
      continue;
    }
    const int nk = n - k, pn = at(ay.rev[nk]);
    const double2 tk = ay.post[k];
    const double en = ay.eig[nk];
    Coef4 c = split(z[pk], z[pn], tk);
    c.ak /= (ek + ew_a) - 4.0;
    c.bk /= (ek + ew_b) - 4.0;
    c.an /= (en + ew_a) - 4.0;
    c.bn /= (en + ew_b) - 4.0;
    z[pk] = pack_inverse(c.ak, c.an, c.bk, c.bn, tk);
    if (nk != k) z[pn] = pack_inverse(c.an, c.ak, c.bn, c.bk, make_double2(-tk.y, -tk.x));
  }
  __syncthreads();
  const double inv_n = 1.0 / (double)n;
  inverse_fft<PRIME>(z, ay, [&](int i, double2 v) {
    col[i] = make_double2(v.x * inv_n, v.y * inv_n);
  });
}

// Pass 3: two rows of T (coefficients along x) -> DCT-III -> u.
template <bool PRIME>
__global__ void __launch_bounds__(kThreads, PRIME ? 1 : 2)
    k_irows_gen(double *__restrict__ u, long long upitch, const double2 *__restrict__ T, int hp,
                int h, Axis ax) {
  extern __shared__ double2 z[];
  const int n = ax.rad.n;
  const RowPair rp(blockIdx.x, h);
  const double *Td = reinterpret_cast<const double *>(T);
  auto coef = [&](int k) {  // (X_a[k], X_b[k])
    const double *p = Td + ((long long)(k >> 1) * hp + rp.p0) * 2 + (k & 1);
    return make_double2(p[0], rp.two ? p[2] : 0.0);
  };
  for (int k = threadIdx.x; k <= n / 2; k += blockDim.x) {
    const double2 xk = coef(k);
    if (k == 0) {
      z[at(ax.rev[0])] = xk;  // W_0 = X_0 (X_n = 0)
      continue;
    }
    const int nk = n - k;
    const double2 xn = coef(nk), tk = ax.post[k];
    z[at(ax.rev[k])] = pack_inverse(xk.x, xn.x, xk.y, xn.y, tk);
    if (nk != k)
      z[at(ax.rev[nk])] = pack_inverse(xn.x, xk.x, xn.y, xk.y, make_double2(-tk.y, -tk.x));
  }
  __syncthreads();
  const double inv_n = 1.0 / (double)n;
  double *ua = u + rp.ra * upitch, *ub = u + rp.rb * upitch;
  inverse_fft<PRIME>(z, ax, [&](int i, double2 v) {
    const int j = mak_sample(i, n);
    ua[j] = v.x * inv_n;
    if (rp.two) ub[j] = v.y * inv_n;
  });
}

// An axis' tables.  `len` > 0: a power of two's own kernels, radix 2^lv, whose table of
// `len` entries (P2::table_offset) takes the place of the plain twiddles.
struct TableJob {
  double2 *tw, *post;
  double *eig;
  unsigned short *rev;
  Radices rad;
  int lv, len;
};
__global__ void k_dct_tables(TableJob rows, TableJob cols) {
  const TableJob &J = blockIdx.y ? cols : rows;
  const int n = J.rad.n, lv = J.lv, len = J.len;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  int e = k;  // exponent of the twiddle in place k
  if (len) {
    int row = n >> lv, step = 1, at = k;  // butterflies of a pass, step of its twiddles
    while (row > 0 && at >= kPowers * row) {
      at -= kPowers * row;
      row >>= lv;
      step <<= lv;
    }
    if (k < len) e = (at % row * step) << (at / row);
  }
  double s, c;
  if (!len || k < len) {
    sincospi(2.0 * (double)e / (double)n, &s, &c);
    J.tw[k] = make_double2(c, -s);
  }
  sincospi((double)k / (2.0 * (double)n), &s, &c);
  J.post[k] = make_double2(c, -s);
  J.eig[k] = 2.0 * cos(M_PI * (double)k / (double)n);
  int pos = 0, f = k;
  for (int q = 0; q < J.rad.count; ++q) {
    pos += (f % J.rad.p[q].r) * J.rad.p[q].m;
    f /= J.rad.p[q].r;
  }
  J.rev[k] = (unsigned short)pos;
}

inline size_t a256(size_t v) { return (v + 255) & ~(size_t)255; }
inline size_t smem_bytes(int n) { return (size_t)((n + 7) & ~7) * sizeof(double2); }
// the most dynamic shared memory any DCT kernel launch asks for
constexpr size_t kMaxSmemBytes = (size_t)kMaxLen * sizeof(double2);

template <int V>
using Int = std::integral_constant<int, V>;

// Call p2(Int<log2 n>{}) for the power-of-two kernels' lengths, gen(PRIME) otherwise
// (16 and 32, which are one or two passes, gain nothing from a kernel of their own).
template <class P2Fn, class GenFn>
void with_kernels(const Radices &r, P2Fn &&p2, GenFn &&gen) {
  switch (r.n) {
    case 64: p2(Int<6>{}); return;
    case 128: p2(Int<7>{}); return;
    case 256: p2(Int<8>{}); return;
    case 512: p2(Int<9>{}); return;
    case 1024: p2(Int<10>{}); return;
    case 2048: p2(Int<11>{}); return;
    case 4096: p2(Int<12>{}); return;
    case 8192: p2(Int<13>{}); return;
    default: break;
  }
  if (has_large_prime(r)) gen(std::true_type{});
  else gen(std::false_type{});
}

}  // namespace dct
}  // namespace gd

using namespace gd;

struct gd_dct_plan_s {
  int h = 0, w = 0;
  int hp = 0;  // rows of T per column pair (h rounded up to an even number)
  dct::Radices rh, rw;
  size_t o_t = 0, o_tab_w = 0, o_tab_h = 0, total = 0;
  char *ws = nullptr;
};

namespace {

struct AxisTables {
  double2 *tw, *post;
  double *eig;
  unsigned short *rev;
};

constexpr size_t kTableBytes = 2 * sizeof(double2) + sizeof(double) + sizeof(unsigned short);

AxisTables tables(gd_dct_plan p, size_t off, int n) {
  char *b = p->ws + off;
  AxisTables t;
  t.tw = reinterpret_cast<double2 *>(b);
  t.post = t.tw + n;
  t.eig = reinterpret_cast<double *>(t.post + n);
  t.rev = reinterpret_cast<unsigned short *>(t.eig + n);
  return t;
}

dct::Axis axis(gd_dct_plan p, bool rows) {
  const int n = rows ? p->w : p->h;
  const AxisTables t = tables(p, rows ? p->o_tab_w : p->o_tab_h, n);
  dct::Axis a;
  a.rad = rows ? p->rw : p->rh;
  a.tw = t.tw;
  a.post = t.post;
  a.eig = t.eig;
  a.rev = t.rev;
  return a;
}

}  // namespace

extern "C" void gd_dct_plan_destroy(gd_dct_plan p) { delete p; }

extern "C" int gd_dct_plan_create(int32_t h, int32_t w, gd_dct_plan *out) {
  GD_REQUIRE(out && h > 1 && w > 1, GD_ERR_ARG,
             "gd_dct_plan_create: the grid needs at least 2 x 2 cells");
  GD_REQUIRE(h <= dct::kMaxLen && w <= dct::kMaxLen, GD_ERR_UNSUPPORTED,
             "gd_dct_plan_create: sides above %d are not supported (grid %d x %d)",
             dct::kMaxLen, h, w);
  *out = nullptr;
  gd_dct_plan p = new gd_dct_plan_s();
  p->h = h;
  p->w = w;
  p->hp = (h + 1) & ~1;
  p->rh = dct::choose_passes(h, w);
  p->rw = dct::choose_passes(w, h);
  size_t o = 0;
  p->o_t = o;
  o = dct::a256(o + (size_t)((w + 1) / 2) * p->hp * sizeof(double2));
  p->o_tab_w = o;
  o = dct::a256(o + (size_t)w * kTableBytes);
  p->o_tab_h = o;
  o = dct::a256(o + (size_t)h * kTableBytes);
  p->total = o;
  *out = p;
  return GD_OK;
}

extern "C" size_t gd_dct_workspace_bytes(gd_dct_plan p) { return p ? p->total : 0; }

extern "C" int gd_dct_plan_bind(gd_dct_plan p, void *ws, size_t bytes, cudaStream_t st) {
  GD_REQUIRE(p && ws, GD_ERR_ARG, "gd_dct_plan_bind: bad arguments");
  GD_REQUIRE(bytes >= p->total, GD_ERR_ARG, "gd_dct_plan_bind: workspace %zu < %zu bytes", bytes,
             p->total);
  GD_REQUIRE(((uintptr_t)ws & 255) == 0, GD_ERR_ARG, "gd_dct_plan_bind: workspace must be "
                                                     "256-byte aligned");
  p->ws = static_cast<char *>(ws);
  const AxisTables tw = tables(p, p->o_tab_w, p->w), th = tables(p, p->o_tab_h, p->h);
  auto job = [&](const AxisTables &t, const dct::Radices &r) {
    dct::TableJob j{t.tw, t.post, t.eig, t.rev, r, 0, 0};
    dct::with_kernels(
        r,
        [&](auto log) {
          j.len = dct::P2<decltype(log)::value>::table_len;
          j.lv = dct::P2<decltype(log)::value>::LV;
        },
        [](auto) {});
    return j;
  };
  const dim3 grid((std::max(p->w, p->h) + 255) / 256, 2);
  dct::k_dct_tables<<<grid, 256, 0, st>>>(job(tw, p->rw), job(th, p->rh));
  GD_CHECK_LAUNCH();
  // the tables must be complete before a solve on any stream (set-up, once per plan)
  GD_CHECK_CUDA(cudaStreamSynchronize(st));
  // Shared memory of the kernels this plan launches.  The limit is one value per
  // kernel for the whole process, so every plan sets the same value, the most any
  // length needs: a plan bound later for a shorter line must not lower the limit
  // under a plan of a longer one (its next launch would fail).
  cudaError_t err = cudaSuccess;
  auto allow = [&](const void *fn) {
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)dct::kMaxSmemBytes);
    if (e != cudaSuccess) err = e;
  };
  dct::with_kernels(
      p->rw,
      [&](auto log) {
        allow((const void *)dct::k_rows_p2<decltype(log)::value>);
        allow((const void *)dct::k_irows_p2<decltype(log)::value>);
      },
      [&](auto prime) {
        allow((const void *)dct::k_rows_gen<decltype(prime)::value>);
        allow((const void *)dct::k_irows_gen<decltype(prime)::value>);
      });
  dct::with_kernels(
      p->rh, [&](auto log) { allow((const void *)dct::k_cols_p2<decltype(log)::value>); },
      [&](auto prime) { allow((const void *)dct::k_cols_gen<decltype(prime)::value>); });
  GD_CHECK_CUDA(err);
  return GD_OK;
}

extern "C" int gd_dct_solve_neumann(gd_dct_plan p, const double *b_in, double *u, int32_t pitch,
                                    cudaStream_t st) {
  GD_REQUIRE(p && p->ws && b_in && u && pitch >= p->w, GD_ERR_ARG,
             "gd_dct_solve_neumann: bad arguments or unbound plan");
  const int h = p->h, w = p->w, hp = p->hp;
  double2 *T = reinterpret_cast<double2 *>(p->ws + p->o_t);
  const dct::Axis ax = axis(p, true), ay = axis(p, false);
  const int rows = (h + 1) / 2, cols = (w + 1) / 2;
  const int tw = dct::gen_threads(p->rw), th = dct::gen_threads(p->rh);
  dct::with_kernels(
      p->rw,
      [&](auto log) {
        using F = dct::P2<decltype(log)::value>;
        dct::k_rows_p2<decltype(log)::value><<<F::ctas(rows), F::threads, F::smem, st>>>(
            T, hp, b_in, pitch, h, ax.tw, ax.post);
      },
      [&](auto prime) {
        dct::k_rows_gen<decltype(prime)::value><<<rows, tw, dct::smem_bytes(w), st>>>(
            T, hp, b_in, pitch, h, ax);
      });
  dct::with_kernels(
      p->rh,
      [&](auto log) {
        using F = dct::P2<decltype(log)::value>;
        dct::k_cols_p2<decltype(log)::value><<<F::ctas(cols), F::threads, F::smem, st>>>(
            T, hp, w, ay.tw, ay.post, ay.eig, ax.eig);
      },
      [&](auto prime) {
        dct::k_cols_gen<decltype(prime)::value><<<cols, th, dct::smem_bytes(h), st>>>(T, hp, w, ay,
                                                                                     ax.eig);
      });
  dct::with_kernels(
      p->rw,
      [&](auto log) {
        using F = dct::P2<decltype(log)::value>;
        dct::k_irows_p2<decltype(log)::value><<<F::ctas(rows), F::threads, F::smem, st>>>(
            u, pitch, T, hp, h, ax.tw, ax.post);
      },
      [&](auto prime) {
        dct::k_irows_gen<decltype(prime)::value><<<rows, tw, dct::smem_bytes(w), st>>>(
            u, pitch, T, hp, h, ax);
      });
  GD_CHECK_LAUNCH();
  return GD_OK;
}
