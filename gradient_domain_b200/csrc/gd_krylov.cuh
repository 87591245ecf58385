// Krylov kernels of the batched MGPCG on level 0: p = z + beta p with p.Ap, and
// d += alpha p, r -= alpha A p with r.r.
//
// Both are streaming passes (12 and 20 bytes a cell in FP32).  A warp walks its
// rows of 128 columns (four per lane) through per-lane cp.async rings, so seven
// rows per lane are in flight while one is processed.  A CTA costs about 3 us
// whatever its height - the chain tile -> descriptors -> first rows, then the
// block sum, the fence and the ticket - so short tiles are expensive: 16-row
// tiles took 43 us (d/r) at 1411 x 1387 x 3 and 256 us at 4096 x 4096 x 3, 64-row
// tiles 30 and 172 us (51 and 171 us with one shared ticket and the classes of
// masked rows loaded on use; event times of single launches, mixed precision).
// tile_rows() has the rule.
//
// The search direction lives in two buffers: k_pupdate reads the current one
// (including halo cells owned by other CTAs) and writes the other, so no CTA
// overwrites a value another CTA still has to read.
//
// Level 0 has wall coefficient 0 (Neumann) or 1, so a cell's diagonal is
// 4 - walls (1 - w), exact in FP32 and formed from a per-lane column term and a
// row term; masked levels always have 4.  Cells without an unknown and the
// padding of a row (columns nx .. pitch - 1) hold zeros in every level-0 array:
// z and p need no test there, and only the update of r, whose neighbours may be
// unknowns, selects (masked levels copy each row's classes through a ring).
#pragma once

#include "gd_stream.cuh"

namespace gd {
namespace kr {

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;

// Rows of an instance's Krylov tiles (a CTA each, a quarter of them per warp),
// from the instance alone, because they group its partial sums.  64, but 32
// where 64 would leave SMs without a tile (1024 x 1024: 13.3 us a launch instead
// of 14.6), and taller while that still gives every SM six CTAs (two waves).
constexpr int kSms = 148;
inline int tile_rows(int ny, int nx) {
  const long long cols = (nx + kFTX - 1) / kFTX;
  auto tiles = [&](int rows) { return cols * ((ny + rows - 1) / rows); };
  if (tiles(64) < kSms) return 32;
  int rows = 64;
  while (rows < 512 && tiles(2 * rows) >= 6 * kSms) rows *= 2;
  return rows;
}

template <typename T>
using Ring = st::Ring<T, kThreads>;

// Per-lane ring of one element per row: the column just outside the warp
// (left of lane 0, right of lane 31), so edge values arrive with their row.
template <typename T>
struct EdgeRing {
  T *base;
  __device__ __forceinline__ explicit EdgeRing(T *smem) : base(smem + threadIdx.x) {}
  __device__ __forceinline__ T *slot(int s) const {
    return base + (s & (st::kRing - 1)) * kThreads;
  }
  __device__ __forceinline__ void issue(int s, const T *src, bool ok) const {
    __pipeline_memcpy_async(slot(s), src, sizeof(T), ok ? 0 : sizeof(T));
  }
  __device__ __forceinline__ T read(int s) const { return *slot(s); }
};

template <typename T>
constexpr size_t edge_bytes() { return (size_t)st::kRing * kThreads * sizeof(T); }
template <typename T>
constexpr size_t pupdate_smem() {
  return 2 * st::ring_bytes<T, kThreads>() + 2 * edge_bytes<T>();
}
template <typename T>
constexpr size_t cgupdate_smem(bool mask) {
  return 3 * st::ring_bytes<T, kThreads>() + edge_bytes<T>() +
         (mask ? (size_t)st::kRing * kThreads * 4 : 0);
}

// One 16-byte-per-lane (FP32; two for FP64) copy into a ring slot.
template <typename T>
__device__ __forceinline__ void copy4(T *dst, const T *src, bool ok) {
#pragma unroll
  for (int k = 0; k < (int)(4 * sizeof(T) / 16); ++k)
    __pipeline_memcpy_async(dst + k * (16 / sizeof(T)), src + (ok ? k * (16 / sizeof(T)) : 0), 16,
                            ok ? 0 : 16);
}

// Where a warp works: its columns, the lane's four, and the diagonal terms.
template <typename T>
struct Place {
  int ny, pitch;     // of the level, in registers (stores could alias the descriptor)
  int x0, xe, nv;    // the lane's first column, the edge column of lanes 0 and 31, columns in the grid
  bool in, edge;     // the lane has columns in the grid; it also copies an in-grid edge column
  T dcol[4], drow;   // column diagonals; what a wall row takes off
  __device__ __forceinline__ Place(const LevelInfo &L, int tx) {
    const int lane = threadIdx.x & 31;
    ny = L.ny;
    pitch = L.pitch;
    x0 = tx * kFTX + 4 * lane;
    xe = lane == 0 ? x0 - 1 : x0 + 4;
    in = x0 < L.nx;
    nv = min(4, L.nx - x0);
    edge = (lane == 0 || lane == 31) && xe >= 0 && xe < L.nx;
    drow = (T)(1.0f - L.wall);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      dcol[j] = T(4) - (T)((x0 + j == 0) + (x0 + j == L.nx - 1)) * drow;
  }
  __device__ __forceinline__ bool row(int y) const { return y >= 0 && y < ny; }
};

// A u on row y of the lane's columns; `e` is the edge value of lanes 0 and 31.
template <typename T>
__device__ __forceinline__ st::V4<T> apply_row(const Place<T> &w, int y, const st::V4<T> &u,
                                               const st::V4<T> &up, const st::V4<T> &dn, T e) {
  const int lane = threadIdx.x & 31;
  T left = st::shfl_up1(u.v[3]), right = st::shfl_dn1(u.v[0]);
  if (lane == 0) left = e;
  if (lane == 31) right = e;
  const T lf[4] = {left, u.v[0], u.v[1], u.v[2]};
  const T rt[4] = {u.v[1], u.v[2], u.v[3], right};
  const T dr = (T)((y == 0) + (y == w.ny - 1)) * w.drow;
  st::V4<T> r;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    r.v[j] = (w.dcol[j] - dr) * u.v[j] - (up.v[j] + dn.v[j] + lf[j] + rt[j]);
  return r;
}

template <typename T>
__device__ __forceinline__ double pupdate_rows(const Place<T> &w, int y0, int y1, T beta,
                                               const T *z, const T *p, T *pn,
                                               unsigned char *smem) {
  constexpr int kE = st::kRing * kThreads;
  T *const s0 = reinterpret_cast<T *>(smem);
  const Ring<T> rz(s0), rp(s0 + 4 * kE);
  const EdgeRing<T> ez(s0 + 8 * kE), ep(s0 + 9 * kE);
  const bool use_p = beta != T(0);  // the first direction is z: the old buffer is not read
  const bool edge_lane = (threadIdx.x & 31) == 0 || (threadIdx.x & 31) == 31;
  const int nsteps = y1 - y0 + 2;   // rows y0 - 1 .. y1; nothing past them is copied
  auto issue = [&](int q) {
    if (q < nsteps) {
      const int y = y0 - 1 + q;
      const bool ok = w.in && w.row(y);
      const long long g = ok ? (long long)y * w.pitch + w.x0 : 0;
      copy4(rz.slot(q), z + g, ok);
      if (use_p) copy4(rp.slot(q), p + g, ok);
      if (edge_lane) {
        const bool eok = w.edge && w.row(y);
        const long long ge = eok ? (long long)y * w.pitch + w.xe : 0;
        ez.issue(q, z + ge, eok);
        if (use_p) ep.issue(q, p + ge, eok);
      }
    }
    __pipeline_commit();
  };
#pragma unroll
  for (int q = 0; q < st::kRing - 1; ++q) issue(q);
  int step = 0;
  T edge_next = T(0);
  auto newp = [&]() {
    __pipeline_wait_prior(st::kRing - 2);
    st::V4<T> zz = rz.read(step);
    T e = edge_lane ? ez.read(step) : T(0);
    if (use_p) {
      const st::V4<T> pp = rp.read(step);
      if (edge_lane) e += beta * ep.read(step);
#pragma unroll
      for (int j = 0; j < 4; ++j) zz.v[j] += beta * pp.v[j];
    }
    edge_next = e;
    issue(step + st::kRing - 1);
    ++step;
    return zz;
  };
  double part = 0.0;
  st::V4<T> up = newp(), cu = newp();
  T edge_cu = edge_next;
  for (int y = y0; y < y1; ++y) {
    const st::V4<T> dn = newp();
    const st::V4<T> ap = apply_row(w, y, cu, up, dn, edge_cu);
    edge_cu = edge_next;
    T acc = T(0);
#pragma unroll
    for (int j = 0; j < 4; ++j) acc += cu.v[j] * ap.v[j];
    part += (double)acc;
    if (w.in) st::st4(pn + (long long)y * w.pitch + w.x0, cu);
    up = cu;
    cu = dn;
  }
  __pipeline_wait_prior(0);
  return part;
}

// p_new = z + beta p_old (read from one buffer, written to the other) and p.Ap.
template <typename T>
__global__ void __launch_bounds__(kThreads) k_pupdate(Args<T> a) {
  const Tile tl = a.tiles[blockIdx.x];
  dep_enter();
  if (blockIdx.x == 0 && threadIdx.x == 0 && a.loop) {
    const int t = *a.trips + 1;
    *a.trips = t;
    if (t >= a.trip_cap) set_condition(a.loop, 0u);
  }
  const InstInfo &I = a.inst[tl.inst];
  InstState &S = a.st[tl.inst];
  // every descriptor field is requested before the first is used
  const int rows = I.kr_rows, ctas = I.kr_end - I.kr_begin, pcur = S.pcur, status = S.status;
  const bool idle = !a.act[blockIdx.x];  // no unknown: p stays zero
  const T beta = (T)S.beta;
  const double rz = S.rz;
  const T *z = a.arena + I.z_off;
  const T *p = a.arena + (pcur ? I.q_off : I.p_off);
  T *pn = a.arena + (pcur ? I.p_off : I.q_off);
  const Place<T> w(a.lv[tl.level], tl.tx);
  if (status != GD_ACTIVE) return;
  extern __shared__ __align__(16) unsigned char smem[];
  const int share = rows / kWarps;
  const int y0 = tl.ty * rows + (threadIdx.x >> 5) * share, y1 = min(y0 + share, w.ny);
  double part = y0 < w.ny && !idle ? pupdate_rows<T>(w, y0, y1, beta, z, p, pn, smem) : 0.0;
  double pAp;
  if (!instance_sum<kThreads>(a.part0, I.kr_begin, ctas, part, &S.ticket, &pAp)) return;
  if (threadIdx.x == 0) {
    const double alpha = rz / pAp;
    S.pAp = pAp;
    S.pcur = pcur ^ 1;
    if (!(pAp > 0.0) || !isfinite(alpha)) {
      S.status = GD_BREAKDOWN;
      S.flags |= FLAG_RU;
      set_condition(a.refresh, 1u);
    } else {
      S.alpha = alpha;
    }
  }
}

template <typename T, bool MASK>
__device__ __forceinline__ double cgupdate_rows(const Place<T> &w, const unsigned char *codes,
                                                int y0, int y1, T alpha, const T *p, T *d, T *r,
                                                bool dzero, unsigned char *smem) {
  constexpr int kE = st::kRing * kThreads;
  T *const s0 = reinterpret_cast<T *>(smem);
  const Ring<T> rp(s0), rd(s0 + 4 * kE), rr(s0 + 8 * kE);
  const EdgeRing<T> ep(s0 + 12 * kE);
  unsigned *const cring = reinterpret_cast<unsigned *>(s0 + 13 * kE) + threadIdx.x;
  const bool edge_lane = (threadIdx.x & 31) == 0 || (threadIdx.x & 31) == 31;
  // p streams rows y0 - 1 .. y1; d, r and the classes the band's own rows, used
  // one step later (the slots of the two halo rows are never read)
  const int nsteps = y1 - y0 + 2;
  auto issue = [&](int q) {
    if (q < nsteps) {
      const int y = y0 - 1 + q;
      const bool ok = w.in && w.row(y);
      const long long g = ok ? (long long)y * w.pitch + w.x0 : 0;
      copy4(rp.slot(q), p + g, ok);
      if (y >= y0 && y < y1) {
        if (!dzero) copy4(rd.slot(q), d + g, ok);
        copy4(rr.slot(q), r + g, ok);
        if constexpr (MASK)
          __pipeline_memcpy_async(cring + (q & (st::kRing - 1)) * kThreads, codes + g, 4,
                                  ok ? 0 : 4);
        if (edge_lane) ep.issue(q, p + (w.edge ? (long long)y * w.pitch + w.xe : 0), w.edge);
      }
    }
    __pipeline_commit();
  };
#pragma unroll
  for (int q = 0; q < st::kRing - 1; ++q) issue(q);
  double part = 0.0;
  __pipeline_wait_prior(st::kRing - 2);
  st::V4<T> up = rp.read(0);
  issue(st::kRing - 1);
  __pipeline_wait_prior(st::kRing - 2);
  st::V4<T> cu = rp.read(1);
  for (int y = y0; y < y1; ++y) {
    const int s = y - y0 + 1;  // ring step of row y
    st::V4<T> dv = st::zero4<T>();
    if (!dzero) dv = rd.read(s);
    st::V4<T> rv = rr.read(s);
    const T e = edge_lane ? ep.read(s) : T(0);
    unsigned c = 0u;
    if constexpr (MASK) c = cring[(s & (st::kRing - 1)) * kThreads];
    issue(s + st::kRing - 1);  // into the slot of step s - 1, whose values were used
    __pipeline_wait_prior(st::kRing - 2);
    const st::V4<T> dn = rp.read(s + 1);
    const st::V4<T> ap = apply_row(w, y, cu, up, dn, e);
    T acc = T(0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool on = MASK ? st::cls(c, j) != 0 : j < w.nv;
      dv.v[j] += alpha * cu.v[j];
      rv.v[j] = on ? rv.v[j] - alpha * ap.v[j] : T(0);
      acc += rv.v[j] * rv.v[j];
    }
    // the columns of a width that is no multiple of four: squares in FP64
    double sq = (double)acc;
    if (sizeof(T) == 4 && w.nv < 4) {
      double q[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) q[j] = (double)rv.v[j] * (double)rv.v[j];
      sq = (q[0] + q[1]) + (q[2] + q[3]);
    }
    part += sq;
    if (w.in) {
      const long long g = (long long)y * w.pitch + w.x0;
      st::st4(d + g, dv);
      st::st4(r + g, rv);
    }
    up = cu;
    cu = dn;
  }
  __pipeline_wait_prior(0);
  return part;
}

// d += alpha p, r -= alpha A p and r.r; schedules FP64 refreshes.  ANY: the
// plan has masked instances.
template <typename T, bool ANY>
__global__ void __launch_bounds__(kThreads) k_cgupdate(Args<T> a) {
  const Tile tl = a.tiles[blockIdx.x];
  dep_enter();
  const InstInfo &I = a.inst[tl.inst];
  InstState &S = a.st[tl.inst];
  const int rows = I.kr_rows, ctas = I.kr_end - I.kr_begin, status = S.status, flags = S.flags;
  const int iters = S.iters + 1;
  const bool idle = !a.act[blockIdx.x];  // no unknown: d and r stay zero
  const T alpha = (T)S.alpha;
  const double rr_ref = S.rr_ref, ff = S.ff;
  const T *p = a.arena + (S.pcur ? I.q_off : I.p_off);
  T *d = a.arena + I.d_off;
  T *r = a.arena + I.r_off;
  const long long code_off = ANY ? a.lv[tl.level].code_off : -1;
  const Place<T> w(a.lv[tl.level], tl.tx);
  if (status != GD_ACTIVE) return;
  extern __shared__ __align__(16) unsigned char smem[];
  const int share = rows / kWarps;
  const int y0 = tl.ty * rows + (threadIdx.x >> 5) * share, y1 = min(y0 + share, w.ny);
  const bool dzero = flags & FLAG_DZERO;
  double part = 0.0;
  if (y0 < w.ny && !idle) {
    if (ANY && code_off >= 0)
      part = cgupdate_rows<T, true>(w, a.codes + code_off, y0, y1, alpha, p, d, r, dzero, smem);
    else
      part = cgupdate_rows<T, false>(w, nullptr, y0, y1, alpha, p, d, r, dzero, smem);
  }
  double rr;
  if (!instance_sum<kThreads>(a.part0, I.kr_begin, ctas, part, &S.ticket, &rr)) return;
  if (threadIdx.x == 0) {
    S.rr = rr;
    S.iters = iters;
    int f = flags & ~FLAG_DZERO;  // every CTA of this instance has read it
    if (rr <= a.delta2 * rr_ref || rr <= a.tol2 * ff || iters >= a.max_iter || !isfinite(rr)) {
      f |= FLAG_RU;
      set_condition(a.refresh, 1u);
    }
    S.flags = f;
  }
}

}  // namespace kr
}  // namespace gd
