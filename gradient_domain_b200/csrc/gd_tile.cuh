// Shared-memory tile kernels for the coarse levels of the V-cycle.
//
// The register-streaming kernels of gd_stream.cuh walk every strip row by row;
// on a small level a launch has too few strips to fill the GPU and each warp
// waits on the latency of its own row chain, so a level costs a fixed 15-30 us
// whatever its size.  Here a CTA instead loads one tile of the level plus a
// halo into shared memory and runs every phase (a red-black half sweep, the
// residual, the restriction or the prolongation) over the whole tile at once,
// with a barrier between phases: all cells of a phase are independent, so the
// CTA's threads work in parallel.
//
// A thread works on groups of four consecutive cells of a row, held as two
// same-colour pairs E = (v0, v2) and O = (v1, v3); region rows start on 16-byte
// boundaries because the horizontal halo is kHX = 8 cells and tiles start on
// multiples of kTX.  A thread's groups - u, b, the diagonal inverses - stay in
// registers for the whole tile; shared memory holds u for the neighbours, so a half
// sweep reads one pair above, one below and one scalar beside, and writes one pair
// (with b, u and the classes in shared memory a half sweep moved three times the
// bytes: 29-instance batch, event times of two levels, 23.1 + 21.8 and 14.4 + 12.9 us
// then, 18.4 + 17.1 and 10.7 + 10.7 us so).
//
// A half sweep that reads neighbours leaves the outermost exact ring of the loaded
// region one cell further in, so the down kernel (whose first half sweep, from zero,
// reads only b and is applied while loading) needs 2 S1 + 1 halo rows (2 S1 - 1 for
// the sweeps, one for the residual's neighbours, one for the restriction's
// reach) and the up kernel 2 S2; kHX covers both in x for up to 3 sweeps.
// Cells outside the grid have class 0: their diagonal inverse is zero, so they stay
// zero, which is the operator's definition of a missing neighbour.
#pragma once

#include "gd_stream.cuh"

namespace gd {
namespace tile {

// Two tile shapes.  Levels with at least one 32 x 64 tile per SM run those
// tiles on CTAs of 512 threads (throughput; at 256 a thread holds four groups and the
// same levels took 19.1 + 20.0 us).  Smaller levels, where one CTA's
// chain of phases is the launch's duration, run 16 x 32 tiles on CTAs of 384
// threads: every phase is one pass per thread, and the level spreads over four
// times as many SMs, so each SM issues a quarter of the instructions.
constexpr int kTY = 32, kTX = 64;    // cells of a large tile (even: whole coarse cells)
constexpr int kTYs = 16, kTXs = 32;  // cells of a small tile
constexpr int kHX = 8;               // halo columns on each side
constexpr int kThreads = 512, kThreadsSmall = 384;

template <typename T, int S1, int TY = kTY, int TX = kTX>
struct DownT {
  static constexpr int H = 2 * S1 + 1;
  static constexpr int RY = TY + 2 * H, RX = TX + 2 * kHX, N = RY * RX, GX = RX / 4;
  static constexpr size_t smem = (size_t)2 * N * sizeof(T);
};

template <typename T, int S2, int TY = kTY, int TX = kTX>
struct UpT {
  static constexpr int H = 2 * S2;
  static constexpr int RY = TY + 2 * H, RX = TX + 2 * kHX, N = RY * RX, GX = RX / 4;
  static constexpr int CY = RY / 2 + 3, CX = RX / 2 + 3, CN = CY * CX;
  static constexpr size_t smem = (size_t)(N + CN) * sizeof(T);
};

static_assert(kHX % 4 == 0 && kTX % 4 == 0 && kTXs % 4 == 0 && kHX >= 7, "tile geometry");
static_assert(kTY % 2 == 0 && kTYs % 2 == 0, "tiles hold whole coarse cells");
// one group of four cells per thread and phase on small tiles (up to three sweeps)
static_assert((kTYs + 2 * 7) * ((kTXs + 2 * kHX) / 4) <= kThreadsSmall, "small tile threads");

template <typename T>
__device__ __forceinline__ void diag_tables(T *tdiag, T *tdinv, float wall) {
  if (threadIdx.x < 8) {
    const int c = threadIdx.x;
    const double d = c >= 1 && c <= 5 ? class_diag(c, wall) : 1.0;
    tdiag[c] = (T)d;
    tdinv[c] = (c >= 1 && c <= 5 && d > 0.0) ? (T)(1.0 / d) : T(0);
  }
}

// Cells x .. x + 3 of row y (x a multiple of 4), zero outside the grid.
template <typename T>
__device__ __forceinline__ st::V4<T> load_group(const T *A, const LevelInfo &L, int y, int x) {
  if (y < 0 || y >= L.ny || x < 0 || x >= L.nx) return st::zero4<T>();
  const T *p = A + (long long)y * L.pitch + x;
  if (x + 3 < L.nx) return st::ld4(p);
  st::V4<T> r;
#pragma unroll
  for (int j = 0; j < 4; ++j) r.v[j] = (x + j < L.nx) ? p[j] : T(0);
  return r;
}

template <typename T>
__device__ __forceinline__ void store_group(T *A, const LevelInfo &L, int y, int x,
                                            const st::V4<T> &v) {
  if (y >= L.ny || x >= L.nx) return;
  T *p = A + (long long)y * L.pitch + x;
  if (x + 3 < L.nx) {
    st::st4(p, v);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (x + j < L.nx) p[j] = v.v[j];
  }
}

// One group of a tile's region in a thread's registers.
template <typename T>
struct Group {
  Duo<T> e, o, be, bo, ie, io;
  int li, ri;   // groups beside it (its own at the region's left and right end)
  int odd;      // parity of the corner cell: the cells of pair J have colour (J + odd) & 1
  unsigned c;   // classes
  bool sweeps;  // an inner row of the region

  __device__ __forceinline__ void place(int g, int RY, int GX, int par0, unsigned classes,
                                        const st::V4<T> &b, const T *dinv) {
    const int ry = g / GX, gx = g - ry * GX;
    li = g - (gx > 0);
    ri = g + (gx < GX - 1);
    odd = (par0 + ry) & 1;
    c = classes;
    sweeps = ry > 0 && ry < RY - 1;
    be = duo(b.v[0], b.v[2]);
    bo = duo(b.v[1], b.v[3]);
    ie = duo(dinv[st::cls(c, 0)], dinv[st::cls(c, 2)]);
    io = duo(dinv[st::cls(c, 1)], dinv[st::cls(c, 3)]);
  }
  // Half sweep of one colour: ((((b + up) + down) + left) + right) / d, the pair chosen by
  // selects (rows of both parities share a warp).
  __device__ __forceinline__ void half(Duo<T> *uE, Duo<T> *uO, int g, int GX, int colour) {
    const bool second = (colour + odd) & 1;
    Duo<T> *const u = second ? uO : uE;
    const T sv = second ? uE[ri].x : uO[li].y;
    const Duo<T> up = u[g - GX], dn = u[g + GX];
    const Duo<T> n = second ? e : o;  // the pair between the updated cells
    const Duo<T> left = duo(second ? n.x : sv, second ? n.y : n.x);
    const Duo<T> right = duo(second ? n.y : n.x, second ? sv : n.y);
    const Duo<T> r = mul2(add2(add2(add2(add2(second ? bo : be, up), dn), left), right),
                          second ? io : ie);
    u[g] = r;
    if (second) o = r;
    else e = r;
  }
  __device__ __forceinline__ st::V4<T> cells() const {
    st::V4<T> v;
    v.v[0] = e.x; v.v[1] = o.x; v.v[2] = e.y; v.v[3] = o.y;
    return v;
  }
};

// A half sweep of every group of the thread, then a barrier.
template <typename T, int NG, int GX, int IT, int NT>
__device__ __forceinline__ void tile_half(Group<T> (&q)[IT], Duo<T> *uE, Duo<T> *uO, int colour) {
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int g = threadIdx.x + it * NT;
    if (g < NG && q[it].sweeps) q[it].half(uE, uO, g, GX, colour);
  }
  __syncthreads();
}

// Restriction index of fine row / column f (Neumann mirrors the ghost at -1
// and, for an even size n, the ghost at n).
__device__ __forceinline__ int tmirror(int f, int n, bool neu) {
  if (neu) {
    if (f == -1) return 0;
    if (f == n && !(n & 1)) return n - 1;
  }
  return f;
}

// Down on one tile: S1 pre-sweeps from zero, the pre-smoothed iterate to w,
// residual, restriction (P^T) into the coarse right-hand side.  Called by the
// whole CTA (NT threads) for an active instance's tile; the CTA's shared
// memory is free on entry and may be reused on return.
template <typename T, int S1, int NT, int TY = kTY, int TX = kTX>
__device__ __forceinline__ void down_tile(const Args<T> &a, const Tile tl, const LevelInfo &L,
                                          const LevelInfo &Lc, unsigned char *smem) {
  using G = DownT<T, S1, TY, TX>;
  constexpr int RY = G::RY, H = G::H, GX = G::GX, NG = RY * GX, IT = (NG + NT - 1) / NT;
  Duo<T> *const uE = reinterpret_cast<Duo<T> *>(smem), *const uO = uE + NG;
  Duo<T> *const rE = uO + NG, *const rO = rE + NG;
  __shared__ T tdiag[8], tdinv[8];
  const int y0 = tl.ty * TY, x0 = tl.tx * TX;
  const int gy0 = y0 - H, gx0 = x0 - kHX;
  const int par0 = (gy0 + gx0) & 1;
  // the coarse cells this thread will write: row I, columns J, J + 1
  constexpr int CTY = TY / 2, QX = TX / 4;
  const int qy = threadIdx.x / QX, qx = threadIdx.x - qy * QX;
  const int I = (y0 >> 1) + qy, J = (x0 >> 1) + 2 * qx;
  const bool restricts = threadIdx.x < CTY * QX && I < Lc.ny && J < Lc.nx;
  static_assert(CTY * QX <= NT, "one coarse pair per thread");
  unsigned coarse_cls = 0x0101u;
  Group<T> q[IT];
  {
    const T *B = a.arena + L.b_off;
    st::V4<T> bv[IT];
    unsigned cv[IT];
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int g = threadIdx.x + it * NT;
      const int ry = g / GX, gx = g - ry * GX;
      const int y = gy0 + ry, x = gx0 + 4 * gx;
      bv[it] = g < NG ? load_group(B, L, y, x) : st::zero4<T>();
      cv[it] = g < NG ? row_classes(L, a.codes, y, x) : 0u;
    }
    if (restricts && Lc.code_off >= 0)
      coarse_cls = *reinterpret_cast<const unsigned short *>(a.codes + Lc.code_off +
                                                             (long long)I * Lc.pitch + J);
    diag_tables(tdiag, tdinv, L.wall);
    __syncthreads();
    // the first half sweep (colour 0 from zero): u = b / d
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int g = threadIdx.x + it * NT;
      if (g >= NG) break;
      q[it].place(g, RY, GX, par0, cv[it], bv[it], tdinv);
      const Duo<T> z = duo(T(0), T(0));
      q[it].e = q[it].odd ? z : mul2(q[it].be, q[it].ie);
      q[it].o = q[it].odd ? mul2(q[it].bo, q[it].io) : z;
      uE[g] = q[it].e;
      uO[g] = q[it].o;
    }
  }
  __syncthreads();
  tile_half<T, NG, GX, IT, NT>(q, uE, uO, 1);
#pragma unroll 1
  for (int s = 1; s < S1; ++s) {
    tile_half<T, NG, GX, IT, NT>(q, uE, uO, 0);
    tile_half<T, NG, GX, IT, NT>(q, uE, uO, 1);
  }
  T *const W = a.arena + L.w_off;
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int g = threadIdx.x + it * NT;
    const int ry = g / GX, gx = g - ry * GX;
    if (ry < H - 1 || ry > H + TY || gx < 1 || gx > QX + 2) continue;
    // the pre-smoothed iterate of the tile, for the up kernel
    if (ry >= H && ry < H + TY && gx >= 2 && gx < QX + 2)
      store_group(W, L, gy0 + ry, gx0 + 4 * gx, q[it].cells());
    // residual on the tile plus one ring
    const Duo<T> e = q[it].e, o = q[it].o;
    const Duo<T> ve = add2(uE[g - GX], uE[g + GX]), vo = add2(uO[g - GX], uO[g + GX]);
    const Duo<T> ne = add2(add2(ve, duo(uO[g - 1].y, o.x)), o);
    const Duo<T> no = add2(add2(vo, e), duo(e.y, uE[g + 1].x));
    auto res = [&](int j, T b, T u, T nbs) {
      const int k = st::cls(q[it].c, j);
      return k ? b - fma1(tdiag[k], u, -nbs) : T(0);
    };
    rE[g] = duo(res(0, q[it].be.x, e.x, ne.x), res(2, q[it].be.y, e.y, ne.y));
    rO[g] = duo(res(1, q[it].bo.x, o.x, no.x), res(3, q[it].bo.y, o.y, no.y));
  }
  __syncthreads();
  if (!restricts) return;
  const bool neu = L.bc == BC_NEU;
  T acc0 = T(0), acc1 = T(0);
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int g = (tmirror(2 * I - 1 + p, L.ny, neu) - gy0) * GX + qx + 2;
    const Duo<T> e = rE[g], o = rO[g];
    T v[6] = {rO[g - 1].y, e.x, o.x, e.y, o.y, rE[g + 1].x};  // columns 2 J - 1 .. 2 J + 4
    if (neu) {
      if (J == 0) v[0] = v[1];
      if (!(L.nx & 1)) {
#pragma unroll
        for (int m = 1; m < 6; ++m)
          if (2 * J - 1 + m == L.nx) v[m] = v[m - 1];
      }
    }
    const T w = (T)rweight(p);
    const T r0 = fma1(T(0.25), v[3], fma1(T(0.75), v[2], fma1(T(0.75), v[1], T(0.25) * v[0])));
    const T r1 = fma1(T(0.25), v[5], fma1(T(0.75), v[4], fma1(T(0.75), v[3], T(0.25) * v[2])));
    acc0 = p ? fma1(w, r0, acc0) : w * r0;
    acc1 = p ? fma1(w, r1, acc1) : w * r1;
  }
  T *Bc = a.arena + Lc.b_off + (long long)I * Lc.pitch + J;
  Bc[0] = (coarse_cls & 0xffu) ? acc0 : T(0);
  if (J + 1 < Lc.nx) Bc[1] = (coarse_cls >> 8) ? acc1 : T(0);
}

// Up on one tile: u = w + P e (bilinear; Neumann clamps at the edge, other
// boundaries read zero outside), then S2 post-sweeps, colour 1 first.  Same
// calling convention as down_tile.
template <typename T, int S2, int NT, int TY = kTY, int TX = kTX>
__device__ __forceinline__ void up_tile(const Args<T> &a, const Tile tl, const LevelInfo &L,
                                        const LevelInfo &Lc, unsigned char *smem) {
  using G = UpT<T, S2, TY, TX>;
  constexpr int RY = G::RY, H = G::H, GX = G::GX, CX = G::CX, NG = RY * GX;
  constexpr int IT = (NG + NT - 1) / NT;
  Duo<T> *const uE = reinterpret_cast<Duo<T> *>(smem), *const uO = uE + NG;
  T *const se = reinterpret_cast<T *>(uO + NG);
  __shared__ T tdiag[8], tdinv[8];
  const int y0 = tl.ty * TY, x0 = tl.tx * TX;
  const int gy0 = y0 - H, gx0 = x0 - kHX;
  const int par0 = (gy0 + gx0) & 1;
  const bool neu = L.bc == BC_NEU;
  // coarse correction around the region, from coarse row / column cy0 / cx0
  const int cy0 = (gy0 >> 1) - 1, cx0 = (gx0 >> 1) - 1;
  Group<T> q[IT];
  {  // every load of a thread is issued before the first is used
    const T *E = a.arena + Lc.u_off;
    const T *B = a.arena + L.b_off;
    const T *W = a.arena + L.w_off;
    constexpr int ITC = (G::CN + NT - 1) / NT;
    T ev[ITC];
    st::V4<T> bv[IT], wv[IT];
    unsigned cv[IT];
#pragma unroll
    for (int it = 0; it < ITC; ++it) {
      const int k = threadIdx.x + it * NT;
      const int ry = k / CX, rx = k - ry * CX;
      int cy = cy0 + ry, cx = cx0 + rx;
      bool ok = k < G::CN;
      if (neu) {
        cy = min(max(cy, 0), Lc.ny - 1);
        cx = min(max(cx, 0), Lc.nx - 1);
      } else {
        ok = ok && cy >= 0 && cy < Lc.ny && cx >= 0 && cx < Lc.nx;
      }
      ev[it] = ok ? E[(long long)cy * Lc.pitch + cx] : T(0);
    }
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int g = threadIdx.x + it * NT;
      const int ry = g / GX, gx = g - ry * GX;
      const int y = gy0 + ry, x = gx0 + 4 * gx;
      cv[it] = g < NG ? row_classes(L, a.codes, y, x) : 0u;
      bv[it] = g < NG ? load_group(B, L, y, x) : st::zero4<T>();
      wv[it] = g < NG ? load_group(W, L, y, x) : st::zero4<T>();
    }
    diag_tables(tdiag, tdinv, L.wall);
#pragma unroll
    for (int it = 0; it < ITC; ++it) {
      const int k = threadIdx.x + it * NT;
      if (k < G::CN) se[k] = ev[it];
    }
    __syncthreads();
    // u = w + P e on cells with an unknown
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int g = threadIdx.x + it * NT;
      if (g >= NG) break;
      q[it].place(g, RY, GX, par0, cv[it], bv[it], tdinv);
      const int ry = g / GX, gx = g - ry * GX;
      const int y = gy0 + ry;
      const int cy = y >> 1, cy2 = (y & 1) ? cy + 1 : cy - 1;
      // coarse columns x/2 - 1 .. x/2 + 2 of rows cy and cy2 (x = gx0 + 4 gx)
      const T *r1 = se + (cy - cy0) * CX + 2 * gx;
      const T *r2 = se + (cy2 - cy0) * CX + 2 * gx;
      T e1[4], e2[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        e1[k] = r1[k];
        e2[k] = r2[k];
      }
      auto cell = [&](int j, int m, int f) {  // near column m, far column f
        const T v = fma1(T(0.0625), e2[f], fma1(T(0.1875), e2[m] + e1[f], T(0.5625) * e1[m]));
        return st::cls(cv[it], j) ? wv[it].v[j] + v : T(0);
      };
      q[it].e = duo(cell(0, 1, 0), cell(2, 2, 1));
      q[it].o = duo(cell(1, 1, 2), cell(3, 2, 3));
      uE[g] = q[it].e;
      uO[g] = q[it].o;
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int s = 0; s < S2; ++s) {
    tile_half<T, NG, GX, IT, NT>(q, uE, uO, 1);
    tile_half<T, NG, GX, IT, NT>(q, uE, uO, 0);
  }
  T *const U = a.arena + L.u_off;
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int g = threadIdx.x + it * NT;
    const int ry = g / GX, gx = g - ry * GX;
    if (ry >= H && ry < H + TY && gx >= 2 && gx < TX / 4 + 2)
      store_group(U, L, gy0 + ry, gx0 + 4 * gx, q[it].cells());
  }
}

// One launch per level: a CTA per tile.  A level's coarse level is the next
// entry of the level table (levels of an instance are stored finest first), so
// the status word and both descriptors are requested together.
template <typename T, int S1, int NT = kThreads, int TY = kTY, int TX = kTX>
__global__ void __launch_bounds__(NT) k_down_t(Args<T> a) {
  const Tile tl = a.tiles[blockIdx.x];
  const LevelInfo L = a.lv[tl.level];
  const LevelInfo Lc = a.lv[tl.level + 1];
  dep_enter();
  if (a.st[tl.inst].status != GD_ACTIVE || !a.act[blockIdx.x]) return;
  extern __shared__ __align__(16) unsigned char smem[];
  down_tile<T, S1, NT, TY, TX>(a, tl, L, Lc, smem);
}

template <typename T, int S2, int NT = kThreads, int TY = kTY, int TX = kTX>
__global__ void __launch_bounds__(NT) k_up_t(Args<T> a) {
  const Tile tl = a.tiles[blockIdx.x];
  const LevelInfo L = a.lv[tl.level];
  const LevelInfo Lc = a.lv[tl.level + 1];
  dep_enter();
  if (a.st[tl.inst].status != GD_ACTIVE || !a.act[blockIdx.x]) return;
  extern __shared__ __align__(16) unsigned char smem[];
  up_tile<T, S2, NT, TY, TX>(a, tl, L, Lc, smem);
}

}  // namespace tile
}  // namespace gd
