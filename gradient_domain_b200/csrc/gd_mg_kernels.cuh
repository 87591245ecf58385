// Kernels of the batched cell-centred MGPCG.  Included by gd_mg.cu only.
//
// Operator: A u = d_p u_p - sum of neighbour values, neighbours outside the
// grid or without an unknown contribute zero; d_p = 4 - walls * (1 - w) with
// w the level's wall coefficient.  On the finest level this is exactly
// -h^2 laplacian (Dirichlet, operators.py:86-107), -divergence(gradient(.))
// (Neumann, test_operators.py:51-57) or the masked Perez matrix negated
// (poisson.py:190-204).
//
// V-cycle (the B200 replacement of multigrid.py:184-215): cell-centred
// coarsening to ceil(n/2), bilinear prolongation P (weights 3/4, 1/4 per axis,
// Neumann ghosts mirror, Dirichlet ghosts zero), restriction R = P^T,
// red-black Gauss-Seidel with colour 0 then 1 before restriction and colour 1
// then 0 after prolongation, so the cycle is a symmetric operator.  Each level
// costs two passes over HBM (the register-streaming kernels of gd_stream.cuh):
// `down` smooths from zero, writes that iterate, forms the residual and restricts
// it; `up` reads the iterate back, adds P e and post-smooths.  Small levels run on
// shared-memory tiles (gd_tile.cuh) and in `k_bottom` (this file), one CTA per
// instance, down to a dense FP64 solve.
#pragma once

#include <cuda_pipeline.h>

#include "gd_mg.cuh"

namespace gd {

// Last-CTA handshake over the `ctas` CTAs of one instance: each calls it once;
// returns true in the last one.  The instance's ticket is zero again after it
// (the CTAs of the next kernel run after this one's), and since every instance
// has its own, its reductions finish side by side instead of one after another
// in the launch's last CTA.
__device__ __forceinline__ bool last_of_instance(unsigned *ticket, int ctas) {
  __shared__ bool am_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned prev = atomicAdd(ticket, 1u);
    am_last = (prev == (unsigned)ctas - 1u);
    if (am_last) *ticket = 0u;
  }
  __syncthreads();
  if (am_last) __threadfence();
  return am_last;
}

// Sum of `count` partials from `p` by the whole CTA in a fixed pattern; valid
// in thread 0.
template <int NT>
__device__ __forceinline__ double block_range_sum(const double *p, int count) {
  double s = 0.0;
#pragma unroll 8
  for (int k = threadIdx.x; k < count; k += NT) s += __ldcg(p + k);
  return block_sum<NT>(s);
}

// Per-instance reduction: this CTA's per-thread values become its partial
// (blockIdx.x, the instance's CTAs being `ctas` consecutive ones from `first`);
// the instance's last CTA returns true, with the sum of all of them in its
// thread 0.  The pattern depends on the instance alone, so a batch gives every
// instance the sums it gets alone.
template <int NT>
__device__ __forceinline__ bool instance_sum(double *part, int first, int ctas, double v,
                                             unsigned *ticket, double *sum) {
  v = block_sum<NT>(v);
  if (threadIdx.x == 0) part[blockIdx.x] = v;
  if (!last_of_instance(ticket, ctas)) return false;
  *sum = block_range_sum<NT>(part + first, ctas);
  return true;
}

__device__ __forceinline__ void finish_rz(InstState &S, double rz,
                                          cudaGraphConditionalHandle refresh) {
  if (!(rz > 0.0) || !isfinite(rz)) {
    S.status = GD_BREAKDOWN;
    S.flags |= FLAG_RU;
    set_condition(refresh, 1u);
    return;
  }
  S.beta = S.first ? 0.0 : rz / S.rz;
  S.first = 0;
  S.rz = rz;
}

// Bilinear-adjoint weights of one axis for fine offsets 2I-1 .. 2I+2.
__device__ __forceinline__ float rweight(int a) { return (a == 0 || a == 3) ? 0.25f : 0.75f; }

// Classes of the 4 cells x0..x0+3 of row y, packed one byte each.
__device__ __forceinline__ unsigned row_classes(const LevelInfo &L, const unsigned char *codes,
                                                int y, int x0) {
  if (y < 0 || y >= L.ny || x0 >= L.nx || x0 + 3 < 0) return 0u;
  if (L.code_off >= 0) {
    if (x0 < 0) return 0u;  // x0 is a multiple of 4: a lane is wholly left of the grid or in it
    return *reinterpret_cast<const unsigned *>(codes + L.code_off + (long long)y * L.pitch + x0);
  }
  const int wy = (y == 0) + (y == L.ny - 1);
  unsigned packed = 0u;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int x = x0 + j;
    if (x >= 0 && x < L.nx) {
      const unsigned c = 1u + wy + (x == 0) + (x == L.nx - 1);
      packed |= c << (8 * j);
    }
  }
  return packed;
}

// ---------------------------------------------------------------------------
// Bottom: the remaining V-cycle of one instance, every level in shared memory,
// one CTA of kBThreads threads per instance.
//
// What bounds it is the chain of phases (a half sweep, the residual, a transfer),
// each a barrier apart, and within a phase the shared-memory wavefronts and
// instructions of one SM.  A thread works on a group of four consecutive cells of
// a row, held as two same-colour pairs E = (v0, v2) and O = (v1, v3): a half sweep
// updates one pair, so it reads only that pair of the rows above and below and one
// scalar beside, and a thread's own u, b and diagonal inverses stay in registers
// for all sweeps of a level.  (One cell per lane and access with byte classes:
// 31.0 us a launch for 64 x 64 cells x 3 instances, 25.1 so; event times.)
//
// u and the residual carry a ring of zero ghosts (a row above, two below - the
// restriction of an odd-sized level reaches two cells past its edge - and one
// group between rows), so a missing neighbour reads 0, as the operator defines,
// and Dirichlet / masked transfers read zero ghosts.  Cells without an unknown,
// the last group's cells beyond the grid among them, have a zero diagonal inverse
// and stay zero.  The dense inverse of the coarsest level is copied in by cp.async
// while the down pass runs.

// Two same-colour cells.
template <typename T>
struct __align__(2 * sizeof(T)) Duo {
  T x, y;
};
template <typename T>
__device__ __forceinline__ Duo<T> duo(T x, T y) {
  Duo<T> r;
  r.x = x;
  r.y = y;
  return r;
}
__device__ __forceinline__ Duo<float> add2(Duo<float> a, Duo<float> b) {
  const float2 r = __fadd2_rn(make_float2(a.x, a.y), make_float2(b.x, b.y));
  return duo(r.x, r.y);
}
__device__ __forceinline__ Duo<double> add2(Duo<double> a, Duo<double> b) {
  return duo(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y));
}
__device__ __forceinline__ Duo<float> mul2(Duo<float> a, Duo<float> b) {
  const float2 r = __fmul2_rn(make_float2(a.x, a.y), make_float2(b.x, b.y));
  return duo(r.x, r.y);
}
__device__ __forceinline__ Duo<double> mul2(Duo<double> a, Duo<double> b) {
  return duo(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y));
}
__device__ __forceinline__ float fma1(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma1(double a, double b, double c) { return __fma_rn(a, b, c); }

// A bottom level, staged in shared memory once per launch: geometry and the byte
// offsets of its arrays.  Group (y, g) of u and the residual is element
// (y + 1) gp + g + 1 of their E and O arrays; of b and the classes, y gx + g.
struct BotLevel {
  int ny, nx, gx, gp, neu, groups, pitch;
  unsigned div;                 // ceil(2^32 / gx), 0 for gx == 1
  const unsigned char *codes;   // class bytes of a masked level, else null
  int uE, uO, rE, rO, bE, bO, c;
};

// Row and group of item k of a level.
__device__ __forceinline__ void bot_item(const BotLevel &L, int k, int *y, int *g) {
  *y = L.div ? (int)__umulhi((unsigned)k, L.div) : k;
  *g = k - *y * L.gx;
}

template <typename T>
__device__ __forceinline__ Duo<T> *bot_duo(unsigned char *smem, int off) {
  return reinterpret_cast<Duo<T> *>(smem + off);
}

// What a thread keeps of a group while it sweeps a level.
template <typename T>
struct BotGroup {
  Duo<T> e, o, be, bo, ie, io;
  int q, parity;  // element of u; parity of the row
  __device__ __forceinline__ void load(unsigned char *smem, const BotLevel &L, const T *dinv,
                                       int k) {
    int y, g;
    bot_item(L, k, &y, &g);
    q = (y + 1) * L.gp + g + 1;
    parity = y & 1;
    e = bot_duo<T>(smem, L.uE)[q];
    o = bot_duo<T>(smem, L.uO)[q];
    be = bot_duo<T>(smem, L.bE)[k];
    bo = bot_duo<T>(smem, L.bO)[k];
    const unsigned c = reinterpret_cast<const unsigned *>(smem + L.c)[k];
    ie = duo(dinv[c & 0xff], dinv[(c >> 16) & 0xff]);
    io = duo(dinv[(c >> 8) & 0xff], dinv[c >> 24]);
  }
  // The cells of `colour` (cell (y, x) has colour (y + x) & 1), all one pair:
  // ((((b + up) + down) + left) + right) / d.  Rows of both parities share a warp, so
  // the pair is chosen by selects, not by a branch that would run both.
  __device__ __forceinline__ void half(unsigned char *smem, const BotLevel &L, int colour) {
    const bool odd = (colour + parity) & 1;
    Duo<T> *const u = bot_duo<T>(smem, odd ? L.uO : L.uE);
    const T *const side = reinterpret_cast<const T *>(smem + (odd ? L.uE : L.uO)) +
                          (odd ? 2 * q + 2 : 2 * q - 1);
    const Duo<T> up = u[q - L.gp], dn = u[q + L.gp];
    const T sv = *side;
    const Duo<T> n = odd ? e : o;  // the pair between the updated cells
    const Duo<T> left = duo(odd ? n.x : sv, odd ? n.y : n.x);
    const Duo<T> right = duo(odd ? n.y : n.x, odd ? sv : n.y);
    const Duo<T> r = mul2(add2(add2(add2(add2(odd ? bo : be, up), dn), left), right),
                          odd ? io : ie);
    u[q] = r;
    if (odd) o = r;
    else e = r;
  }
};

// `sweeps` sweeps of a level, colour `first` first.  A thread's first group stays in
// registers; a level of more than kBThreads groups goes through shared memory for
// the others.  (Loops are not unrolled: every launch of this kernel starts with a
// cold instruction cache, and code that runs once costs its fetches.)
template <typename T>
__device__ __forceinline__ void bot_sweeps(unsigned char *smem, const BotLevel &L, const T *dinv,
                                           int first, int sweeps) {
  BotGroup<T> own;
  const bool has = threadIdx.x < L.groups;
  if (has) own.load(smem, L, dinv, threadIdx.x);
#pragma unroll 1
  for (int h = 0; h < 2 * sweeps; ++h) {
    const int colour = (first + h) & 1;
    if (has) own.half(smem, L, colour);
    if (L.groups > kBThreads)
#pragma unroll 1
      for (int k = threadIdx.x + kBThreads; k < L.groups; k += kBThreads) {
        BotGroup<T> more;
        more.load(smem, L, dinv, k);
        more.half(smem, L, colour);
      }
    __syncthreads();
  }
}

// Row or column f of a level of n for the restriction: Neumann mirrors the
// ghost at -1 and, for an even size n, the ghost at n (the adjoint of the
// clamped prolongation); every other ghost reads zero.
__device__ __forceinline__ int bot_mirror(int f, int n, bool neu) {
  if (neu) {
    if (f == -1) return 0;
    if (f == n && !(n & 1)) return n - 1;
  }
  return f;
}

// Cell (y, x) of an array stored as pairs (E and O at byte offsets oE and oO, `base` the
// element of the row's group 0).
template <typename T>
__device__ __forceinline__ T *bot_cell(unsigned char *smem, int oE, int oO, int base, int x) {
  return reinterpret_cast<T *>(smem + ((x & 1) ? oO : oE)) + 2 * (base + (x >> 2)) + ((x >> 1) & 1);
}

// The bottom of one active instance, by the whole CTA (kBThreads threads); the
// CTA's shared memory is free on entry and may be reused on return.
template <typename T, int S1, int S2>
__device__ __forceinline__ void bottom_instance(const Args<T> &a, const int inst,
                                                unsigned char *smem) {
  InstState &S = a.st[inst];
  __shared__ T tdiag[kBottomLevels][8], tdinv[kBottomLevels][8];
  __shared__ BotLevel bl[kBottomLevels];
  // the instance's entry holds all that the first loads need
  const InstInfo &I = a.inst[inst];
  const int bottom = I.bottom, nb = I.coarsest - bottom + 1;
  const bool top_is_fine = bottom == I.level0;
  const int nq = I.bot_nq, sm_d = I.bot_sm_d, tny = I.bot_ny, tnx = I.bot_nx;
  const long long tpitch = I.bot_pitch;
  const T *const Bg = a.arena + I.bot_b_off;
  T *const U = a.arena + I.bot_u_off;
  const double *const inv_g = a.dense + I.bot_inv_off;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int NW = kBThreads / 32;
  const int tgx = (tnx + 3) / 4;
  Duo<T> be = duo(T(0), T(0)), bo = be;  // b of the thread's first group of the top level
  {
    const int k = threadIdx.x, y = k / tgx, g = k - y * tgx;
    if (k < tny * tgx) {  // a row's padding up to its pitch holds zeros
      const T *p = Bg + y * tpitch + 4 * g;
      be = duo(p[0], p[2]);
      bo = duo(p[1], p[3]);
    }
  }
  double *const inv_s = reinterpret_cast<double *>(smem + sm_d) + kCoarsestCells;
  // the coarsest inverse travels while the levels above are worked on
#pragma unroll 1
  for (int k = threadIdx.x; k < nq * nq; k += kBThreads)
    __pipeline_memcpy_async(inv_s + k, inv_g + k, sizeof(double));
  __pipeline_commit();
  for (int q = threadIdx.x; q < nb * 8; q += kBThreads) {
    const int l = q >> 3, c = q & 7;
    const LevelInfo &L = a.lv[bottom + l];
    const double d = c >= 1 && c <= 5 ? class_diag(c, L.wall) : 1.0;
    tdiag[l][c] = (T)d;
    tdinv[l][c] = (c >= 1 && c <= 5 && d > 0.0) ? (T)(1.0 / d) : T(0);
    if (c == 0) {
      BotLevel B;
      B.ny = L.ny;
      B.nx = L.nx;
      B.gx = (L.nx + 3) / 4;
      B.gp = B.gx + 1;
      B.neu = L.bc == BC_NEU ? 1 : 0;
      B.groups = B.ny * B.gx;
      B.pitch = L.pitch;
      B.div = B.gx > 1 ? 0xffffffffu / (unsigned)B.gx + 1u : 0u;
      B.codes = L.code_off >= 0 ? a.codes + L.code_off : nullptr;
      const int ring = ((B.ny + 3) * B.gp + 1) * (int)sizeof(Duo<T>);
      const int plain = B.groups * (int)sizeof(Duo<T>);
      B.uE = L.sm_u;
      B.uO = B.uE + ring;
      B.rE = B.uO + ring;
      B.rO = B.rE + ring;
      B.bE = L.sm_b;
      B.bO = B.bE + plain;
      B.c = L.sm_c;
      bl[l] = B;
    }
  }
  __syncthreads();
  // zero u and the residual of every level (their ghosts stay zero); its classes
#pragma unroll 1
  for (int l = 0; l < nb; ++l) {
    const BotLevel &B = bl[l];
    uint4 *z = reinterpret_cast<uint4 *>(smem + B.uE);
    const int n16 = (B.bE - B.uE) / 16;
#pragma unroll 1
    for (int k = threadIdx.x; k < n16; k += kBThreads) z[k] = make_uint4(0, 0, 0, 0);
#pragma unroll 1
    for (int k = threadIdx.x; k < B.groups; k += kBThreads) {
      int y, g;
      bot_item(B, k, &y, &g);
      unsigned c;
      if (B.codes) {
        c = *reinterpret_cast<const unsigned *>(B.codes + (long long)y * B.pitch + 4 * g);
      } else {  // 1 + walls; the group's cells beyond the grid have class 0
        const unsigned in = (unsigned)min(B.nx - 4 * g, 4);
        c = (0x01010101u + 0x01010101u * ((y == 0) + (y == B.ny - 1))) >> (32 - 8 * in);
        if (g == 0) c += 1u;
        if (g == B.gx - 1) c += 1u << (8 * in - 8);
      }
      reinterpret_cast<unsigned *>(smem + B.c)[k] = c;
    }
  }
  {
    const BotLevel &B = bl[0];
    if (threadIdx.x < B.groups) {
      bot_duo<T>(smem, B.bE)[threadIdx.x] = be;
      bot_duo<T>(smem, B.bO)[threadIdx.x] = bo;
    }
#pragma unroll 1
    for (int k = threadIdx.x + kBThreads; k < B.groups; k += kBThreads) {
      int y, g;
      bot_item(B, k, &y, &g);
      const T *p = Bg + y * tpitch + 4 * g;
      bot_duo<T>(smem, B.bE)[k] = duo(p[0], p[2]);
      bot_duo<T>(smem, B.bO)[k] = duo(p[1], p[3]);
    }
  }
  __syncthreads();
  // down: smooth from zero, residual, restriction
#pragma unroll 1
  for (int l = 0; l + 1 < nb; ++l) {
    const BotLevel L = bl[l];
    const BotLevel C = bl[l + 1];
    bot_sweeps<T>(smem, L, tdinv[l], 0, S1);
    {
      const Duo<T> *uE = bot_duo<T>(smem, L.uE), *uO = bot_duo<T>(smem, L.uO);
#pragma unroll 1
      for (int k = threadIdx.x; k < L.groups; k += kBThreads) {
        int y, g;
        bot_item(L, k, &y, &g);
        const int q = (y + 1) * L.gp + g + 1;
        const unsigned c = reinterpret_cast<const unsigned *>(smem + L.c)[k];
        const Duo<T> e = uE[q], o = uO[q];
        const Duo<T> ve = add2(uE[q - L.gp], uE[q + L.gp]), vo = add2(uO[q - L.gp], uO[q + L.gp]);
        const Duo<T> ne = add2(add2(ve, duo(uO[q - 1].y, o.x)), o);
        const Duo<T> no = add2(add2(vo, e), duo(e.y, uE[q + 1].x));
        const Duo<T> be = bot_duo<T>(smem, L.bE)[k], bo = bot_duo<T>(smem, L.bO)[k];
        auto res = [&](unsigned cl, T b, T u, T nbs) {
          return cl ? b - fma1(tdiag[l][cl], u, -nbs) : T(0);
        };
        bot_duo<T>(smem, L.rE)[q] = duo(res(c & 0xff, be.x, e.x, ne.x),
                                        res((c >> 16) & 0xff, be.y, e.y, ne.y));
        bot_duo<T>(smem, L.rO)[q] = duo(res((c >> 8) & 0xff, bo.x, o.x, no.x),
                                        res(c >> 24, bo.y, o.y, no.y));
      }
    }
    __syncthreads();
    {  // coarse row I, fine group g: coarse columns 2 g and 2 g + 1 (none beyond the
       // coarse groups: a group whose cells are all in the grid's last odd column pair)
      const Duo<T> *rE = bot_duo<T>(smem, L.rE), *rO = bot_duo<T>(smem, L.rO);
      const bool neu = L.neu != 0;
#pragma unroll 1
      for (int k = threadIdx.x; k < C.ny * L.gx; k += kBThreads) {
        int I, g;
        bot_item(L, k, &I, &g);
        T acc0 = T(0), acc1 = T(0);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const int q = (bot_mirror(2 * I - 1 + p, L.ny, neu) + 1) * L.gp + g + 1;
          const Duo<T> e = rE[q], o = rO[q];
          T v[6] = {rO[q - 1].y, e.x, o.x, e.y, o.y, rE[q + 1].x};  // columns 4 g - 1 .. 4 g + 4
          if (neu) {
            if (g == 0) v[0] = v[1];
            if (!(L.nx & 1)) {
#pragma unroll
              for (int m = 1; m < 6; ++m)
                if (4 * g - 1 + m == L.nx) v[m] = v[m - 1];
            }
          }
          const T w = (T)rweight(p);
          const T r0 = fma1(T(0.25), v[3], fma1(T(0.75), v[2], fma1(T(0.75), v[1], T(0.25) * v[0])));
          const T r1 = fma1(T(0.25), v[5], fma1(T(0.75), v[4], fma1(T(0.75), v[3], T(0.25) * v[2])));
          acc0 = p ? fma1(w, r0, acc0) : w * r0;
          acc1 = p ? fma1(w, r1, acc1) : w * r1;
        }
        const int gc = I * C.gx + (g >> 1), hi = g & 1;  // cells 0, 1 or 2, 3 of the coarse group
        const unsigned c = reinterpret_cast<const unsigned *>(smem + C.c)[gc] >> (16 * hi);
        reinterpret_cast<T *>(bot_duo<T>(smem, C.bE) + gc)[hi] = (c & 0xff) ? acc0 : T(0);
        reinterpret_cast<T *>(bot_duo<T>(smem, C.bO) + gc)[hi] = (c & 0xff00) ? acc1 : T(0);
        // an odd number of fine groups leaves the last coarse group's upper half without one
        if ((L.gx & 1) && g == L.gx - 1) {
          reinterpret_cast<T *>(bot_duo<T>(smem, C.bE) + gc)[1] = T(0);
          reinterpret_cast<T *>(bot_duo<T>(smem, C.bO) + gc)[1] = T(0);
        }
      }
    }
    __syncthreads();
  }
  const BotLevel Lc = bl[nb - 1];
  {  // coarsest: dense FP64 inverse, one warp per row
    const int n = Lc.ny * Lc.nx;
    double *bd = reinterpret_cast<double *>(smem + sm_d);
    for (int k = threadIdx.x; k < n; k += kBThreads) {
      const int y = k / Lc.nx, x = k - y * Lc.nx;
      bd[k] = (double)*bot_cell<T>(smem, Lc.bE, Lc.bO, y * Lc.gx, x);
    }
    __pipeline_wait_prior(0);
    __syncthreads();
    // a warp's rows (at most kRowsPerWarp) are summed side by side, so their
    // shuffle reductions overlap
    constexpr int kRowsPerWarp = (kCoarsestCells + NW - 1) / NW;
    const double *inv = inv_s;
    double acc[kRowsPerWarp];
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r) {
      const int t = warp + r * NW;
      double v = 0.0;
      if (t < n)
        for (int j = lane; j < n; j += 32) v += inv[(long long)t * n + j] * bd[j];
      acc[r] = v;
    }
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r) acc[r] = warp_sum(acc[r]);
    if (lane == 0) {
#pragma unroll
      for (int r = 0; r < kRowsPerWarp; ++r) {
        const int t = warp + r * NW;
        if (t < n) {
          const int y = t / Lc.nx, x = t - y * Lc.nx;
          *bot_cell<T>(smem, Lc.uE, Lc.uO, (y + 1) * Lc.gp + 1, x) = (T)acc[r];
        }
      }
    }
    __syncthreads();
  }
  // up: add the prolonged correction, post-smooth
#pragma unroll 1
  for (int l = nb - 2; l >= 0; --l) {
    const BotLevel L = bl[l];
    const BotLevel C = bl[l + 1];
    const bool neu = L.neu != 0;
    Duo<T> *uE = bot_duo<T>(smem, L.uE), *uO = bot_duo<T>(smem, L.uO);
#pragma unroll 1
    for (int k = threadIdx.x; k < L.groups; k += kBThreads) {
      int y, g;
      bot_item(L, k, &y, &g);
      const unsigned c = reinterpret_cast<const unsigned *>(smem + L.c)[k];
      if (!c) continue;
      const int q = (y + 1) * L.gp + g + 1;
      const int cy = y >> 1;
      int cy2 = (y & 1) ? cy + 1 : cy - 1;
      if (neu) cy2 = min(max(cy2, 0), C.ny - 1);
      const int b1 = (cy + 1) * C.gp + 1, b2 = (cy2 + 1) * C.gp + 1;
      T e1[4], e2[4];  // coarse columns 2 g - 1 .. 2 g + 2 of the two rows
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        int x = 2 * g - 1 + m;
        if (neu) x = min(max(x, 0), C.nx - 1);
        e1[m] = *bot_cell<T>(smem, C.uE, C.uO, b1, x);
        e2[m] = *bot_cell<T>(smem, C.uE, C.uO, b2, x);
      }
      auto plus = [&](unsigned cl, T u, int m, int f) {  // near column m, far column f
        const T v = fma1(T(0.0625), e2[f],
                         fma1(T(0.1875), e2[m] + e1[f], T(0.5625) * e1[m]));
        return cl ? u + v : u;
      };
      const Duo<T> e = uE[q], o = uO[q];
      uE[q] = duo(plus(c & 0xff, e.x, 1, 0), plus((c >> 16) & 0xff, e.y, 2, 1));
      uO[q] = duo(plus((c >> 8) & 0xff, o.x, 1, 2), plus(c >> 24, o.y, 2, 3));
    }
    __syncthreads();
    bot_sweeps<T>(smem, L, tdinv[l], 1, S2);
  }
  const BotLevel L0 = bl[0];
  double part = 0.0;
#pragma unroll 1
  for (int k = threadIdx.x; k < L0.groups; k += kBThreads) {
    int y, g;
    bot_item(L0, k, &y, &g);
    const int q = (y + 1) * L0.gp + g + 1;
    const Duo<T> e = bot_duo<T>(smem, L0.uE)[q], o = bot_duo<T>(smem, L0.uO)[q];
    T *p = U + y * tpitch + 4 * g;
    const T v[4] = {e.x, o.x, e.y, o.y};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (4 * g + j < L0.nx) p[j] = v[j];
    if (top_is_fine) {
      const Duo<T> be = bot_duo<T>(smem, L0.bE)[k], bo = bot_duo<T>(smem, L0.bO)[k];
      part += ((double)be.x * (double)e.x + (double)bo.x * (double)o.x) +
              ((double)be.y * (double)e.y + (double)bo.y * (double)o.y);
    }
  }
  if (top_is_fine) {
    part = block_sum<kBThreads>(part);
    if (threadIdx.x == 0) finish_rz(S, part, a.refresh);
  }
}

// One CTA per instance.
template <typename T, int S1, int S2>
__global__ void __launch_bounds__(kBThreads, 1) k_bottom(Args<T> a) {
  dep_enter();
  if (a.st[blockIdx.x].status != GD_ACTIVE) return;
  extern __shared__ __align__(16) unsigned char smem[];
  bottom_instance<T, S1, S2>(a, blockIdx.x, smem);
}

// ---------------------------------------------------------------------------
// Elementwise level-0 kernels over 64 x 128 tiles (the Krylov kernels are in
// gd_krylov.cuh, the FP64 refresh in gd_stream.cuh).  A thread owns a column of the
// tile, so every warp access is 32 consecutive elements.

// Sum of column x over rows y0 .. y1 - 1 of an FP64 array, eight independent
// loads in flight per thread and a fixed summation tree.
__device__ __forceinline__ double column_sum(const double *A, long long pitch, int y0, int y1,
                                             int x) {
  double s[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) s[k] = 0.0;
  for (int yb = y0; yb < y1; yb += 8) {
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = yb + k < y1 ? A[(long long)(yb + k) * pitch + x] : 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) s[k] += v[k];
  }
  return ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
}

// Mean of the right-hand side of zero-mean (Neumann) instances: the constant
// component of f is outside the range of A and is dropped, as the DCT solver
// drops it by zeroing the DC coefficient (solvers.py:258-261).  Four threads share
// a column of a fine tile and each requests its 16 rows before it adds the first:
// one memory latency a tile (29-instance batch: 37 us a launch with one thread a
// column and eight rows at a time, 15 us).
constexpr int kMeanThreads = 512, kMeanRows = kFTY / (kMeanThreads / kFTX);
template <typename T>
__global__ void __launch_bounds__(kMeanThreads) k_fmean(Args<T> a) {
  const Tile tl = a.tiles[blockIdx.x];
  dep_enter();
  if (blockIdx.x == 0 && threadIdx.x == 0) {  // a solve starts
    a.counter[kErrWord] = 0u;
    *a.n_active = 0;
    *a.trips = 0;
  }
  const InstInfo &I = a.inst[tl.inst];
  if (!I.zero_mean) {
    if (blockIdx.x == I.fine_begin && threadIdx.x == 0) a.st[tl.inst].fmean = 0.0;
    return;
  }
  const int gx = tl.tx * kFTX + threadIdx.x % kFTX;
  const int y0 = tl.ty * kFTY + threadIdx.x / kFTX * kMeanRows;
  const double *f = I.f + y0 * I.upitch + gx;
  const long long pitch = I.upitch;
  const int rows = gx < I.nx ? I.ny - y0 : 0;
  double v[kMeanRows];
#pragma unroll
  for (int k = 0; k < kMeanRows; ++k) v[k] = k < rows ? f[k * pitch] : 0.0;
#pragma unroll
  for (int o = kMeanRows / 2; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < o; ++k) v[k] += v[k + o];
  double sum;
  if (instance_sum<kMeanThreads>(a.part0, I.fine_begin, I.fine_end - I.fine_begin, v[0],
                                 &a.st[tl.inst].ticket, &sum) &&
      threadIdx.x == 0)
    a.st[tl.inst].fmean = sum / ((double)I.ny * (double)I.nx);
}

// Mean removal for zero-mean (Neumann) instances: partial sums, then subtract.
template <typename T>
__global__ void __launch_bounds__(kFThreads) k_mean(Args<T> a) {
  const Tile tl = a.tiles[blockIdx.x];
  dep_enter();
  const InstInfo &I = a.inst[tl.inst];
  // only solutions no refresh has summed: a caller's x that met the tolerance at once
  if (!I.zero_mean || a.st[tl.inst].mean_known) return;
  const bool own = a.st[tl.inst].xcur != 0;
  const double *X = own ? a.xs + I.xs_off : I.x;
  const long long pitch = own ? (long long)I.pitch : I.upitch;
  const int Y0 = tl.ty * kFTY, gx = tl.tx * kFTX + threadIdx.x;
  const double part = gx < I.nx ? column_sum(X, pitch, Y0, min(Y0 + kFTY, I.ny), gx) : 0.0;
  double sum;
  if (instance_sum<kFThreads>(a.part0, I.fine_begin, I.fine_end - I.fine_begin, part,
                              &a.st[tl.inst].ticket, &sum) &&
      threadIdx.x == 0)
    a.st[tl.inst].mean = sum / ((double)I.ny * (double)I.nx);
}

// The solution into the caller's buffer: x - mean for zero-mean instances, a
// copy when the last refresh left the solution in the plan's own copy, zeros
// when a zero-start solve ended without folding a correction (the caller's x
// was never read and may hold anything).
template <typename T>
__global__ void __launch_bounds__(kFThreads) k_submean(Args<T> a) {
  const Tile tl = a.tiles[blockIdx.x];
  dep_enter();
  const InstInfo &Ig = a.inst[tl.inst];
  const bool own = a.st[tl.inst].xcur != 0;
  // tiles without unknowns are zero, and no refresh writes them
  const bool idle = !a.act[blockIdx.x];
  const bool xz = idle || a.st[tl.inst].xzero != 0;
  if (!Ig.zero_mean && !own && !xz) return;
  const int ny = Ig.ny, nx = Ig.nx;
  const long long upitch = Ig.upitch;
  double *const X = Ig.x;
  const double *const src = own ? a.xs + Ig.xs_off : X;
  const long long spitch = own ? (long long)Ig.pitch : upitch;
  const double m = Ig.zero_mean ? a.st[tl.inst].mean : 0.0;
  const int Y0 = tl.ty * kFTY, gx = tl.tx * kFTX + threadIdx.x;
  if (gx >= nx) return;
  const int y1 = min(Y0 + kFTY, ny);
  for (int yb = Y0; yb < y1; yb += 8) {
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      v[k] = (yb + k < y1 && !xz) ? src[(long long)(yb + k) * spitch + gx] : 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (yb + k < y1) X[(long long)(yb + k) * upitch + gx] = v[k] - m;
  }
}

// ---------------------------------------------------------------------------
// Setup kernels.

// Activity (0 / 1) of every level of a masked instance from the caller's unknown
// mask, in one launch: a coarse cell has an unknown when any of its children has.
// A CTA reduces 64 x 64 cells of the mask through shared memory down to one cell
// of level 6; the last one carries the few cells left to the coarsest level.
constexpr int kMaskBlock = 64, kMaskThreads = 256;
constexpr int kMaxMaskLevels = 32;  // sides below 2^31 have at most this many levels
__global__ void __launch_bounds__(kMaskThreads)
k_mask_levels(const LevelInfo *lv, int level0, int coarsest, unsigned char *codes,
              const unsigned char *mask, int mpitch, unsigned *ticket) {
  __shared__ unsigned char s[2][kMaskBlock * kMaskBlock];
  // every level's descriptor at once, so that no level of the pyramid waits for its own
  struct Level {
    int ny, nx, pitch;
    unsigned char *c;
  };
  __shared__ Level lev[kMaxMaskLevels];
  if (threadIdx.x <= coarsest - level0) {
    const LevelInfo &L = lv[level0 + threadIdx.x];
    lev[threadIdx.x] = Level{L.ny, L.nx, L.pitch, codes + L.code_off};
  }
  const int across = (lv[level0].nx + kMaskBlock - 1) / kMaskBlock;  // blocks of a row
  const int by = (int)blockIdx.x / across * kMaskBlock, bx = (int)blockIdx.x % across * kMaskBlock;
  {
    const LevelInfo &L = lv[level0];
    const int ny = L.ny, nx = L.nx, pitch = L.pitch;
    unsigned char *c = codes + L.code_off;
    for (int g = threadIdx.x; g < kMaskBlock * kMaskBlock / 4; g += kMaskThreads) {
      const int ry = g / (kMaskBlock / 4), rx = 4 * (g % (kMaskBlock / 4));
      const int y = by + ry, x = bx + rx;
      unsigned packed = 0u;
      if (y < ny)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (x + j < nx && mask[(long long)y * mpitch + x + j]) packed |= 1u << (8 * j);
      *reinterpret_cast<unsigned *>(&s[0][ry * kMaskBlock + rx]) = packed;
      if (y < ny && x < pitch) *reinterpret_cast<unsigned *>(c + (long long)y * pitch + x) = packed;
    }
  }
  int l = 1;
  for (int size = kMaskBlock / 2; size >= 1 && level0 + l <= coarsest; size >>= 1, ++l) {
    __syncthreads();
    const Level L = lev[l];
    const unsigned char *f = s[(l + 1) & 1];
    unsigned char *o = s[l & 1];
    for (int g = threadIdx.x; g < size * size; g += kMaskThreads) {
      const int ry = g / size, rx = g - ry * size;
      const unsigned char *q = f + 4 * ry * size + 2 * rx;  // the finer block is 2 size wide
      const unsigned char any = q[0] | q[1] | q[2 * size] | q[2 * size + 1];
      o[ry * size + rx] = any;
      const int y = (by >> l) + ry, x = (bx >> l) + rx;
      if (y < L.ny && x < L.nx) L.c[(long long)y * L.pitch + x] = any;
    }
  }
  if (level0 + l > coarsest) return;  // the same for every CTA
  if (!last_of_instance(ticket, (int)gridDim.x)) return;
  for (; level0 + l <= coarsest; ++l) {
    const Level F = lev[l - 1], L = lev[l];
    for (int k = threadIdx.x; k < L.ny * L.nx; k += kMaskThreads) {
      const int y = k / L.nx, x = k - y * L.nx;
      unsigned char any = 0;
      for (int dy = 0; dy < 2; ++dy)
        for (int dx = 0; dx < 2; ++dx)
          if (2 * y + dy < F.ny && 2 * x + dx < F.nx)
            any |= __ldcg(F.c + (long long)(2 * y + dy) * F.pitch + 2 * x + dx);
      L.c[(long long)y * L.pitch + x] = any;
    }
    __syncthreads();
  }
}

// Rows y0 .. y1 - 1, columns x0 .. x1 - 1 of an array set to zero by the whole CTA.
template <typename T>
__device__ __forceinline__ void zero_region(T *A, int pitch, int y0, int y1, int x0, int x1) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  for (int y = y0 + warp; y < y1; y += warps)
    for (int x = x0 + lane; x < x1; x += 32) A[(long long)y * pitch + x] = T(0);
}

// The rest of the mask set-up, for all masked instances in one launch: activity to
// classes (1 + walls) on every level - CTAs 0 .. nclass - 1, a 32 x 128 block each -
// and the activity of every tile (MaskItem).  A class is non-zero exactly where the
// activity was, so neighbours may be read before or after they are converted, and
// the tiles need not wait for the classes.
constexpr int kClassRows = 32, kClassCols = 128, kSetupThreads = 128;
template <typename T>
__global__ void __launch_bounds__(kSetupThreads)
k_mask_setup(const LevelInfo *lv, const InstInfo *inst, unsigned char *codes, T *arena,
             const Tile *blocks, int nclass, const MaskItem *items, unsigned char *act) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int NW = kSetupThreads / 32;
  if ((int)blockIdx.x < nclass) {
    const Tile b = blocks[blockIdx.x];
    const LevelInfo &L = lv[b.level];
    const int ny = L.ny, nx = L.nx, pitch = L.pitch;
    unsigned char *c = codes + L.code_off;
    const int x = b.tx * kClassCols + 4 * lane;
    if (x >= nx) return;
    const int y1 = min((b.ty + 1) * kClassRows, ny);
    for (int y = b.ty * kClassRows + warp; y < y1; y += NW) {
      unsigned char *row = c + (long long)y * pitch + x;
      const unsigned own = *reinterpret_cast<const unsigned *>(row);
      if (!own) continue;
      const unsigned up = y > 0 ? *reinterpret_cast<const unsigned *>(row - pitch) : 0u;
      const unsigned dn = y + 1 < ny ? *reinterpret_cast<const unsigned *>(row + pitch) : 0u;
      const unsigned left = x > 0 ? row[-1] : 0u, right = x + 4 < nx ? row[4] : 0u;
      unsigned packed = 0u;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const unsigned m = 0xffu << (8 * j);
        if (!(own & m)) continue;
        const bool l = j == 0 ? left != 0u : (own & (m >> 8)) != 0u;
        const bool r = j == 3 ? right != 0u : (own & (m << 8)) != 0u;
        packed |= (1u + !(up & m) + !(dn & m) + !l + !r) << (8 * j);
      }
      *reinterpret_cast<unsigned *>(row) = packed;
    }
    return;
  }
  const MaskItem it = items[blockIdx.x - nclass];
  const LevelInfo &L = lv[it.level];
  const int pitch = L.pitch;
  const unsigned char *c = codes + L.code_off;
  unsigned any = 0u;
  for (int y = it.y0 + warp; y < it.y1; y += NW)
    for (int x = it.x0 + 4 * lane; x < it.x1; x += 128)
      any |= *reinterpret_cast<const unsigned *>(c + (long long)y * pitch + x);
  const bool on = __syncthreads_or(any != 0u);
  if (threadIdx.x == 0) act[it.tile] = on ? 1 : 0;
  if (on) return;
  const InstInfo &I = inst[it.inst];
  if (it.kind == kFine) zero_region(arena + I.r_off, pitch, it.y0, it.y1, it.x0, it.x1);
  if (it.kind == kKrylov) {
    zero_region(arena + I.p_off, pitch, it.y0, it.y1, it.x0, it.x1);
    zero_region(arena + I.q_off, pitch, it.y0, it.y1, it.x0, it.x1);
  }
  if (it.kind == kUp || it.kind == kTiles)
    zero_region(arena + L.u_off, pitch, it.y0, it.y1, it.x0, it.x1);
  if (it.kind == kDown || it.kind == kTiles) {
    const LevelInfo &C = lv[it.level + 1];
    zero_region(arena + C.b_off, C.pitch, it.y0 / 2, (it.y1 + 1) / 2, it.x0 / 2, (it.x1 + 1) / 2);
  }
}

// Dense FP64 inverse of the coarsest operator of each instance by in-place
// Gauss-Jordan (the matrix is SPD, or SPD after adding J/n for Neumann).  A thread
// keeps 4 x 4 elements in registers (rows ti + 16 a, columns tj + 16 b).  Each pivot's
// row and column go through shared memory, in two copies by turns, so that a pivot
// costs one barrier; with the pivot's own row and column cleared and -1 in its place
// in the column, one multiply-add serves every element.  The next pivot's owner
// divides once for all.  (32 instances of 64 cells: 140 us with the matrix in shared
// memory and an index division per element, 37 us with 1024 threads of four elements,
// 30 us.)
constexpr int kInvThreads = 256;
__global__ void __launch_bounds__(kInvThreads) k_coarse_inverse(const LevelInfo *lv,
                                                                const InstInfo *inst,
                                                                const unsigned char *codes,
                                                                double *dense) {
  static_assert(kCoarsestCells == 64, "16 x 16 threads of 4 x 4 elements");
  const InstInfo &I = inst[blockIdx.x];
  const LevelInfo L = lv[I.coarsest];
  const int n = L.ny * L.nx;
  __shared__ unsigned char cls[kCoarsestCells];
  __shared__ double prow[2][kCoarsestCells], pcol[2][kCoarsestCells], pinv[2];
  for (int k = threadIdx.x; k < n; k += kInvThreads)
    cls[k] = (unsigned char)cell_class(L, codes, k / L.nx, k % L.nx);
  __syncthreads();
  const double reg = (L.bc == BC_NEU) ? 1.0 / n : 0.0;
  const int ti = threadIdx.x >> 4, tj = threadIdx.x & 15;
  double A[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = ti + 16 * r, j = tj + 16 * c;
      double v = i == j ? 1.0 : 0.0;  // rows and columns beyond n: the identity
      if (i < n && j < n) {
        const int yi = i / L.nx, xi = i - yi * L.nx, yj = j / L.nx, xj = j - yj * L.nx;
        v = reg;
        if (!cls[i] || !cls[j]) {
          v = (i == j && !cls[i]) ? 1.0 : 0.0;
        } else if (i == j) {
          v += class_diag(cls[i], L.wall);
        } else if (abs(yi - yj) + abs(xi - xj) == 1) {
          v -= 1.0;
        }
      }
      A[r][c] = v;
    }
  if (threadIdx.x == 0) pinv[0] = 1.0 / A[0][0];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
#pragma unroll 1
    for (int t = 0; t < 16; ++t) {
      const int k = 16 * q + t;
      if (k >= n) break;
      double *row = prow[k & 1], *col = pcol[k & 1];
      if (ti == t) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          row[tj + 16 * c] = tj + 16 * c == k ? 1.0 : A[q][c];
          if (tj + 16 * c != k) A[q][c] = 0.0;
        }
      }
      if (tj == t) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          col[ti + 16 * r] = ti + 16 * r == k ? -1.0 : A[r][q];
          A[r][q] = 0.0;
        }
      }
      __syncthreads();
      const double inv = pinv[k & 1];
      double rs[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) rs[c] = row[tj + 16 * c] * inv;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const double f = col[ti + 16 * r];
#pragma unroll
        for (int c = 0; c < 4; ++c) A[r][c] -= f * rs[c];
      }
      if (ti == tj && ti == ((t + 1) & 15)) {  // the thread of pivot k + 1
        double d = A[q][q];
        if (t == 15 && q < 3) d = A[q < 3 ? q + 1 : 3][q < 3 ? q + 1 : 3];
        pinv[(k + 1) & 1] = 1.0 / d;
      }
    }
  }
  double *out = dense + L.inv_off;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = ti + 16 * r, j = tj + 16 * c;
      if (i < n && j < n) out[i * n + j] = A[r][c];
    }
}

}  // namespace gd
