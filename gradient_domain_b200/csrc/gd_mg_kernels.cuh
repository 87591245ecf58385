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
// `down` smooths from zero, forms the residual and restricts it; `up`
// recomputes that pre-smoothed iterate from b instead of storing it, adds P e
// and post-smooths.  Small levels run in `k_bottom` (this file), one CTA per
// instance, down to a dense FP64 solve.
#pragma once

#include <cuda_pipeline.h>

#include "gd_mg.cuh"

namespace gd {

__device__ __forceinline__ bool in_grid(const LevelInfo &L, int y, int x) {
  return y >= 0 && y < L.ny && x >= 0 && x < L.nx;
}

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

// The search direction lives in two buffers: k_pupdate reads the current one
// (including halo cells owned by other CTAs) and writes the other, so no CTA
// overwrites a value another CTA still has to read.
__device__ __forceinline__ long long p_offset(const InstInfo &I, int which) {
  return which ? I.q_off : I.p_off;
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

template <typename T>
__device__ __forceinline__ void make_tables(T *diag, T *dinv, float wall) {
  if (threadIdx.x < 8) {
    const int c = threadIdx.x;
    const double d = c >= 1 && c <= 5 ? class_diag(c, wall) : 1.0;
    diag[c] = (T)d;
    dinv[c] = (c >= 1 && c <= 5 && d > 0.0) ? (T)(1.0 / d) : (T)0;
  }
}

// Bilinear-adjoint weights of one axis for fine offsets 2I-1 .. 2I+2.
__device__ __forceinline__ float rweight(int a) { return (a == 0 || a == 3) ? 0.25f : 0.75f; }

// Neumann restriction reads the mirrored residual at fine index -1 and, for an
// even fine size n, at index n (the clamped ghost of P^T).
__device__ __forceinline__ int mirror_fine(int f, int n, bool neumann) {
  if (!neumann) return f;
  if (f == -1) return 0;
  if (f == n && !(n & 1)) return n - 1;
  return f;
}

// ---------------------------------------------------------------------------
// Bottom: the remaining V-cycle of one instance, every level in shared memory,
// one CTA of kBThreads threads per instance.
//
// Each level keeps b, u and the cell classes in arrays padded with a ring of
// zero ghosts (one row / column before the grid, two after; the restriction of
// an odd-sized level reaches two cells past its edge).  A missing neighbour
// then reads 0, as the operator defines, and Dirichlet / masked transfers read
// zero ghosts, so no stencil needs a bounds check.  A warp works on whole rows
// and its lanes on columns, so no index is divided.  The residual goes to its
// own array, so b stays in shared memory for the up pass; only the top level's
// b comes from (and its u goes back to) global memory.  The dense inverse of
// the coarsest level is copied in by cp.async while the down pass runs.

template <typename T>
__device__ __forceinline__ void bot_sweep(T *u, const T *b, const unsigned char *c, int ny,
                                          int nx, int px, const T *dinv, int colour) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int y = warp; y < ny; y += kBThreads / 32) {
    const int row = (y + 1) * px + 1;
    for (int x = 2 * lane + ((colour + y) & 1); x < nx; x += 64) {
      const int i = row + x;
      const int cl = c[i];
      if (cl) u[i] = (b[i] + u[i - px] + u[i + px] + u[i - 1] + u[i + 1]) * dinv[cl];
    }
  }
  __syncthreads();
}

// Padded index of fine row / column f for the restriction: Neumann mirrors the
// ghost at -1 and, for an even size n, the ghost at n (the adjoint of the
// clamped prolongation); every other ghost reads zero.
__device__ __forceinline__ int bot_mirror(int f, int n, bool neu) {
  if (neu) {
    if (f == -1) return 0;
    if (f == n && !(n & 1)) return n - 1;
  }
  return f;
}

// The few fields of a bottom level its phases read, staged in shared memory
// once per launch: every phase after a barrier then finds them at shared-memory
// latency instead of reloading the level descriptors from global memory.
struct BotLevel {
  int ny, nx, px, neu;
  int sm_b, sm_u, sm_r, sm_c;
};

// The bottom of one active instance, by the whole CTA (kBThreads threads); the
// CTA's shared memory is free on entry and may be reused on return.  Every
// phase runs on all warps: a phase's time is the chain of rows its busiest warp
// walks, so fewer warps on the small levels were measured slower.
template <typename T, int S1, int S2>
__device__ __forceinline__ void bottom_instance(const Args<T> &a, const int inst,
                                                unsigned char *smem) {
  InstState &S = a.st[inst];
  __shared__ T tdiag[kBottomLevels][8], tdinv[kBottomLevels][8];
  __shared__ BotLevel bl[kBottomLevels];
  const int bottom = a.inst[inst].bottom, coarsest = a.inst[inst].coarsest;
  const bool top_is_fine = bottom == a.inst[inst].level0;
  const int nb = coarsest - bottom + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int NW = kBThreads / 32;
  const int nq = a.lv[coarsest].ny * a.lv[coarsest].nx;
  const int sm_d = a.lv[coarsest].sm_d;
  double *const inv_s = reinterpret_cast<double *>(smem + sm_d) + kCoarsestCells;
  {  // the coarsest inverse travels while the levels above are worked on
    const double *inv_g = a.dense + a.lv[coarsest].inv_off;
    for (int k = threadIdx.x; k < nq * nq; k += kBThreads)
      __pipeline_memcpy_async(inv_s + k, inv_g + k, sizeof(double));
    __pipeline_commit();
  }
  {  // zero every padded array up to the inverse (ghost rings stay zero for the whole launch)
    const int bytes = sm_d + kCoarsestCells * (int)sizeof(double);
    uint4 *z = reinterpret_cast<uint4 *>(smem);
    for (int k = threadIdx.x; k < bytes / 16; k += kBThreads) z[k] = make_uint4(0, 0, 0, 0);
  }
  for (int q = threadIdx.x; q < nb * 8; q += kBThreads) {
    const int l = q >> 3, c = q & 7;
    const float w = a.lv[bottom + l].wall;
    const double d = c >= 1 && c <= 5 ? class_diag(c, w) : 1.0;
    tdiag[l][c] = (T)d;
    tdinv[l][c] = (c >= 1 && c <= 5 && d > 0.0) ? (T)(1.0 / d) : T(0);
    if (c == 0) {
      const LevelInfo &L = a.lv[bottom + l];
      bl[l] = BotLevel{L.ny, L.nx, L.sm_px, L.bc == BC_NEU ? 1 : 0, L.sm_b, L.sm_u, L.sm_r,
                       L.sm_c};
    }
  }
  __syncthreads();
  // classes of every level, and b of the top level
  for (int q = 0; q < nb; ++q) {
    const LevelInfo L = a.lv[bottom + q];
    unsigned char *c = smem + L.sm_c;
    const int px = L.sm_px;
    for (int y = warp; y < L.ny; y += NW)
      for (int x = lane; x < L.nx; x += 32)
        c[(y + 1) * px + 1 + x] = (unsigned char)cell_class(L, a.codes, y, x);
  }
  {
    const LevelInfo &L = a.lv[bottom];
    const T *B = a.arena + L.b_off;
    const long long pitch = L.pitch;
    const BotLevel Q = bl[0];
    T *b = reinterpret_cast<T *>(smem + Q.sm_b);
    for (int y = warp; y < Q.ny; y += NW)
      for (int x = lane; x < Q.nx; x += 32)
        b[(y + 1) * Q.px + 1 + x] = B[(long long)y * pitch + x];
  }
  __syncthreads();
  // down: smooth from zero, residual (into b), restriction
  for (int q = 0; q + 1 < nb; ++q) {
    const BotLevel L = bl[q];
    const BotLevel C = bl[q + 1];
    T *u = reinterpret_cast<T *>(smem + L.sm_u);
    const T *b = reinterpret_cast<const T *>(smem + L.sm_b);
    T *res = reinterpret_cast<T *>(smem + L.sm_r);
    const unsigned char *c = smem + L.sm_c;
    const int px = L.px;
    for (int s = 0; s < S1; ++s) {
      bot_sweep(u, b, c, L.ny, L.nx, px, tdinv[q], 0);
      bot_sweep(u, b, c, L.ny, L.nx, px, tdinv[q], 1);
    }
    for (int y = warp; y < L.ny; y += NW) {
      const int row = (y + 1) * px + 1;
      for (int x = lane; x < L.nx; x += 32) {
        const int i = row + x;
        const int cl = c[i];
        const T nbs = u[i - px] + u[i + px] + u[i - 1] + u[i + 1];
        res[i] = cl ? b[i] - (tdiag[q][cl] * u[i] - nbs) : T(0);
      }
    }
    __syncthreads();
    T *bc = reinterpret_cast<T *>(smem + C.sm_b);
    const unsigned char *cc = smem + C.sm_c;
    const bool neu = L.neu != 0;
    const int cpx = C.px;
    for (int Iy = warp; Iy < C.ny; Iy += NW) {
      int fy[4];
#pragma unroll
      for (int pp = 0; pp < 4; ++pp) fy[pp] = (bot_mirror(2 * Iy - 1 + pp, L.ny, neu) + 1) * px + 1;
      for (int Jx = lane; Jx < C.nx; Jx += 32) {
        const int ci = (Iy + 1) * cpx + 1 + Jx;
        T acc = T(0);
        if (cc[ci]) {
          int fx[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) fx[r] = bot_mirror(2 * Jx - 1 + r, L.nx, neu);
#pragma unroll
          for (int pp = 0; pp < 4; ++pp) {
            T rowv = T(0);
#pragma unroll
            for (int r = 0; r < 4; ++r) rowv += (T)rweight(r) * res[fy[pp] + fx[r]];
            acc += (T)rweight(pp) * rowv;
          }
        }
        bc[ci] = acc;
      }
    }
    __syncthreads();
  }
  const BotLevel Lc = bl[nb - 1];
  {  // coarsest: dense FP64 inverse, one warp per row
    const int n = Lc.ny * Lc.nx;
    const int px = Lc.px;
    double *bd = reinterpret_cast<double *>(smem + sm_d);
    const T *b = reinterpret_cast<const T *>(smem + Lc.sm_b);
    T *u = reinterpret_cast<T *>(smem + Lc.sm_u);
    for (int k = threadIdx.x; k < n; k += kBThreads) {
      const int y = k / Lc.nx, x = k - y * Lc.nx;
      bd[k] = (double)b[(y + 1) * px + 1 + x];
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
          u[(y + 1) * px + 1 + x] = (T)acc[r];
        }
      }
    }
    __syncthreads();
  }
  // up: reload b, add the prolonged correction, post-smooth
  for (int q = nb - 2; q >= 0; --q) {
    const BotLevel L = bl[q];
    const BotLevel C = bl[q + 1];
    T *u = reinterpret_cast<T *>(smem + L.sm_u);
    T *b = reinterpret_cast<T *>(smem + L.sm_b);
    const T *e = reinterpret_cast<const T *>(smem + C.sm_u);
    const unsigned char *c = smem + L.sm_c;
    const bool neu = L.neu != 0;
    const int px = L.px, cpx = C.px;
    for (int y = warp; y < L.ny; y += NW) {
      const int row = (y + 1) * px + 1;
      const int cy = y >> 1;
      int cy2 = (y & 1) ? cy + 1 : cy - 1;
      if (neu) cy2 = min(max(cy2, 0), C.ny - 1);
      const int r1 = (cy + 1) * cpx + 1, r2 = (cy2 + 1) * cpx + 1;
      for (int x = lane; x < L.nx; x += 32) {
        const int i = row + x;
        if (!c[i]) continue;
        const int cx = x >> 1;
        int cx2 = (x & 1) ? cx + 1 : cx - 1;
        if (neu) cx2 = min(max(cx2, 0), C.nx - 1);
        u[i] += (T)0.5625 * e[r1 + cx] + (T)0.1875 * (e[r2 + cx] + e[r1 + cx2]) +
                (T)0.0625 * e[r2 + cx2];
      }
    }
    __syncthreads();
    for (int s = 0; s < S2; ++s) {
      bot_sweep(u, b, c, L.ny, L.nx, px, tdinv[q], 1);
      bot_sweep(u, b, c, L.ny, L.nx, px, tdinv[q], 0);
    }
  }
  const BotLevel L0 = bl[0];
  const LevelInfo &G0 = a.lv[bottom];
  T *U = a.arena + G0.u_off;
  const long long pitch0 = G0.pitch;
  const T *u0 = reinterpret_cast<const T *>(smem + L0.sm_u);
  const T *b0 = reinterpret_cast<const T *>(smem + L0.sm_b);
  double part = 0.0;
  for (int y = warp; y < L0.ny; y += NW) {
    const int row = (y + 1) * L0.px + 1;
    for (int x = lane; x < L0.nx; x += 32) {
      const T v = u0[row + x];
      U[(long long)y * pitch0 + x] = v;
      part += (double)b0[row + x] * (double)v;
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
// Elementwise level-0 kernels over 64 x 128 tiles (the Krylov kernels with
// halos are in gd_stream.cuh).

// x += d for instances with a pending FP64 refresh (d then restarts from zero
// through FLAG_DZERO instead of being cleared here).  A thread owns one
// column of the 64 x 128 tile, so every warp access is 32 consecutive
// elements; the independent rows are unrolled for several loads in flight.
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
// drops it by zeroing the DC coefficient (solvers.py:258-261).
template <typename T>
__global__ void __launch_bounds__(kFThreads) k_fmean(Args<T> a) {
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
  const int Y0 = tl.ty * kFTY, gx = tl.tx * kFTX + threadIdx.x;
  const double part = gx < I.nx ? column_sum(I.f, I.upitch, Y0, min(Y0 + kFTY, I.ny), gx) : 0.0;
  double sum;
  if (instance_sum<kFThreads>(a.part0, I.fine_begin, I.fine_end - I.fine_begin, part,
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
__global__ void __launch_bounds__(kMaskThreads)
k_mask_levels(const LevelInfo *lv, int level0, int coarsest, unsigned char *codes,
              const unsigned char *mask, int mpitch, unsigned *ticket) {
  __shared__ unsigned char s[2][kMaskBlock * kMaskBlock];
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
    const LevelInfo &L = lv[level0 + l];
    const unsigned char *f = s[(l + 1) & 1];
    unsigned char *o = s[l & 1];
    for (int g = threadIdx.x; g < size * size; g += kMaskThreads) {
      const int ry = g / size, rx = g - ry * size;
      const unsigned char *q = f + 4 * ry * size + 2 * rx;  // the finer block is 2 size wide
      const unsigned char any = q[0] | q[1] | q[2 * size] | q[2 * size + 1];
      o[ry * size + rx] = any;
      const int y = (by >> l) + ry, x = (bx >> l) + rx;
      if (y < L.ny && x < L.nx) codes[L.code_off + (long long)y * L.pitch + x] = any;
    }
  }
  if (level0 + l > coarsest) return;  // the same for every CTA
  if (!last_of_instance(ticket, (int)gridDim.x)) return;
  for (; level0 + l <= coarsest; ++l) {
    const LevelInfo &F = lv[level0 + l - 1], &L = lv[level0 + l];
    for (int k = threadIdx.x; k < L.ny * L.nx; k += kMaskThreads) {
      const int y = k / L.nx, x = k - y * L.nx;
      unsigned char any = 0;
      for (int dy = 0; dy < 2; ++dy)
        for (int dx = 0; dx < 2; ++dx)
          if (2 * y + dy < F.ny && 2 * x + dx < F.nx)
            any |= __ldcg(codes + F.code_off + (long long)(2 * y + dy) * F.pitch + 2 * x + dx);
      codes[L.code_off + (long long)y * L.pitch + x] = any;
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
// keeps its elements (column tid % 64, every 16th row) in registers; each pivot's
// row and column go through shared memory, alternating between two copies so that
// a pivot costs one barrier (32 instances of 64 cells: 140 us with the matrix in
// shared memory on 256 threads and an index division per element).
constexpr int kInvThreads = 1024;
__global__ void __launch_bounds__(kInvThreads) k_coarse_inverse(const LevelInfo *lv,
                                                                const InstInfo *inst,
                                                                const unsigned char *codes,
                                                                double *dense) {
  static_assert(kCoarsestCells == 64 && kInvThreads == 1024, "four rows of a column per thread");
  const InstInfo &I = inst[blockIdx.x];
  const LevelInfo L = lv[I.coarsest];
  const int n = L.ny * L.nx;
  __shared__ unsigned char cls[kCoarsestCells];
  __shared__ double prow[2][kCoarsestCells], pcol[2][kCoarsestCells];
  for (int k = threadIdx.x; k < n; k += kInvThreads)
    cls[k] = (unsigned char)cell_class(L, codes, k / L.nx, k % L.nx);
  __syncthreads();
  const double reg = (L.bc == BC_NEU) ? 1.0 / n : 0.0;
  const int j = threadIdx.x & 63, i0 = threadIdx.x >> 6;
  double A[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = i0 + 16 * r;
    A[r] = 0.0;
    if (i >= n || j >= n) continue;
    const int yi = i / L.nx, xi = i - yi * L.nx, yj = j / L.nx, xj = j - yj * L.nx;
    double v = reg;
    if (!cls[i] || !cls[j]) {
      v = (i == j && !cls[i]) ? 1.0 : 0.0;
    } else if (i == j) {
      v += class_diag(cls[i], L.wall);
    } else if (abs(yi - yj) + abs(xi - xj) == 1) {
      v -= 1.0;
    }
    A[r] = v;
  }
  for (int k = 0; k < n; ++k) {
    double *row = prow[k & 1], *col = pcol[k & 1];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (i0 + 16 * r == k) row[j] = A[r];
      if (j == k) col[i0 + 16 * r] = A[r];
    }
    __syncthreads();
    const double inv = 1.0 / row[k];
    const double scaled = (j == k ? 1.0 : row[j]) * inv;  // the pivot row after its division
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = i0 + 16 * r;
      A[r] = i == k ? scaled : (j == k ? 0.0 : A[r]) - col[i] * scaled;
    }
  }
  double *out = dense + L.inv_off;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = i0 + 16 * r;
    if (i < n && j < n) out[i * n + j] = A[r];
  }
}

}  // namespace gd
