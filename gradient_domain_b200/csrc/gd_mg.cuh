// Data structures and kernel declarations of the batched cell-centred MGPCG.
#pragma once

#include "gd_internal.cuh"

namespace gd {

// Hierarchy rules.  A level is coarsened (ceil(ny/2) x ceil(nx/2)) while it has
// more than kCoarsestCells cells; the first level with at most kBottomCells
// cells (a plan may choose another limit) whose levels down to the coarsest
// fit in kBottomSmem bytes of shared memory (padded b, u and classes) is
// handled, with everything below it, by one CTA per instance; the coarsest
// level is solved with a dense FP64 inverse.
constexpr int kCoarsestCells = 64;
constexpr int kBottomCells = 4096;
constexpr int kBottomSmem = 220 * 1024;
constexpr int kBottomLevels = 24;  // most levels one bottom holds
// Coarse levels (below level 0, above the bottom) with at most kTileCells cells, or
// kTileCellsMasked on masked instances, run on the shared-memory tile kernels; larger
// ones on the strips.  Time of an iteration on tiles over that on strips, by the cells of
// the level in question, one and three equal instances in the plan:
//                         280k   350k   392k   420k   490k   520k   560k   640k   800k  1000k
//   mixed             1  0.928  0.918  0.927  0.931  0.933  0.939  0.959  0.967  0.966  0.987
//                     3  0.983  0.977  0.994  1.014  1.010  1.015  1.030  1.031  1.045  1.058
//   FP64              1  0.941  0.968  0.972  0.965  0.967  0.973  1.007  1.018  1.021  1.041
//                     3  1.043  1.014  1.011  1.042  1.058  1.057  1.085  1.084  1.088  1.119
//   masked, a disc    1  0.938  0.956  0.948  0.956  0.958  0.957  0.959  0.955  0.971  0.967
//                     3  0.973  0.972  0.976  0.980  0.987  0.991  0.982  0.989  1.006  1.028
//   masked, FP64 disc 1  0.927  0.946  0.969  0.993  0.992  0.993  0.993  0.996  1.003  1.026
//   masked, all cells 3  0.988  0.976  0.985  0.999  1.011  1.017  1.012  1.017  1.029  1.042
// The more instances, the earlier the strips win, but the rule may look at one instance
// only, because the two kernels round differently and a batch gives every instance its own
// bits.  The lines lie where a colour image (three instances) changes sides: between 392k
// and 420k on rectangles in mixed precision (FP64 loses 1 % there and wins 3 % alone), and
// between 420k (every cell an unknown) and 800k (a disc) on masked levels, whose strips
// carry the classes' code.
constexpr int kTileCells = 3 << 17, kTileCellsMasked = 1 << 19;

// Tiles of the level-0 kernels that walk no strips (means, FP64 refresh, solution): 64 rows
// x 128 columns, 128 threads unless a kernel says otherwise.
constexpr int kFTY = 64, kFTX = 128, kFThreads = 128;
constexpr int kBThreads = 1024;    // bottom kernel

enum : int { BC_DIR = 0, BC_NEU = 1, BC_MASK = 2 };
// FLAG_RU: an FP64 refresh is due (set by cgupdate, cleared by the residual).
// FLAG_DZERO: the correction d restarts from zero (set when a solve starts and
// at every refresh, cleared by the next cgupdate, which then writes d = alpha p
// without reading the stale d, so nobody has to write zeros into it).
enum : int { FLAG_RU = 1, FLAG_DZERO = 2 };
// Slot of the plan's counter array that holds the device error word: bits set
// by a kernel whose bounded wait gave up, cleared when a solve starts.
constexpr int kErrWord = 15;

// Programmatic dependent launch.  The kernels of a solve may be launched with
// cudaLaunchAttributeProgrammaticStreamSerialization, which lets their CTAs be
// scheduled before the kernel ahead of them in the stream has finished.  Such a
// kernel reads only the plan's tables that no kernel writes (the tile lists and
// the level descriptors) before dep_wait(), which returns once the kernel
// ahead has completed and its writes are visible; then dep_release() lets the
// next kernel's CTAs be scheduled in turn.  Without the attribute both are
// no-ops.
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_release() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void dep_enter() {
  dep_wait();
  dep_release();
}

struct LevelInfo {
  int ny, nx, pitch, inst;
  int bc, level, coarse, is_bottom;
  float wall, pad0;
  int rows_per_warp;  // strip height of the down / up kernels on this level (even)
  // bottom levels: byte offsets of u (then the residual, up to b), b and the classes
  // in the bottom kernel's shared memory (BotLevel), of the FP64 right-hand side of
  // the dense solve (coarsest level; the dense inverse follows it at
  // sm_d + kCoarsestCells doubles) and the end of the layout
  int sm_b, sm_u, sm_c, sm_d, sm_end;
  long long b_off, u_off;  // element offsets into the T arena
  long long w_off;         // pre-smoothed iterate written by down, read by up
  long long code_off;      // byte offset into the code arena, -1 if rectangle
  long long inv_off;       // coarsest level: element offset of its dense inverse, else -1
};

struct InstInfo {
  int ny, nx, pitch, bc;
  int level0, bottom, coarsest, nlevels;
  long long r_off, p_off, d_off, z_off, q_off;  // p is double-buffered: p_off / q_off
  long long xs_off;  // the plan's own FP64 copy of the solution (element offset, row pitch `pitch`)
  int fine_begin, fine_end;  // tile range in the fine map
  int kr_begin, kr_end;      // tile range in the Krylov map
  int kr_rows;               // rows of its Krylov tiles (depends on the instance alone)
  int up0_begin, up0_end;    // range of its r.z group partials (empty if bottom is level 0)
  int up0_ctas;              // CTAs of the level-0 up kernel
  int zero_mean;
  int rz_rows;  // rows per r.z group partial: level 0's strip height for the instance alone
  // the bottom's top level and coarsest solve, as their levels have them
  int bot_ny, bot_nx, bot_pitch, bot_nq, bot_sm_d;
  long long bot_b_off, bot_u_off, bot_inv_off;
  // set per solve
  const double *f;
  double *x;
  long long upitch;
  double scale;
  double cells_active;
};

struct InstState {
  double rz, beta, pAp, alpha, rr, rr_ref, ff, rr_true, mean, fmean, rr_prev;
  int status, iters, flags, first;
  int pcur;  // which of the two p buffers holds the current direction
  int xcur;  // where the current solution is: 0 the caller's x, 1 the plan's copy
  int refreshes;  // FP64 refreshes after the initial residual
  int xzero;      // the solution is known to be zero (zero-start solve, nothing folded yet)
  int mean_known; // mean holds the solution's mean (set by a refresh that folds)
  unsigned ticket; // CTAs of the instance that have finished their part of a reduction
};

struct Tile {
  int level;  // LevelInfo index (fine level for down/up, level 0 for fine maps)
  int inst;
  int ty, tx;
};

// What the mask set-up does for one tile of a masked instance: act[tile] says whether
// any cell of the tile's own region (rows y0 .. y1 - 1, columns x0 .. x1 - 1 of its
// level; x0 a multiple of 4) holds an unknown.  Kernels return at once from a tile
// without one, so what they would have written there, zeros, is written by the
// set-up: r (kFine), both p buffers (kKrylov), the level's u (kUp, kTiles), its
// coarse level's b (kDown, kTiles).
enum : int { kFine = 0, kKrylov = 1, kDown = 2, kUp = 3, kTiles = 4 };
struct MaskItem {
  int tile, level, inst, kind;
  int y0, y1, x0, x1;
};

template <typename T>
struct Args {
  const LevelInfo *lv;
  const InstInfo *inst;
  InstState *st;
  T *arena;
  double *xs;  // the plan's FP64 solution copies
  const unsigned char *codes;
  const double *dense;
  double *part0;
  double *part1;
  unsigned *counter;
  int *n_active;
  const Tile *tiles;
  const unsigned char *act;  // per tile of `tiles`: holds an unknown (1 for rectangles)
  int ninst;
  double tol2, delta2;
  int max_iter;
  int zero_start;  // solves start from x = 0 without reading the caller's x
  // Conditional handles of the solve graph (0 in direct launches): the loop over
  // iterations, set by the initial residual while an instance is active and
  // cleared by the refresh that stops the last one; and the FP64 refresh of an
  // iteration, set by whoever asks for one (FLAG_RU) and cleared by the refresh.
  // trips counts the loop's iterations and ends it at trip_cap, whatever the
  // states say.
  cudaGraphConditionalHandle loop, refresh;
  int *trips;
  int trip_cap;
};

// Sets a condition of the solve graph (nothing in direct launches).
__device__ __forceinline__ void set_condition(cudaGraphConditionalHandle h, unsigned value) {
  if (h) cudaGraphSetConditional(h, value);
}

// Cell class: 0 = no unknown, else 1 + number of walls (missing neighbours).
__host__ __device__ __forceinline__ int rect_class(int y, int x, int ny, int nx) {
  return 1 + (y == 0) + (y == ny - 1) + (x == 0) + (x == nx - 1);
}

__device__ __forceinline__ int cell_class(const LevelInfo &L, const unsigned char *codes, int y,
                                          int x) {
  if (y < 0 || y >= L.ny || x < 0 || x >= L.nx) return 0;
  if (L.code_off >= 0) return codes[L.code_off + (long long)y * L.pitch + x];
  return rect_class(y, x, L.ny, L.nx);
}

// Diagonal of the positive operator for a cell of class c on a level with wall
// coefficient w: interior neighbours count 1, walls count w (Neumann w = 0,
// Dirichlet w = 1 on the finest level and 2 on coarse levels).
__host__ __device__ __forceinline__ double class_diag(int c, float w) {
  return 4.0 - (double)(c - 1) * (1.0 - (double)w);
}

}  // namespace gd
