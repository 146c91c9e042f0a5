// mg_solver.cu -- multigrid-preconditioned conjugate gradients for the same
// discrete system the red-black SOR path solves, behind PT_FLAG_MULTIGRID.
//
// The system and its stopping bar are the reference's (crates/paintop-cpu/src/
// poisson.rs): interior cells are mask > 0.5 off the image border (:340-355),
// b is the guidance Laplacian fma(4, -c, L + R + U + D) (:364-373), non-interior
// cells hold the anchor, the residual is
//   r = fma(lambda + 4, -u, nsum) - fma(lambda, -anchor, b)        (:315-321)
// and a channel has converged when ||r|| <= tolerance * ||r(anchor)||, ||.||
// taken in FP64. What differs is the iteration: instead of thousands of
// sweeps, each outer step solves the correction equation A e = r
// (A = (4 + lambda) I - adjacency over interior cells) with conjugate
// gradients in FP32, preconditioned by one symmetric multigrid V-cycle, and
// adds e to the FP64 solution; the FP64 residual decides when to stop.
//
// Multigrid (cell-centred): level k halves level k-1 (ceil), a coarse cell is
// active when at least 3 of its 2 x 2 children are; the level-k operator is
// (4 e - sum of active neighbours) / 4^k + lambda e with zero outside the
// active cells; prolongation is bilinear (weights 3/4, 1/4 per axis) into
// active fine cells and restriction its transpose / 4; smoothing is red-black
// SOR (kSmoothOmega; plain Gauss-Seidel on the coarsest level), red then black
// before the coarse correction and black then red after it, so the V-cycle is
// a symmetric operator and a valid CG preconditioner. The channels of an image
// share its level masks. Every reduction is a fixed-order tree, so a rerun is
// byte-identical.
//
// Batches: every problem of a call (pt_poisson_solve_batch) keeps its own
// level hierarchy, its own CG scalars per channel and its own stopping, but
// all of them share each launch. A launch walks a table of blocks, each block
// a few strips (or one 32 x 8 tile) of one instance's plane. Sums are taken by
// bands of rows of an instance's plane, whatever the strips; every other value
// is computed from values no other block of the launch writes, so it does not
// depend on them either. An instance's results are therefore bit for bit what
// it gets when solved alone. An (instance, channel) pair whose run has stopped
// skips the launches.
//
// Report (pt_report): iterations = preconditioned CG iterations (each one
// V-cycle and one operator application); history[k] = relative residual after
// iteration k -- the CG recurrence's estimate scaled by the outer step's FP64
// residual, replaced by the exact FP64 value at the end of every outer step;
// refinements = outer steps after the first; omega_used = the smoother's
// relaxation factor. Stop reasons: converged at the FP64 bar; max-iterations
// when the CG iterations reach max_iterations; stalled when an outer step fails to
// lower the FP64 residual, or at once (0 iterations, interior set to NaN)
// when a NaN or infinity in the inputs makes the residual non-finite.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/paintop_cuda.h"
#include "ctx.h"
#include "quotient.h"

namespace {

constexpr double kInnerFloor = 2e-6;  // deepest relative reduction asked of one FP32 CG run

// Assembly, coarsening and output run on tiles of (32, 8) threads over columns
// and rows; a tile strides over the rows of its instance's plane. The other
// kernels run on strips (below), grid.z is the channel.
constexpr int kTx = 32, kTy = 8;

// One instance's plane as one launch cuts it. The blocks of a launch are the
// instances' tiles, or their strips kStripWarps a block, one after another;
// bmap[blockIdx.x] names the entry. Rows are P apart, a multiple of four.
struct Geo {
  int W, H, P;        // the plane (coarsening: the coarse one)
  int gx, gy;         // tiles across and striding the rows; strip columns and strips down a column
  int rows;           // rows of a strip, a multiple of kBand
  int blk0;           // the instance's first block in the launch
  int C;              // its channels
  int unit0;          // its first (instance, channel) unit: CG scalars, scales, run flags, reductions
  int pad;
  long long part0;    // its first partial sum: C times one a band and strip column of level 0, channel-major
  long long f;        // its first band flag of the level
  long long o, oc;    // the plane's first cell in its level's one-channel (interior flags) and C-channel arrays
  long long o2, oc2;  // the same for the other plane of a two-level kernel
  int W2, H2, P2;     // that plane (coarsening: the fine level; else: the coarse level)
  float s, d;         // the level's 4^-k and diagonal 4^(1-k) + lambda
  double lambda;
};

// The block's entry, the entry's first unit and its channels: from the block
// table, or -- a launch over one instance, bmap null -- from the kernel's own
// parameter `one`, with no load before the block's first data.
__device__ __forceinline__ int4 entry_of(const int4 *__restrict__ bmap, const Geo &one) {
  return bmap ? bmap[blockIdx.x] : make_int4(0, one.unit0, one.C, 0);
}

// Which tile of its instance a block works on
__device__ __forceinline__ int tile_b(const Geo &g) { return (int)blockIdx.x - g.blk0; }

// Per-unit CG scalars: sc[unit] = {rho, beta, p.q}
enum { S_RHO, S_BETA, S_PQ, S_N };

// The caller-side buffers of one instance (device memory: the caller's, or
// the staged copies of host buffers)
struct Io {
  const float *guid, *anchor, *mask, *guess;
  float *out;
};

// Strips (below): columns, those owned, the halo either side; rows of a band, and
// one flag a band and strip column: it has active cells among the owned ones.
constexpr int kStripCols = 128, kStripStep = 112, kStripHalo = 8;
constexpr int kStripWarps = 4;   // per block
constexpr int kBand = 8;

__host__ __device__ inline int strip_cols(int w) {
  return w <= kStripCols ? 1 : 1 + (w - kStripCols + kStripStep - 1) / kStripStep;
}

// The flag of active cell (i, j)'s band (several threads may set one; all were
// cleared before). With a kernel a level for them, reading the interior flags again,
// a call without iterations took 129 us on 300 x 200, now 97.
__device__ __forceinline__ void set_flag(const Geo &g, uint8_t *__restrict__ flags, int i, int j) {
  const int gx = strip_cols(g.W), sx = i < kStripHalo ? 0 : min((i - kStripHalo) / kStripStep, gx - 1);
  flags[g.f + (long long)(j / kBand) * gx + sx] = 1;
}

// ---- assembly ----------------------------------------------------------------
// interior flag, u = anchor (or the warm guess at interior cells), b' =
// fma(lambda, -anchor, laplacian(guidance)) at interior cells; level-0 tiles,
// grid.z 1 (each thread does all channels of its cells).
__global__ void __launch_bounds__(kTx * kTy) k_mg_assemble(const Geo *__restrict__ geo,
                                                           const int4 *__restrict__ bmap, const Geo one,
                                                           const Io *__restrict__ io, uint8_t *__restrict__ act,
                                                           uint8_t *__restrict__ flags,
                                                           double *__restrict__ u, double *__restrict__ bl,
                                                           double *__restrict__ uw) {
  const int4 bt = entry_of(bmap, one);
  const int gi = bt.x;
  const Geo g = bmap ? geo[gi] : one;
  const Io f = io[gi];
  const int C = g.C, W = g.W, H = g.H, b = tile_b(g), i = (b % g.gx) * kTx + threadIdx.x;
  const size_t N = (size_t)g.P * H;
  uint8_t *a = act + g.o;
  double *u0 = u + g.oc, *b0 = bl + g.oc, *w0 = uw ? uw + g.oc : nullptr;
  for (int j = (b / g.gx) * kTy + threadIdx.y; j < H && i < g.P; j += g.gy * kTy) {
    const size_t k = (size_t)j * g.P + i, q = (size_t)j * W + i;
    if (i >= W) {  // padding
      a[k] = 0;
      continue;
    }
    auto interior = [&](int x, int y) {
      return W >= 3 && H >= 3 && x > 0 && y > 0 && x < W - 1 && y < H - 1 && f.mask[(size_t)y * W + x] > 0.5f;
    };
    const bool in = interior(i, j);
    a[k] = in ? 1 : 0;
    if (in) set_flag(g, flags, i, j);
    // u is read at interior cells and their neighbours, b' at interior cells:
    // elsewhere neither is written (all cells of 4096 x 4096 took 285 us)
    if (!in && !interior(i - 1, j) && !interior(i + 1, j) && !interior(i, j - 1) && !interior(i, j + 1)) continue;
    for (int c = 0; c < C; ++c) {  // a thread's channels are adjacent in the interleaved inputs
      const double av = (double)f.anchor[q * C + c];
      u0[c * N + k] = av;
      double bv = 0.0;
      if (in) {
        // poisson.rs:364-373: L, R, U, D, then fma(4, -centre, sum)
        const float *gd = f.guid;
        const double ctr = (double)gd[q * C + c];
        const double s = (double)gd[(q - 1) * C + c] + (double)gd[(q + 1) * C + c] + (double)gd[(q - W) * C + c] +
                         (double)gd[(q + W) * C + c];
        bv = fma(4.0, -ctr, s);
      }
      if (in) b0[c * N + k] = fma(g.lambda, -av, bv);
      if (w0) w0[c * N + k] = (in && f.guess) ? (double)f.guess[q * C + c] : av;
    }
  }
}

// ---- multigrid -----------------------------------------------------------------
// A coarse cell is active when at least kCoarseRule of its 2 x 2 children
// are. A cell made mostly of boundary would carry a correction the fine grid
// cannot use; on a CPU model of this preconditioner, requiring 3 children took
// the CG iterations to 1e-6 from 14 to 7 on eight polygons, 10 to 7 on an
// ellipse and 50 to 9 on a mask with 30% of its pixels missing at random.
constexpr int kCoarseRule = 3;

// Relaxation of the smoother's half-sweeps (symmetric SOR: the post-smoothing
// sweeps run the colours in reverse, so the V-cycle stays symmetric). The CPU
// model gave 6 CG iterations for 1.2-1.4 where plain Gauss-Seidel took 7 on
// the same four masks; the coarsest level keeps plain Gauss-Seidel.
constexpr float kSmoothOmega = 1.25f;

// Coarse interior flags from the fine ones; tiles of the coarse plane (the
// fine plane is the entry's second).
__global__ void __launch_bounds__(kTx * kTy) k_mg_coarsen(const Geo *__restrict__ geo,
                                                          const int4 *__restrict__ bmap, const Geo one,
                                                          const uint8_t *__restrict__ af, uint8_t *__restrict__ ac,
                                                          uint8_t *__restrict__ flags) {
  const int4 bt = entry_of(bmap, one);
  const Geo g = bmap ? geo[bt.x] : one;
  const int Hc = g.H, Wf = g.W2, Hf = g.H2, b = tile_b(g), I = (b % g.gx) * kTx + threadIdx.x;
  const uint8_t *f = af + g.o2;
  uint8_t *cc = ac + g.o;
  for (int J = (b / g.gx) * kTy + threadIdx.y; J < Hc && I < g.P; J += g.gy * kTy) {  // (padding: 0)
    int n = 0;
    for (int dy = 0; dy < 2; ++dy)
      for (int dx = 0; dx < 2; ++dx) {
        const int i = 2 * I + dx, j = 2 * J + dy;
        if (i < Wf && j < Hf) n += f[(size_t)j * g.P2 + i];
      }
    cc[(size_t)J * g.P + I] = n >= kCoarseRule ? 1 : 0;
    if (n >= kCoarseRule) set_flag(g, flags, I, J);
  }
}

// ---- strips --------------------------------------------------------------------
// The level and vector kernels give each warp a strip: 128 columns of which it
// owns 112 (the first and last strips of a row more: there is no halo outside
// the image), four a lane, and `rows` rows that it walks downwards, keeping
// the last few rows in registers; horizontal neighbours come by shuffles. One
// pass down a level (k_mg_down) runs four half-sweeps, the residual and its
// restriction as stages on consecutive rows, one pass up (k_mg_up) the
// prolongation and four half-sweeps, so a level's arrays cross the memory
// system once each way instead of once a half-sweep, and no barrier is needed.
// What a strip computes in its halo again, the strips beside it compute alike:
// a cell's value does not depend on the strips.
//
// Rows are padded to a multiple of four cells (pitch P), so that a lane moves
// 16 bytes at once. Strips are skipped by bands of kBand rows without an active
// cell (flags, one byte a band and strip column): their cells are never
// written, and whoever reads them masks them with the interior flags -- or
// reads zero: a level's correction is cleared before the first V-cycle.
//
// Border cells are inactive on every level (a coarse border cell has at most
// two active children), so neighbours outside the image, which the edge lanes
// replace by their own values, are never used.
struct Strip {
  int x0;        // the lane's first column
  int y0, y1;    // rows, trimmed to bands with active cells
  int sx;        // strip column
  bool in, own;  // the lane's columns are inside the pitch; owned
};

// The warp's strip; false if there is none or no active cell in it.
__device__ __forceinline__ bool strip_of(const Geo &g, const uint8_t *__restrict__ flags, Strip &t) {
  const int lane = threadIdx.x & 31, s = tile_b(g) * kStripWarps + (threadIdx.x >> 5);
  t.sx = s % g.gx;
  const int sy = s / g.gx, b0 = sy * (g.rows / kBand), nb = (g.H + kBand - 1) / kBand;
  if (sy >= g.gy) return false;
  const int b = b0 + lane;  // (rows / kBand <= 32)
  const bool f = lane < g.rows / kBand && b < nb && flags[g.f + (long long)b * g.gx + t.sx];
  const unsigned m = __ballot_sync(0xffffffffu, f);
  if (!m) return false;
  t.y0 = (b0 + __ffs(m) - 1) * kBand;
  t.y1 = min(g.H, (b0 + 32 - __clz(m)) * kBand);
  t.x0 = kStripStep * t.sx + 4 * lane;
  t.in = t.x0 < g.P;
  const int lo = t.sx ? kStripStep * t.sx + kStripHalo : 0;
  const int hi = t.sx + 1 == g.gx ? g.P : kStripStep * (t.sx + 1) + kStripHalo;
  t.own = t.x0 >= lo && t.x0 < hi;
  return true;
}

__device__ __forceinline__ unsigned nibble(uint32_t c) {  // four flag bytes -> four bits
  return (c & 1u) | ((c >> 7) & 2u) | ((c >> 14) & 4u) | ((c >> 21) & 8u);
}

// A lane's four cells of a row
struct Row {
  float v[4];
};
__device__ __forceinline__ Row row0() { return Row{{0.f, 0.f, 0.f, 0.f}}; }
__device__ __forceinline__ Row ld_row(const float *p) {
  const float4 q = *reinterpret_cast<const float4 *>(p);
  return Row{{q.x, q.y, q.z, q.w}};
}
__device__ __forceinline__ void st_row(float *p, const Row &r) {
  *reinterpret_cast<float4 *>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
}
__device__ __forceinline__ float from_left(float x) { return __shfl_up_sync(0xffffffffu, x, 1); }
__device__ __forceinline__ float from_right(float x) { return __shfl_down_sync(0xffffffffu, x, 1); }

// Rows on their way: each lane's 16 bytes (and its four flags) of the next
// kRing - 1 rows, copied asynchronously into a ring in shared memory that only
// the lane itself reads. With two rows held ahead in registers instead, a third
// of the passes' time went by waiting for loads.
constexpr int kRing = 6;
struct RowRing {
  float4 v[kRing][32];
};
struct FlagRing {
  uint32_t v[kRing][32];
};
__device__ __forceinline__ void ring_put(void *dst, const void *src, int bytes, bool in) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (bytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(in ? 16 : 0) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(in ? 4 : 0) : "memory");
}
__device__ __forceinline__ void ring_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void ring_wait() {  // all but the newest kRing - 2 rows have arrived
  asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 2) : "memory");
}
__device__ __forceinline__ void ring_drain() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ Row ring_row(const RowRing &q, int k) {
  const float4 x = q.v[k][threadIdx.x & 31];
  return Row{{x.x, x.y, x.z, x.w}};
}

// v / d. With POW2 d is a power of two (lambda 0) and the product with its
// reciprocal is the quotient, bit for bit.
template <bool POW2>
__device__ __forceinline__ float over(float v, float d, float inv) {
  return POW2 ? v * inv : divided(v, d, inv);
}

// Red-black SOR on A_k e = rhs at cells F, F + 2 of the row: gs = (rhs + s *
// sum of neighbours) / d, e += kSmoothOmega (gs - e), at active cells (inactive
// cells hold 0).
template <bool POW2, int F>
__device__ __forceinline__ void relax_row(Row &e, const Row &up, const Row &dn, const Row &r, unsigned a, float s,
                                          float d, float inv) {
  float l0, r0, l1, r1;
  if (F == 0) {
    l0 = from_left(e.v[3]); r0 = e.v[1]; l1 = e.v[1]; r1 = e.v[3];
  } else {
    l0 = e.v[0]; r0 = e.v[2]; l1 = e.v[2]; r1 = from_right(e.v[0]);
  }
  const float n0 = ((l0 + r0) + up.v[F]) + dn.v[F], n1 = ((l1 + r1) + up.v[F + 2]) + dn.v[F + 2];
  const float g0 = over<POW2>(r.v[F] + s * n0, d, inv), g1 = over<POW2>(r.v[F + 2] + s * n1, d, inv);
  if (a & (1u << F)) e.v[F] = e.v[F] + kSmoothOmega * (g0 - e.v[F]);
  if (a & (4u << F)) e.v[F + 2] = e.v[F + 2] + kSmoothOmega * (g1 - e.v[F + 2]);
}

// The per-band partial sums (part[start ..], the same places for every kernel:
// a band without active cells is never written and stays 0), the blocks that
// have finished (cleared again by the last), and the CG scalars.
struct Sums {
  double *part;
  unsigned *done;
  double *sc;
};

// A band's sum: lanes by an xor butterfly.
__device__ __forceinline__ void band_sum(const Geo &g, const Strip &t, int c, int lane, int j, double v,
                                         double *__restrict__ part) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) {
    const int nb = (g.H + kBand - 1) / kBand;
    part[g.part0 + ((long long)c * nb + j / kBand) * g.gx + t.sx] = v;
  }
}

// By every thread of a strip block: true in one thread of the last block of the
// unit to finish, with the unit's sum, its partials taken in a fixed order
// (thread t takes t, t + 128, ..., then a tree).
__device__ __forceinline__ bool unit_sum(const Geo &g, int c, const Sums &s, double *out) {
  constexpr int T = kStripWarps * 32;
  __shared__ bool last;
  __shared__ double sh[T];
  const int tid = threadIdx.x;
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    const unsigned blocks = (unsigned)((g.gx * g.gy + kStripWarps - 1) / kStripWarps);
    last = atomicAdd(s.done + g.unit0 + c, 1u) == blocks - 1u;
    __threadfence();
  }
  __syncthreads();
  if (!last) return false;
  const long long n = (long long)((g.H + kBand - 1) / kBand) * g.gx, p0 = g.part0 + c * n;
  double acc = 0.0;
  for (long long k = tid; k < n; k += T) acc += __ldcg(s.part + p0 + k);
  sh[tid] = acc;
  __syncthreads();
  for (int o = T / 2; o > 0; o >>= 1) {
    if (tid < o) sh[tid] += sh[tid + o];
    __syncthreads();
  }
  if (tid != 0) return false;
  s.done[g.unit0 + c] = 0;
  *out = sh[0];
  return true;
}

__device__ __forceinline__ void new_rho(double *sc, double rho, int first) {
  sc[S_BETA] = first || sc[S_RHO] == 0.0 ? 0.0 : rho / sc[S_RHO];
  sc[S_RHO] = rho;
}

// ---- the FP64 residual and update ------------------------------------------------
// r = fma(lambda + 4, -u, nsum) - b' at interior cells (0 elsewhere); ||r||^2.
struct Row64 {
  double v[4];
};
__device__ __forceinline__ Row64 ld_row64(const double *p) {
  const double2 a = *reinterpret_cast<const double2 *>(p), b = *reinterpret_cast<const double2 *>(p + 2);
  return Row64{{a.x, a.y, b.x, b.y}};
}
__device__ __forceinline__ void st_row64(double *p, const Row64 &r) {
  *reinterpret_cast<double2 *>(p) = make_double2(r.v[0], r.v[1]);
  *reinterpret_cast<double2 *>(p + 2) = make_double2(r.v[2], r.v[3]);
}
__global__ void __launch_bounds__(kStripWarps * 32) k_mg_residual64(const Geo *__restrict__ geo,
                                                                    const int4 *__restrict__ bmap, const Geo one,
                                                                    const uint8_t *__restrict__ flags,
                                                                    const uint8_t *__restrict__ act,
                                                                    const double *__restrict__ u,
                                                                    const double *__restrict__ bl,
                                                                    double *__restrict__ r64, Sums sums,
                                                                    double *__restrict__ rr) {
  const int4 bt = entry_of(bmap, one);
  const int c = blockIdx.z, lane = threadIdx.x & 31;
  if (c >= bt.z) return;
  const Geo g = bmap ? geo[bt.x] : one;
  Strip t;
  if (strip_of(g, flags, t)) {
    const long long at = g.oc + (long long)c * g.P * g.H + t.x0;
    const double lambda = g.lambda;
    auto fetch = [&](int y) { return t.in && y >= 0 && y < g.H ? ld_row64(u + at + (long long)y * g.P) : Row64{}; };
    Row64 m = fetch(t.y0 - 1), k = fetch(t.y0), n = fetch(t.y0 + 1);
    double acc = 0.0;
    for (int j = t.y0; j < t.y1; ++j) {
      const Row64 next = fetch(j + 2);
      const double l = __shfl_up_sync(0xffffffffu, k.v[3], 1), r = __shfl_down_sync(0xffffffffu, k.v[0], 1);
      if (t.own) {
        const unsigned a = nibble(*reinterpret_cast<const uint32_t *>(act + g.o + (long long)j * g.P + t.x0));
        const Row64 b = ld_row64(bl + at + (long long)j * g.P);
        Row64 res;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          // L, R, U, D (poisson.rs:275-298)
          const double nsum = (((i ? k.v[i ? i - 1 : 0] : l) + (i < 3 ? k.v[i < 3 ? i + 1 : 3] : r)) + m.v[i]) + n.v[i];
          res.v[i] = a & (1u << i) ? fma(lambda + 4.0, -k.v[i], nsum) - b.v[i] : 0.0;
          acc += res.v[i] * res.v[i];
        }
        st_row64(r64 + at + (long long)j * g.P, res);
      }
      if ((j & (kBand - 1)) == kBand - 1 || j == t.y1 - 1) {
        band_sum(g, t, c, lane, j, acc, sums.part);
        acc = 0.0;
      }
      m = k;
      k = n;
      n = next;
    }
  }
  double v;
  if (unit_sum(g, c, sums, &v)) rr[g.unit0 + c] = v;
}

// r32 = r64 / scale[unit], x = 0; a unit that is not being corrected (scale 0) is left
__global__ void __launch_bounds__(kStripWarps * 32) k_mg_scale(const Geo *__restrict__ geo,
                                                               const int4 *__restrict__ bmap, const Geo one,
                                                               const uint8_t *__restrict__ flags,
                                                               const double *__restrict__ r64,
                                                               const double *__restrict__ scale, float *__restrict__ r32,
                                                               float *__restrict__ x) {
  const int4 bt = entry_of(bmap, one);
  const int c = blockIdx.z;
  if (c >= bt.z) return;
  const Geo g = bmap ? geo[bt.x] : one;
  const double s = scale[g.unit0 + c];
  if (!(s > 0.0)) return;
  Strip t;
  if (!strip_of(g, flags, t) || !t.own) return;
  const long long at = g.oc + (long long)c * g.P * g.H + t.x0;
#pragma unroll 4
  for (int j = t.y0; j < t.y1; ++j) {
    const long long o = at + (long long)j * g.P;
    const Row64 r = ld_row64(r64 + o);
    Row v;
#pragma unroll
    for (int i = 0; i < 4; ++i) v.v[i] = (float)(r.v[i] / s);
    st_row(r32 + o, v);
    st_row(x + o, row0());
  }
}

// u += scale[unit] * x at interior cells; a unit with scale 0 (not being
// corrected) is left as it is, bit for bit. x null: 0.
__global__ void __launch_bounds__(kStripWarps * 32) k_mg_update(const Geo *__restrict__ geo,
                                                                const int4 *__restrict__ bmap, const Geo one,
                                                                const uint8_t *__restrict__ flags,
                                                                const uint8_t *__restrict__ act,
                                                                const float *__restrict__ x,
                                                                const double *__restrict__ scale,
                                                                double *__restrict__ u) {
  const int4 bt = entry_of(bmap, one);
  const int c = blockIdx.z;
  if (c >= bt.z) return;
  const Geo g = bmap ? geo[bt.x] : one;
  const double s = scale[g.unit0 + c];
  if (s == 0.0) return;
  Strip t;
  if (!strip_of(g, flags, t) || !t.own) return;
  const long long at = g.oc + (long long)c * g.P * g.H + t.x0;
#pragma unroll 4
  for (int j = t.y0; j < t.y1; ++j) {
    const long long o = at + (long long)j * g.P;
    const unsigned a = nibble(*reinterpret_cast<const uint32_t *>(act + g.o + (long long)j * g.P + t.x0));
    const Row v = x ? ld_row(x + o) : row0();
    Row64 w = ld_row64(u + o);
#pragma unroll
    for (int i = 0; i < 4; ++i) w.v[i] = a & (1u << i) ? fma(s, (double)v.v[i], w.v[i]) : w.v[i];
    st_row64(u + o, w);
  }
}

// ---- the V-cycle -----------------------------------------------------------------
// The products' roundings, spelled out: the residual and the prolongation are
// the same bit for bit wherever they are evaluated.
__device__ __forceinline__ float level_residual(float rhs, float d, float e, float s, float nb) {
  return rhs - fmaf(d, e, -(s * nb));
}
// row + weight * x of a restriction's row sum, two roundings
__device__ __forceinline__ float add_weighted(float row, float weight, float x) {
  return __fadd_rn(row, __fmul_rn(weight, x));
}
// e(I0, J0), e(I1, J0), e(I0, J1), e(I1, J1): weights 9, 3, 3, 1 sixteenths
__device__ __forceinline__ float bilinear(float a, float b, float c, float d) {
  return fmaf(0.0625f, d, fmaf(0.1875f, b + c, 0.5625f * a));
}

// V-cycle kernels return at once for a unit whose run flag is 0.
//
// Down one level: from e = 0 the half-sweeps red, black, red, black, then the
// restriction of the residual, rhs_c(I, J) = sum over fine (2I + a, 2J + b), a,
// b in -1..2, of wx wy res / 4 (weights 1/4, 3/4, 3/4, 1/4; res = rhs - A e at
// active cells, 0 elsewhere). Row y comes in as rows y - 1, y - 2, y - 3 get
// their later half-sweeps, row y - 4 its residual.
template <bool POW2>
__device__ __forceinline__ void mg_down(const Geo &g, const Strip &t, int c, const uint8_t *__restrict__ act,
                                        const float *__restrict__ rhs, float *__restrict__ e,
                                        const uint8_t *__restrict__ actc, float *__restrict__ rhsc, RowRing &rr,
                                        FlagRing &ra) {
  const long long N = (long long)g.P * g.H, Nc = (long long)g.P2 * g.H2;
  const uint8_t *a0 = act + g.o + t.x0;
  const float *r0 = rhs + g.oc + c * N + t.x0;
  float *e0 = e + g.oc + c * N + t.x0;
  const int I = t.x0 >> 1;
  const uint8_t *ca = actc + g.o2 + I;
  float *rc = rhsc + g.oc2 + c * Nc + I;
  const float s = g.s, d = g.d, inv = 1.0f / d;
  const int J0 = t.y0 >> 1, J1 = (t.y1 + 1) >> 1, last = 2 * J1 + 4;
  Row E[6], R[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) E[k] = R[k] = row0();
  unsigned a = 0;  // active bits, the newest row's lowest
  float vp0 = 0.f, vp1 = 0.f, vn0 = 0.f, vn1 = 0.f;
  const int y0 = t.y0 - 6, lane = threadIdx.x & 31;  // (rows after `last` are walked in vain)
  auto fetch = [&](int y, int k) {
    const bool in = t.in && y >= 0 && y < g.H;
    const long long o = in ? (long long)y * g.P : -(long long)t.x0;  // (the plane's first cell: not read)
    ring_put(&rr.v[k][lane], r0 + o, 16, in);
    ring_put(&ra.v[k][lane], a0 + o, 4, in);
    ring_commit();
  };
#pragma unroll
  for (int k = 0; k < kRing - 1; ++k) fetch(y0 + k, k);
  for (int yb = y0; yb <= last; yb += 6) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int y = yb + k;
      constexpr auto at = [](int k, int i) { return (k + 6 - i) % 6; };
      const int par = k & 1;  // y0 is even
      ring_wait();
      R[k] = ring_row(rr, k);
      a = (a << 4) | nibble(ra.v[k][lane]);
      fetch(y + kRing - 1, at(k, 1));
      Row &E0 = E[k], &E1 = E[at(k, 1)], &E2 = E[at(k, 2)], &E3 = E[at(k, 3)], &E4 = E[at(k, 4)], &E5 = E[at(k, 5)];
      // red of row y from e = 0; black 0
#pragma unroll
      for (int i = 0; i < 4; ++i)
        E0.v[i] = ((i + par) & 1) == 0 && (a & (1u << i)) ? kSmoothOmega * over<POW2>(R[k].v[i], d, inv) : 0.0f;
      if (par == 0) {  // rows y - 1 and y - 3 are odd, row y - 2 is even
        relax_row<POW2, 0>(E1, E2, E0, R[at(k, 1)], a >> 4, s, d, inv);
        relax_row<POW2, 0>(E2, E3, E1, R[at(k, 2)], a >> 8, s, d, inv);
        relax_row<POW2, 0>(E3, E4, E2, R[at(k, 3)], a >> 12, s, d, inv);
      } else {
        relax_row<POW2, 1>(E1, E2, E0, R[at(k, 1)], a >> 4, s, d, inv);
        relax_row<POW2, 1>(E2, E3, E1, R[at(k, 2)], a >> 8, s, d, inv);
        relax_row<POW2, 1>(E3, E4, E2, R[at(k, 3)], a >> 12, s, d, inv);
      }
      if (t.own && y - 3 >= t.y0 && y - 3 < t.y1) st_row(e0 + (long long)(y - 3) * g.P, E3);
      // residual of row j = y - 4
      const int j = y - 4;
      const float el = from_left(E4.v[3]), er = from_right(E4.v[0]);
      float res[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float l = i ? E4.v[i ? i - 1 : 0] : el, r = i < 3 ? E4.v[i < 3 ? i + 1 : 3] : er;
        const float nb = ((l + r) + E5.v[i]) + E3.v[i];
        const float v = level_residual(R[at(k, 4)].v[i], d, E4.v[i], s, nb);
        res[i] = (a >> 16) & (1u << i) ? v : 0.0f;
      }
      const float rl = from_left(res[3]), rr = from_right(res[0]);
      float w0 = 0.25f * rl, w1 = 0.25f * res[1];
      w0 = add_weighted(w0, 0.75f, res[0]); w1 = add_weighted(w1, 0.75f, res[2]);
      w0 = add_weighted(w0, 0.75f, res[1]); w1 = add_weighted(w1, 0.75f, res[3]);
      w0 = add_weighted(w0, 0.25f, res[2]); w1 = add_weighted(w1, 0.25f, rr);
      if (par) {  // j = 2 J - 1
        vp0 = fmaf(0.75f, w0, vp0); vp1 = fmaf(0.75f, w1, vp1);
        vn0 = 0.25f * w0; vn1 = 0.25f * w1;
      } else {    // j = 2 J: coarse row J - 1 is complete
        vn0 = fmaf(0.75f, w0, vn0); vn1 = fmaf(0.75f, w1, vn1);
        vp0 = fmaf(0.25f, w0, vp0); vp1 = fmaf(0.25f, w1, vp1);
        const int J = (j >> 1) - 1;
        if (t.own && I < g.P2 && J >= J0 && J < J1) {
          const uchar2 q = *reinterpret_cast<const uchar2 *>(ca + (long long)J * g.P2);
          *reinterpret_cast<float2 *>(rc + (long long)J * g.P2) = make_float2(q.x ? vp0 * 0.25f : 0.0f, q.y ? vp1 * 0.25f : 0.0f);
        }
        vp0 = vn0; vp1 = vn1;
      }
    }
  }
  ring_drain();
}

__global__ void __launch_bounds__(kStripWarps * 32, 4) k_mg_down(const Geo *__restrict__ geo,
                                                                 const int4 *__restrict__ bmap, const Geo one,
                                                                 const uint8_t *__restrict__ flags,
                                                                 const uint8_t *__restrict__ act,
                                                                 const float *__restrict__ rhs, float *__restrict__ e,
                                                                 const uint8_t *__restrict__ actc,
                                                                 float *__restrict__ rhsc,
                                                                 const double *__restrict__ run) {
  const int4 bt = entry_of(bmap, one);
  const int c = blockIdx.z;
  if (c >= bt.z || run[bt.y + c] == 0.0) return;
  const Geo g = bmap ? geo[bt.x] : one;
  __shared__ RowRing rr[kStripWarps];
  __shared__ FlagRing ra[kStripWarps];
  const int w = threadIdx.x >> 5;
  Strip t;
  if (!strip_of(g, flags, t)) return;
  if (g.lambda == 0.0) mg_down<true>(g, t, c, act, rhs, e, actc, rhsc, rr[w], ra[w]);
  else mg_down<false>(g, t, c, act, rhs, e, actc, rhsc, rr[w], ra[w]);
}

// Up one level: e += the bilinear prolongation of the coarse correction at
// active cells, then the half-sweeps black, red, black, red; the result goes
// to another array (the strips beside read e). DOT: also the partial sums of
// rhs . result, one a band and strip column.
template <bool POW2, bool DOT>
__device__ __forceinline__ void mg_up(const Geo &g, const Strip &t, int c, const uint8_t *__restrict__ act,
                                      const float *__restrict__ rhs, const float *__restrict__ e,
                                      const float *__restrict__ ec, float *__restrict__ out,
                                      double *__restrict__ part, RowRing &re, RowRing &rr, FlagRing &ra) {
  const int lane = threadIdx.x & 31;
  const long long N = (long long)g.P * g.H, Nc = (long long)g.P2 * g.H2;
  const uint8_t *a0 = act + g.o + t.x0;
  const float *r0 = rhs + g.oc + c * N + t.x0, *e0 = e + g.oc + c * N + t.x0;
  float *o0 = out + g.oc + c * N + t.x0;
  const int I = t.x0 >> 1;
  const float *c0 = ec + g.oc2 + c * Nc + I;
  const float s = g.s, d = g.d, inv = 1.0f / d;
  const int last = t.y1 + 3;
  Row E[6], R[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) E[k] = R[k] = row0();
  unsigned a = 0;
  double acc = 0.0;
  const int y0 = t.y0 - 4;
  auto fetch = [&](int y, int k) {
    const bool in = t.in && y >= 0 && y < g.H;
    const long long o = in ? (long long)y * g.P : -(long long)t.x0;  // (the plane's first cell: not read)
    ring_put(&re.v[k][lane], e0 + o, 16, in);
    ring_put(&rr.v[k][lane], r0 + o, 16, in);
    ring_put(&ra.v[k][lane], a0 + o, 4, in);
    ring_commit();
  };
  auto fetch_c = [&](int J) {
    return I < g.P2 && J >= 0 && J < g.H2 ? *reinterpret_cast<const float2 *>(c0 + (long long)J * g.P2) : make_float2(0.f, 0.f);
  };
  // four coarse values a row around the lane's four cells: columns I - 1 .. I + 2
  auto wide = [&](float2 v) { return Row{{from_left(v.y), v.x, v.y, from_right(v.x)}}; };
#pragma unroll
  for (int k = 0; k < kRing - 1; ++k) fetch(y0 + k, k);
  // coarse rows J - 1, J (J = y / 2), and J + 1, J + 2 on their way
  Row cm = wide(fetch_c((y0 >> 1) - 1)), cj = wide(fetch_c(y0 >> 1));
  float2 cn = fetch_c((y0 >> 1) + 1), cnn = fetch_c((y0 >> 1) + 2);
  for (int yb = y0; yb <= last; yb += 6) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int y = yb + k;
      constexpr auto at = [](int k, int i) { return (k + 6 - i) % 6; };
      const int par = k & 1;  // y0 is even
      Row &E0 = E[k], &E1 = E[at(k, 1)], &E2 = E[at(k, 2)], &E3 = E[at(k, 3)], &E4 = E[at(k, 4)], &E5 = E[at(k, 5)];
      ring_wait();
      R[k] = ring_row(rr, k);
      const Row pe = ring_row(re, k);
      a = (a << 4) | nibble(ra.v[k][lane]);
      fetch(y + kRing - 1, at(k, 1));
      Row near;
      if (par == 0) {
        near = cm;
      } else {
        near = wide(cn);
        cm = cj;
        // (cj moves on after this row)
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        // columns: I0 = i / 2 (index 1 + i / 2), I1 beside it
        const int m0 = 1 + (i >> 1), m1 = (i & 1) ? m0 + 1 : m0 - 1;
        const Row &rj = par == 0 ? cj : cm;  // row J (cm holds it after the move)
        const float v = bilinear(rj.v[m0], rj.v[m1], near.v[m0], near.v[m1]);
        E0.v[i] = a & (1u << i) ? pe.v[i] + v : 0.0f;
      }
      if (par) {
        cj = near;
        cn = cnn;
        cnn = fetch_c(((y + 1) >> 1) + 2);
      }
      if (par == 0) {  // rows y - 1 and y - 3 are odd: black cells 0, 2; rows y - 2, y - 4 even: red 0, 2
        relax_row<POW2, 0>(E1, E2, E0, R[at(k, 1)], a >> 4, s, d, inv);
        relax_row<POW2, 0>(E2, E3, E1, R[at(k, 2)], a >> 8, s, d, inv);
        relax_row<POW2, 0>(E3, E4, E2, R[at(k, 3)], a >> 12, s, d, inv);
        relax_row<POW2, 0>(E4, E5, E3, R[at(k, 4)], a >> 16, s, d, inv);
      } else {
        relax_row<POW2, 1>(E1, E2, E0, R[at(k, 1)], a >> 4, s, d, inv);
        relax_row<POW2, 1>(E2, E3, E1, R[at(k, 2)], a >> 8, s, d, inv);
        relax_row<POW2, 1>(E3, E4, E2, R[at(k, 3)], a >> 12, s, d, inv);
        relax_row<POW2, 1>(E4, E5, E3, R[at(k, 4)], a >> 16, s, d, inv);
      }
      const int j = y - 4;
      if (j >= t.y0 && j < t.y1) {
        if (t.own) {
          st_row(o0 + (long long)j * g.P, E4);
          if (DOT) {
#pragma unroll
            for (int i = 0; i < 4; ++i) acc = fma((double)R[at(k, 4)].v[i], (double)E4.v[i], acc);
          }
        }
        if (DOT && ((j & (kBand - 1)) == kBand - 1 || j == t.y1 - 1)) {
          band_sum(g, t, c, lane, j, acc, part);
          acc = 0.0;
        }
      }
    }
  }
  ring_drain();
}

template <bool DOT>
__global__ void __launch_bounds__(kStripWarps * 32, 4) k_mg_up(const Geo *__restrict__ geo,
                                                               const int4 *__restrict__ bmap, const Geo one,
                                                               const uint8_t *__restrict__ flags,
                                                               const uint8_t *__restrict__ act,
                                                               const float *__restrict__ rhs,
                                                               const float *__restrict__ e,
                                                               const float *__restrict__ ec, float *__restrict__ out,
                                                               const double *__restrict__ run, Sums sums, int first) {
  const int4 bt = entry_of(bmap, one);
  const int c = blockIdx.z;
  if (c >= bt.z || run[bt.y + c] == 0.0) return;
  const Geo g = bmap ? geo[bt.x] : one;
  __shared__ RowRing re[kStripWarps], rr[kStripWarps];
  __shared__ FlagRing ra[kStripWarps];
  const int w = threadIdx.x >> 5;
  Strip t;
  if (strip_of(g, flags, t)) {
    if (g.lambda == 0.0) mg_up<true, DOT>(g, t, c, act, rhs, e, ec, out, sums.part, re[w], rr[w], ra[w]);
    else mg_up<false, DOT>(g, t, c, act, rhs, e, ec, out, sums.part, re[w], rr[w], ra[w]);
  }
  if (!DOT) return;
  double rho;
  if (unit_sum(g, c, sums, &rho)) new_rho(sums.sc + (long long)(g.unit0 + c) * S_N, rho, first);
}

// The levels of at most kTailCells cells, in one block's shared memory: the
// V-cycle from level k0 of an instance down to its coarsest and up again; one
// block per instance (blockIdx.x) and channel (blockIdx.z). The coarsest level
// (at most kCoarseMax cells) takes kCoarseSweeps plain red-black Gauss-Seidel
// sweeps and as many in reverse colour order. Bound by the latency of its
// phases, a barrier each, and beyond a few thousand cells by one SM's shared
// memory: a level of 119 x 91 cells cost 20 us more here than its two strip
// launches, one of 60 x 46 about 10 us less (per pass over 237 x 181: 849 us
// a solve with 12288 cells in the tail, 797 with 4096, 816 with 1100).
constexpr int kCoarseMax = 64, kTailCells = 4096, kTailLevels = 10, kCoarseSweeps = 24;
constexpr int kTailX = 32, kTailY = 32;
struct alignas(16) Tail {
  int C, unit0, n;                   // channels, first unit, levels (from k0 to the coarsest)
  int pow2;                          // lambda is 0: every level's d is a power of two (over)
  int w[kTailLevels], h[kTailLevels], P[kTailLevels];
  long long o[kTailLevels];          // the planes' first cells in the levels' flags
  const uint8_t *act[kTailLevels];   // the levels' flags
  const float *rhs;                  // level k0, C planes of P[0] * h[0]
  float *e;
  float s[kTailLevels], d[kTailLevels];
};
// Shared memory: e, rhs and flags of every level; the first level's residual.
constexpr int kTailSmem = 224 * 1024;
size_t tail_bytes(size_t all, size_t first) { return all * 9 + 16 + first * 4; }

__global__ void __launch_bounds__(kTailX * kTailY, 1) k_mg_tail(const Tail *__restrict__ tails,
                                                                const double *__restrict__ run) {
  extern __shared__ __align__(16) float tsm[];
  __shared__ Tail T;
  __shared__ int off[kTailLevels + 1], table[kCoarseMax];
  const int c = blockIdx.z, tx = threadIdx.x, ty = threadIdx.y, tid = ty * kTailX + tx;
  for (int k = tid; k < (int)(sizeof(Tail) / 4); k += kTailX * kTailY)
    reinterpret_cast<int *>(&T)[k] = reinterpret_cast<const int *>(tails + blockIdx.x)[k];
  __syncthreads();
  if (c >= T.C || run[T.unit0 + c] == 0.0) return;
  if (tid < kCoarseMax) table[tid] = -1;
  if (tid == 0) {
    off[0] = 0;
    for (int l = 0; l < T.n; ++l) off[l + 1] = off[l] + T.w[l] * T.h[l];
  }
  __syncthreads();
  const int all = off[T.n];
  float *E = tsm, *R = tsm + all;
  float *X = R + all;  // the residual of the level on the way down
  uint8_t *A = reinterpret_cast<uint8_t *>(X + T.w[0] * T.h[0]);
  {
    const float *r = T.rhs + (long long)c * T.P[0] * T.h[0];
    const int w = T.w[0];
#pragma unroll 4
    for (int j = ty; j < T.h[0]; j += kTailY)
      for (int i = tx; i < w; i += kTailX) R[j * w + i] = r[(long long)j * T.P[0] + i];
  }
  for (int l = 0; l < T.n; ++l) {
    const uint8_t *f = T.act[l] + T.o[l];
    const int w = T.w[l];
#pragma unroll 4
    for (int j = ty; j < T.h[l]; j += kTailY)
      for (int i = tx; i < w; i += kTailX) A[off[l] + j * w + i] = f[(long long)j * T.P[l] + i];
  }
  __syncthreads();
  const bool pow2 = T.pow2;
  auto quotient = [&](float v, float d, float inv) { return pow2 ? v * inv : divided(v, d, inv); };
  // one colour of level l (kSmoothOmega); two rows at once, loads first: the
  // neighbours are of the other colour
  auto half = [&](int l, int color) {
    const int w = T.w[l], h = T.h[l];
    const float s = T.s[l], d = T.d[l], inv = 1.0f / d;
    float *e = E + off[l];
    const float *r = R + off[l];
    const uint8_t *a = A + off[l];
    // (kTailY is even: a thread's rows have one parity)
    for (int i = 2 * tx + ((ty + color) & 1); i < w; i += 2 * kTailX)
      for (int j = ty, q = ty * w + i; j < h; j += 2 * kTailY, q += 2 * kTailY * w) {
        const int q1 = q + kTailY * w;
        const bool on0 = a[q], on1 = j + kTailY < h && a[q1];  // (an active cell is never on the border)
        float n0, n1, r0, r1, e0, e1;
        if (on0) {
          n0 = ((e[q - 1] + e[q + 1]) + e[q - w]) + e[q + w];
          r0 = r[q];
          e0 = e[q];
        }
        if (on1) {
          n1 = ((e[q1 - 1] + e[q1 + 1]) + e[q1 - w]) + e[q1 + w];
          r1 = r[q1];
          e1 = e[q1];
        }
        if (on0) e[q] = e0 + kSmoothOmega * (quotient(r0 + s * n0, d, inv) - e0);
        if (on1) e[q1] = e1 + kSmoothOmega * (quotient(r1 + s * n1, d, inv) - e1);
      }
    __syncthreads();
  };
  for (int l = 0; l + 1 < T.n; ++l) {
    const int w = T.w[l], h = T.h[l], W = T.w[l + 1], H = T.h[l + 1];
    const float s = T.s[l], d = T.d[l], inv = 1.0f / d;
    float *e = E + off[l];
    const float *r = R + off[l];
    const uint8_t *a = A + off[l];
    for (int i = tx; i < w; i += kTailX)
#pragma unroll 2
      for (int j = ty, q = ty * w + i; j < h; j += kTailY, q += kTailY * w)
        e[q] = a[q] && ((i + ty) & 1) == 0 ? kSmoothOmega * quotient(r[q], d, inv) : 0.0f;
    __syncthreads();
    half(l, 1);
    half(l, 0);
    half(l, 1);
    for (int i = tx; i < w; i += kTailX)
#pragma unroll 2
      for (int j = ty, q = ty * w + i; j < h; j += kTailY, q += kTailY * w) {
        X[q] = a[q] ? level_residual(r[q], d, e[q], s, ((e[q - 1] + e[q + 1]) + e[q - w]) + e[q + w]) : 0.0f;
      }
    __syncthreads();
    for (int J = ty; J < H; J += kTailY)
      for (int I = tx; I < W; I += kTailX) {
        float v = 0.0f;
        if (A[off[l + 1] + J * W + I]) {  // (not on the border: all its 4 x 4 fine cells exist)
#pragma unroll
          for (int b = -1; b <= 2; ++b) {
            const float *x = X + (2 * J + b) * w + 2 * I;
            float row = 0.0f;
#pragma unroll
            for (int k = -1; k <= 2; ++k) row = add_weighted(row, (k == 0 || k == 1) ? 0.75f : 0.25f, x[k]);
            v = fmaf((b == 0 || b == 1) ? 0.75f : 0.25f, row, v);
          }
          v *= 0.25f;
        }
        R[off[l + 1] + J * W + I] = v;
      }
    __syncthreads();
  }
  // lane of a cell of the coarsest level: the cells of its colour before it, row-major
  auto lane_of = [&](int w, int q) {
    const int j = q / w, i = q - j * w, color = (i + j) & 1;
    const int even = (w + 1 - color) / 2, odd = (w + color) / 2;  // of this colour in even rows, in odd rows
    return ((j + 1) >> 1) * even + (j >> 1) * odd + (i >> 1);
  };
  if (tid < kCoarseMax) {
    const int w = T.w[T.n - 1], n = w * T.h[T.n - 1];
    if (tid < n) table[((tid % w + tid / w) & 1) * 32 + lane_of(w, tid)] = tid;
    asm volatile("bar.sync 1, 64;" ::: "memory");
  }
  if (tid < 32) {
    // the coarsest level: one warp, a red and a black cell a lane (64 cells have
    // 32 of each), neighbours by shuffles from the lanes that hold them
    const int l = T.n - 1, w = T.w[l];
    const float s = T.s[l], d = T.d[l], inv = 1.0f / d;
    float v[2] = {0.0f, 0.0f}, r[2] = {0.0f, 0.0f};
    const int cell[2] = {table[tid], table[32 + tid]};
    int at[2][4];
    bool on[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int q = cell[k];
      on[k] = q >= 0 && A[off[l] + q];  // (never on the border)
      if (on[k]) r[k] = R[off[l] + q];
      at[k][0] = on[k] ? lane_of(w, q - 1) : 0;
      at[k][1] = on[k] ? lane_of(w, q + 1) : 0;
      at[k][2] = on[k] ? lane_of(w, q - w) : 0;
      at[k][3] = on[k] ? lane_of(w, q + w) : 0;
    }
    auto step = [&](int k) {
      const float x0 = __shfl_sync(0xffffffffu, v[1 - k], at[k][0]), x1 = __shfl_sync(0xffffffffu, v[1 - k], at[k][1]);
      const float x2 = __shfl_sync(0xffffffffu, v[1 - k], at[k][2]), x3 = __shfl_sync(0xffffffffu, v[1 - k], at[k][3]);
      const float nb = ((x0 + x1) + x2) + x3;
      if (on[k]) v[k] = quotient(r[k] + s * nb, d, inv);
    };
    for (int k = 0; k < kCoarseSweeps; ++k) {
      step(0);
      step(1);
    }
    for (int k = 0; k < kCoarseSweeps; ++k) {
      step(1);
      step(0);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (cell[k] >= 0) E[off[l] + cell[k]] = v[k];
  }
  __syncthreads();
  for (int l = T.n - 2; l >= 0; --l) {
    const int w = T.w[l], h = T.h[l], W = T.w[l + 1];
    float *e = E + off[l];
    const float *x = E + off[l + 1];
    const uint8_t *a = A + off[l];
    for (int i = tx; i < w; i += kTailX) {
      const int I0 = i >> 1, I1 = (i & 1) ? I0 + 1 : I0 - 1;
#pragma unroll 2
      for (int j = ty, q = ty * w + i; j < h; j += kTailY, q += kTailY * w) {
        if (!a[q]) continue;  // (an active cell's coarse neighbours exist)
        const float *x0 = x + (j >> 1) * W, *x1 = (j & 1) ? x0 + W : x0 - W;
        e[q] += bilinear(x0[I0], x0[I1], x1[I0], x1[I1]);
      }
    }
    __syncthreads();
    half(l, 1);
    half(l, 0);
    half(l, 1);
    half(l, 0);
  }
  float *out = T.e + (long long)c * T.P[0] * T.h[0];
  for (int j = ty; j < T.h[0]; j += kTailY)
    for (int i = tx; i < T.P[0]; i += kTailX) out[(long long)j * T.P[0] + i] = i < T.w[0] ? E[j * T.w[0] + i] : 0.0f;
}

// ---- conjugate gradients (level-0 strips) ---------------------------------------
// rho = r.z of an instance whose finest level is its coarsest (k_mg_up sums the
// others').
__global__ void __launch_bounds__(kStripWarps * 32) k_cg_dot(const Geo *__restrict__ geo,
                                                             const int4 *__restrict__ bmap, const Geo one,
                                                             const uint8_t *__restrict__ flags,
                                                             const float *__restrict__ x, const float *__restrict__ y,
                                                             const double *__restrict__ run, Sums sums, int first) {
  const int4 bt = entry_of(bmap, one);
  const int c = blockIdx.z, lane = threadIdx.x & 31;
  if (c >= bt.z || run[bt.y + c] == 0.0) return;
  const Geo g = bmap ? geo[bt.x] : one;
  Strip t;
  if (strip_of(g, flags, t)) {
    const long long at = g.oc + (long long)c * g.P * g.H + t.x0;
    double acc = 0.0;
    for (int j = t.y0; j < t.y1; ++j) {
      if (t.own) {
        const Row a = ld_row(x + at + (long long)j * g.P), b = ld_row(y + at + (long long)j * g.P);
#pragma unroll
        for (int i = 0; i < 4; ++i) acc = fma((double)a.v[i], (double)b.v[i], acc);
      }
      if ((j & (kBand - 1)) == kBand - 1 || j == t.y1 - 1) {
        band_sum(g, t, c, lane, j, acc, sums.part);
        acc = 0.0;
      }
    }
  }
  double rho;
  if (unit_sum(g, c, sums, &rho)) new_rho(sums.sc + (long long)(g.unit0 + c) * S_N, rho, first);
}

// A_0 p at a row's active cells: d p - (left + right + up + down)
__device__ __forceinline__ Row apply_row(const Row &k, const Row &up, const Row &dn, unsigned a, float d) {
  const float l = from_left(k.v[3]), r = from_right(k.v[0]);
  Row v;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float sum = (((i ? k.v[i ? i - 1 : 0] : l) + (i < 3 ? k.v[i < 3 ? i + 1 : 3] : r)) + up.v[i]) + dn.v[i];
    v.v[i] = a & (1u << i) ? d * k.v[i] - sum : 0.0f;
  }
  return v;
}

// p' = z + beta p (p' = z on the first iteration) and p'.q, q = A_0 p' at active
// cells. The strips beside read p, so p' is another array. q is not stored: the
// step evaluates it again from p', which it reads anyway (8 of 41 bytes a cell
// and iteration saved).
__global__ void __launch_bounds__(kStripWarps * 32) k_cg_apply(const Geo *__restrict__ geo,
                                                               const int4 *__restrict__ bmap, const Geo one,
                                                               const uint8_t *__restrict__ flags,
                                                               const uint8_t *__restrict__ act,
                                                               const float *__restrict__ z, const float *__restrict__ p,
                                                               float *__restrict__ pn,
                                                               const double *__restrict__ run, Sums sums, int first) {
  const int4 bt = entry_of(bmap, one);
  const int c = blockIdx.z, lane = threadIdx.x & 31;
  if (c >= bt.z || run[bt.y + c] == 0.0) return;  // (a stopped unit's p may never have been written)
  const Geo g = bmap ? geo[bt.x] : one;
  double *sc = sums.sc + (long long)(g.unit0 + c) * S_N;
  Strip t;
  if (strip_of(g, flags, t)) {
    const float beta = first ? 0.0f : (float)sc[S_BETA], d = g.d;
    const long long at = g.oc + (long long)c * g.P * g.H + t.x0;
    const uint8_t *a0 = act + g.o + t.x0;
    auto fetch = [&](const float *v, int y) { return t.in && y >= 0 && y < g.H ? ld_row(v + at + (long long)y * g.P) : row0(); };
    auto fetch_a = [&](int y) {
      return t.in && y >= 0 && y < g.H ? *reinterpret_cast<const uint32_t *>(a0 + (long long)y * g.P) : 0u;
    };
    Row m = row0(), k = row0();  // rows y - 2, y - 1 of p'
    unsigned ak = 0;
    double acc = 0.0;
    Row fz = fetch(z, t.y0 - 1), fp = first ? row0() : fetch(p, t.y0 - 1);
    uint32_t fa = fetch_a(t.y0 - 1);
#pragma unroll 3
    for (int y = t.y0 - 1; y <= t.y1; ++y) {
      const unsigned a = nibble(fa);
      Row n;
#pragma unroll
      for (int i = 0; i < 4; ++i) n.v[i] = a & (1u << i) ? (first ? fz.v[i] : fz.v[i] + beta * fp.v[i]) : 0.0f;
      fz = fetch(z, y + 1);
      if (!first) fp = fetch(p, y + 1);
      fa = fetch_a(y + 1);
      if (t.own && y >= t.y0 && y < t.y1) st_row(pn + at + (long long)y * g.P, n);
      const int j = y - 1;
      const Row v = apply_row(k, m, n, ak, d);
      if (j >= t.y0) {
        if (t.own) {
#pragma unroll
          for (int i = 0; i < 4; ++i) acc = fma((double)k.v[i], (double)v.v[i], acc);
        }
        if ((j & (kBand - 1)) == kBand - 1 || j == t.y1 - 1) {
          band_sum(g, t, c, lane, j, acc, sums.part);
          acc = 0.0;
        }
      }
      m = k;
      k = n;
      ak = a;
    }
  }
  double pq;
  if (unit_sum(g, c, sums, &pq)) sc[S_PQ] = pq;
}

// x += alpha p, r -= alpha q (alpha = rho / p.q, q = A_0 p); ||r||^2
__global__ void __launch_bounds__(kStripWarps * 32) k_cg_step(const Geo *__restrict__ geo,
                                                              const int4 *__restrict__ bmap, const Geo one,
                                                              const uint8_t *__restrict__ flags,
                                                              const uint8_t *__restrict__ act,
                                                              const float *__restrict__ p, float *__restrict__ x,
                                                              float *__restrict__ r, const double *__restrict__ run,
                                                              Sums sums, double *__restrict__ rr) {
  const int4 bt = entry_of(bmap, one);
  const int c = blockIdx.z, lane = threadIdx.x & 31;
  if (c >= bt.z || run[bt.y + c] == 0.0) return;  // a stopped unit: x and r stay
  const Geo g = bmap ? geo[bt.x] : one;
  const double *sc = sums.sc + (long long)(g.unit0 + c) * S_N;
  Strip t;
  if (strip_of(g, flags, t)) {
    const float alpha = sc[S_PQ] > 0.0 ? (float)(sc[S_RHO] / sc[S_PQ]) : 0.0f, d = g.d;
    const long long at = g.oc + (long long)c * g.P * g.H + t.x0;
    const uint8_t *a0 = act + g.o + t.x0;
    // p was written only in bands with active cells: elsewhere it is 0
    auto fetch = [&](int y, unsigned a) {
      Row v = t.in && y >= 0 && y < g.H ? ld_row(p + at + (long long)y * g.P) : row0();
#pragma unroll
      for (int i = 0; i < 4; ++i) v.v[i] = a & (1u << i) ? v.v[i] : 0.0f;
      return v;
    };
    auto flag = [&](int y) {
      return t.in && y >= 0 && y < g.H ? nibble(*reinterpret_cast<const uint32_t *>(a0 + (long long)y * g.P)) : 0u;
    };
    double acc = 0.0;
    unsigned a = flag(t.y0);
    Row up = fetch(t.y0 - 1, flag(t.y0 - 1)), k = fetch(t.y0, a);
    // the rows of a band in two halves, each half's loads before its stores
    constexpr int kHalf = kBand / 2;
    for (int j0 = t.y0; j0 < t.y1; j0 += kHalf) {
      const int n = min(kHalf, t.y1 - j0);
      unsigned an[kHalf];
      Row P[kHalf], X[kHalf], S[kHalf];
#pragma unroll
      for (int q = 0; q < kHalf; ++q) an[q] = flag(j0 + q + 1);
#pragma unroll
      for (int q = 0; q < kHalf; ++q) {
        const long long o = at + (long long)(j0 + min(q, n - 1)) * g.P;
        P[q] = fetch(j0 + q + 1, an[q]);
        X[q] = t.own ? ld_row(x + o) : row0();
        S[q] = t.own ? ld_row(r + o) : row0();
      }
#pragma unroll
      for (int q = 0; q < kHalf; ++q) {
        if (q >= n) break;
        const Row Q = apply_row(k, up, P[q], a, d);
        if (t.own) {
          const long long o = at + (long long)(j0 + q) * g.P;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            X[q].v[i] = X[q].v[i] + alpha * k.v[i];
            S[q].v[i] = S[q].v[i] - alpha * Q.v[i];
            acc = fma((double)S[q].v[i], (double)S[q].v[i], acc);
          }
          st_row(x + o, X[q]);
          st_row(r + o, S[q]);
        }
        up = k;
        k = P[q];
        a = an[q];
      }
      const int j = j0 + n - 1;
      if ((j & (kBand - 1)) == kBand - 1 || j == t.y1 - 1) {
        band_sum(g, t, c, lane, j, acc, sums.part);
        acc = 0.0;
      }
    }
  }
  double v;
  if (unit_sum(g, c, sums, &v)) rr[g.unit0 + c] = v;
}

// out = interleave(u) at interior cells, the anchor elsewhere (bit for bit);
// level-0 tiles, grid.z 1. A thread takes four consecutive values of a row of
// the interleaved image; whole where both images allow (16-byte alignment).
__global__ void __launch_bounds__(kTx * kTy) k_mg_emit(const Geo *__restrict__ geo,
                                                       const int4 *__restrict__ bmap, const Geo one,
                                                       const Io *__restrict__ io, const uint8_t *__restrict__ act,
                                                       const double *__restrict__ u) {
  const int4 bt = entry_of(bmap, one);
  const int gi = bt.x;
  const Geo g = bmap ? geo[gi] : one;
  const Io f = io[gi];
  const int C = g.C, W = g.W, H = g.H, b = tile_b(g);
  const size_t N = (size_t)g.P * H, row = (size_t)W * C;
  const uint8_t *a = act + g.o;
  const double *u0 = u + g.oc;
  const int first = (b % g.gx) * kTx, values = min(kTx, W - first) * C;
  const bool whole = ((reinterpret_cast<uintptr_t>(f.out) | reinterpret_cast<uintptr_t>(f.anchor)) & 15) == 0 && row % 4 == 0;
  for (int j = (b / g.gx) * kTy + threadIdx.y; j < H; j += g.gy * kTy)
    // the tile's columns hold C values each: the lanes walk over them
    for (int e = 4 * threadIdx.x; e < values; e += 4 * kTx) {
      int i = first + e / C, c = e % C;
      const int n = min(4, values - e);
      float v[4];
      const size_t o = j * row + (size_t)first * C + e;
      const float *from = f.anchor + o;
      if (whole && n == 4) {
        const float4 q = *reinterpret_cast<const float4 *>(from);
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = k < n ? from[k] : 0.0f;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (k < n) {
          const size_t at = (size_t)j * g.P + i;
          if (a[at]) v[k] = (float)u0[c * N + at];
        }
        if (++c == C) {
          c = 0;
          ++i;
        }
      }
      float *to = f.out + o;
      if (whole && n == 4) {
        *reinterpret_cast<float4 *>(to) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (k < n) to[k] = v[k];
      }
    }
}

// ---- host ----------------------------------------------------------------------
size_t aup(size_t b) { return (b + 255) & ~(size_t)255; }

// (32, 8)-thread tiles over w columns and h rows of one instance: at most
// about 8 tiles per SM per channel.
void tiles2(int w, int h, int sms, int &gx, int &gy) {
  gx = std::max(1, (w + kTx - 1) / kTx);
  gy = std::min(std::max(1, (h + kTy - 1) / kTy), std::max(1, sms * 8 / gx));
  gy = std::min(gy, 65535);
}
const dim3 kBlock2(kTx, kTy), kStrip(kStripWarps * 32);

int pitch(int w) { return (w + 3) / 4 * 4; }
long long bands(int w, int h) { return (long long)strip_cols(w) * ((h + kBand - 1) / kBand); }

float level_s(int k) { return 1.0f / (float)(1u << (2 * std::min(k, 15))); }

// A call is cut into groups of at most this many level-0 bands (and units);
// every launch of a group then has fewer blocks.
constexpr long long kGroupTiles = 1ll << 22;

// Strips: at most kMostRows rows, fewer until a launch has kFewStrips an SM.
constexpr int kMostRows = 64, kFewStrips = 16;

// One instance (a problem with channels) of a group
struct Inst {
  int idx;                       // its index in the caller's arrays
  int W, H, C, L;                // extent, channels, levels
  double lambda;
  std::vector<int> w, h;         // level extents
  std::vector<long long> o, oc, f;  // level offsets in the one-channel, C-channel and flag arrays
  int k0 = 0;                    // the first level of the one-block tail
  int unit0 = 0;                 // first (instance, channel) unit
  long long part0 = 0;           // first level-0 partial sum
  bool dev = false, warm = false;
  size_t in = 0, mask = 0, guess = 0, out = 0;  // staged copies of host buffers
};

// One kind of launch at one level: its table entries and blocks
struct Launch {
  size_t geo = 0, bmap = 0;  // byte offsets of the tables in the table area
  int n = 0;                 // entries (instances)
  long long blocks = 0;
  Geo one{};                 // the entry of a launch over one instance (passed by value)
};

// A level's arrays: interior flags, band flags, the correction after the pass
// down and after the pass up, the right-hand side
struct LevelArr {
  size_t act = 0, flags = 0, e = 0, eu = 0, rhs = 0;
};

// Tables built on the host and uploaded in one copy
struct Blob {
  std::vector<unsigned char> b;
  size_t put(const void *p, size_t n) {
    const size_t o = (b.size() + 15) & ~(size_t)15;
    b.resize(o + n);
    if (n) std::memcpy(b.data() + o, p, n);
    return o;
  }
};

// Strip launches (strips true) have kStripWarps strips a block.
Launch make_launch(Blob &blob, std::vector<Geo> &gs, bool strips) {
  auto count = [&](const Geo &g) {
    const long long n = (long long)g.gx * g.gy;
    return strips ? (n + kStripWarps - 1) / kStripWarps : n;
  };
  Launch l;
  l.n = (int)gs.size();
  if (gs.size() == 1) {  // one instance: its geometry goes by value, no block map
    gs[0].blk0 = 0;
    l.one = gs[0];
    l.blocks = count(gs[0]);
    l.geo = blob.put(gs.data(), sizeof(Geo));
    return l;
  }
  std::vector<int4> bm;
  long long blk = 0;
  for (size_t k = 0; k < gs.size(); ++k) {
    gs[k].blk0 = (int)blk;
    const long long nb = count(gs[k]);
    bm.insert(bm.end(), (size_t)nb, make_int4((int)k, gs[k].unit0, gs[k].C, 0));
    blk += nb;
  }
  l.blocks = blk;
  l.geo = blob.put(gs.data(), gs.size() * sizeof(Geo));
  l.bmap = blob.put(bm.data(), bm.size() * sizeof(int4));
  return l;
}

struct Mg {
  pt_ctx *ctx;
  cudaStream_t st;
  char *base = nullptr;
  unsigned Cmax = 1;
  int U = 0;
  std::vector<Inst> in;
  std::vector<LevelArr> lv;
  Launch tiles0, strips0, dot0;  // level 0: tiles; strips; strips of instances without a finer level than the coarsest
  std::vector<Launch> strips, coarsen;  // per level
  size_t tails = 0;              // table of the tails, in the table area
  int ntails = 0;
  size_t tail_smem = 0;
  size_t tab = 0, io = 0;
  size_t u = 0, bl = 0, uw = 0, r64 = 0, part = 0, done = 0, red = 0, sc = 0, scale = 0, run = 0, x = 0, r = 0, z = 0,
         q = 0;
  size_t p[2] = {0, 0};          // the search direction's two arrays (k_cg_apply), in r64's place
  long long launches = 0;
  template <class T> T *at(size_t off) { return reinterpret_cast<T *>(base + off); }
  const Geo *geo(const Launch &l) { return at<Geo>(tab + l.geo); }
  const int4 *bmap(const Launch &l) { return l.n == 1 ? nullptr : at<int4>(tab + l.bmap); }
  dim3 grid(const Launch &l, unsigned z) { return dim3((unsigned)l.blocks, 1, z); }
};

// One V-cycle z = M r (level 0's correction on the way is the vector q), and
// with its last pass rho = r.z and beta.
void vcycle(Mg &m, int first) {
  const int L = (int)m.strips.size();
  const unsigned Cz = m.Cmax;
  const double *run = m.at<double>(m.run);
  const Sums sums{m.at<double>(m.part), m.at<unsigned>(m.done), m.at<double>(m.sc)};
  auto rhs = [&](int k) { return k ? m.at<float>(m.lv[k].rhs) : m.at<float>(m.r); };
  auto down = [&](int k) { return k ? m.at<float>(m.lv[k].e) : m.at<float>(m.q); };
  for (int k = 0; k < L; ++k) {
    const Launch &S = m.strips[k];
    if (!S.n) continue;
    k_mg_down<<<m.grid(S, Cz), kStrip, 0, m.st>>>(m.geo(S), m.bmap(S), S.one, m.at<uint8_t>(m.lv[k].flags),
                                                  m.at<uint8_t>(m.lv[k].act), rhs(k), down(k),
                                                  m.at<uint8_t>(m.lv[k + 1].act), rhs(k + 1), run);
    ++m.launches;
  }
  k_mg_tail<<<dim3((unsigned)m.ntails, 1, Cz), dim3(kTailX, kTailY), m.tail_smem, m.st>>>(
      m.at<Tail>(m.tab + m.tails), run);
  ++m.launches;
  for (int k = L - 1; k >= 0; --k) {
    const Launch &S = m.strips[k];
    if (!S.n) continue;
    float *out = k ? m.at<float>(m.lv[k].eu) : m.at<float>(m.z);
    if (k == 0)
      k_mg_up<true><<<m.grid(S, Cz), kStrip, 0, m.st>>>(m.geo(S), m.bmap(S), S.one, m.at<uint8_t>(m.lv[k].flags),
                                                        m.at<uint8_t>(m.lv[k].act), rhs(k), down(k),
                                                        m.at<float>(m.lv[k + 1].eu), out, run, sums, first);
    else
      k_mg_up<false><<<m.grid(S, Cz), kStrip, 0, m.st>>>(m.geo(S), m.bmap(S), S.one, m.at<uint8_t>(m.lv[k].flags),
                                                         m.at<uint8_t>(m.lv[k].act), rhs(k), down(k),
                                                         m.at<float>(m.lv[k + 1].eu), out, run, sums, first);
    ++m.launches;
  }
  if (m.dot0.n) {
    k_cg_dot<<<m.grid(m.dot0, Cz), kStrip, 0, m.st>>>(m.geo(m.dot0), m.bmap(m.dot0), m.dot0.one,
                                                      m.at<uint8_t>(m.lv[0].flags), m.at<float>(m.r), m.at<float>(m.z),
                                                      run, sums, first);
    ++m.launches;
  }
}

pt_status mfail(pt_ctx *ctx, pt_status s, const std::string &msg) {
  ctx->last_error = msg;
  return s;
}

// One group of instances (ids: indices into ps, all with channels > 0)
pt_status solve_group(pt_ctx *ctx, const pt_problem *ps, const std::vector<int> &ids, float *const *outs,
                      pt_report *const *reports, double *const *histories, double &solve_ms, double &call_ms,
                      long long &launches) {
  const int sms = ctx->sms;
  Mg m;
  m.ctx = ctx;
  m.st = ctx->stream;
  // instances, their levels (halve, ceil, while a level has more than
  // kCoarseMax cells), units and level-0 partial sums
  int Lmax = 0;
  long long P = 0;
  bool any_warm = false;
  for (int id : ids) {
    const pt_problem &p = ps[id];
    Inst I;
    I.idx = id; I.W = (int)p.width; I.H = (int)p.height; I.C = (int)p.channels; I.lambda = p.lambda;
    I.dev = (p.flags & PT_FLAG_DEVICE_POINTERS) != 0;
    I.warm = (p.flags & PT_FLAG_WARM_START) != 0;
    int w = I.W, h = I.H, k = 0;
    for (;;) {
      I.w.push_back(w);
      I.h.push_back(h);
      if ((long long)w * h <= kCoarseMax || k >= 30) break;
      w = (w + 1) / 2; h = (h + 1) / 2; ++k;
    }
    I.L = (int)I.w.size();
    // the tail: the levels of few cells, and at least the coarsest
    auto in_tail = [&](int k) {
      size_t all = 0;
      for (int l = k; l < I.L; ++l) all += (size_t)I.w[l] * I.h[l];
      const size_t first = (size_t)I.w[k] * I.h[k];
      return first <= (size_t)kTailCells && I.L - k <= kTailLevels && tail_bytes(all, first) <= (size_t)kTailSmem;
    };
    while (I.k0 < I.L - 1 && (I.k0 == 0 || !in_tail(I.k0))) ++I.k0;
    I.unit0 = m.U;
    m.U += I.C;
    I.part0 = P;
    P += (long long)I.C * bands(I.W, I.H);
    Lmax = std::max(Lmax, I.L);
    m.Cmax = std::max(m.Cmax, (unsigned)I.C);
    any_warm |= I.warm;
    m.in.push_back(std::move(I));
  }
  const int U = m.U;
  std::vector<long long> cells(Lmax, 0), ccells(Lmax, 0), nflags(Lmax, 0);
  for (Inst &I : m.in)
    for (int k = 0; k < I.L; ++k) {
      I.o.push_back(cells[k]);
      I.oc.push_back(ccells[k]);
      I.f.push_back(nflags[k]);
      const long long n = (long long)pitch(I.w[k]) * I.h[k];
      cells[k] += n;
      ccells[k] += I.C * n;
      nflags[k] += bands(I.w[k], I.h[k]);
    }

  // launch tables
  Blob blob;
  auto geo_at = [&](const Inst &I, int k) {
    Geo g{};
    g.W = I.w[k]; g.H = I.h[k]; g.P = pitch(g.W);
    g.C = I.C; g.unit0 = I.unit0; g.part0 = I.part0;
    g.o = I.o[k]; g.oc = I.oc[k]; g.f = I.f[k];
    g.s = level_s(k);
    g.d = 4.0f * g.s + (float)I.lambda;
    g.lambda = I.lambda;
    return g;
  };
  auto second = [](Geo &g, const Inst &I, int k) {
    g.W2 = I.w[k]; g.H2 = I.h[k]; g.P2 = pitch(g.W2); g.o2 = I.o[k]; g.oc2 = I.oc[k];
  };
  auto tiled = [&](Geo g) {
    tiles2(g.P, g.H, sms, g.gx, g.gy);
    return g;
  };
  auto stripped = [&](Geo g, int rows) {
    g.rows = rows;
    g.gx = strip_cols(g.W);
    g.gy = (g.H + rows - 1) / rows;
    return g;
  };
  // Rows a strip: as many as leave the launch kFewStrips strips. A strip walks
  // about ten rows more than it owns (five halo rows either side), so long ones
  // do less twice; short ones fill the GPU on small levels.
  auto rows_for = [&](int k, bool all) {
    for (int rows = kMostRows; rows > kBand; rows /= 2) {
      long long n = 0;
      for (const Inst &I : m.in)
        if (all || k < I.k0) n += (long long)I.C * strip_cols(I.w[std::min(k, I.L - 1)]) * ((I.h[std::min(k, I.L - 1)] + rows - 1) / rows);
      if (n >= (long long)kFewStrips * sms) return rows;
    }
    return kBand;
  };
  {
    std::vector<Geo> gt, gs, gd;
    const int rows = rows_for(0, true);
    for (const Inst &I : m.in) {
      Geo g = geo_at(I, 0);
      gt.push_back(tiled(g));
      gs.push_back(stripped(g, rows));
      if (I.k0 == 0) gd.push_back(stripped(g, rows));
    }
    m.tiles0 = make_launch(blob, gt, false);
    m.strips0 = make_launch(blob, gs, true);
    m.dot0 = make_launch(blob, gd, true);
  }
  m.strips.resize(Lmax); m.coarsen.resize(Lmax);
  for (int k = 0; k < Lmax; ++k) {
    std::vector<Geo> gs, gc;
    const int rows = rows_for(k, k == 0);
    for (const Inst &I : m.in) {
      if (k < I.k0) {
        Geo g = geo_at(I, k);
        second(g, I, k + 1);
        gs.push_back(stripped(g, rows));
      }
      if (k + 1 < I.L) {
        Geo g = geo_at(I, k + 1);
        second(g, I, k);
        gc.push_back(tiled(g));
      }
    }
    m.strips[k] = make_launch(blob, gs, true);
    m.coarsen[k] = make_launch(blob, gc, false);
  }

  // arena: tables, levels, level-0 vectors, then the staged host buffers
  size_t o = 0;
  auto take = [&](size_t b) { size_t r = o; o = aup(o + std::max<size_t>(b, 1)); return r; };
  m.tails = blob.b.size() + 64;  // (the tails' table follows: it holds arena addresses)
  m.ntails = (int)m.in.size();
  m.tails = (m.tails + 15) & ~(size_t)15;
  m.tab = take(m.tails + m.in.size() * sizeof(Tail));
  m.io = take(m.in.size() * sizeof(Io));
  m.lv.resize(Lmax);
  for (int k = 0; k < Lmax; ++k) {
    m.lv[k].act = take((size_t)cells[k]);
    if (k > 0) {
      m.lv[k].e = take((size_t)ccells[k] * sizeof(float));
      m.lv[k].rhs = take((size_t)ccells[k] * sizeof(float));
    }
  }
  // cleared once a call, in one piece: the corrections after the passes up, the
  // bands' flags and partial sums, the counts of finished blocks
  const size_t clear0 = o;
  for (int k = 1; k < Lmax; ++k) m.lv[k].eu = take((size_t)ccells[k] * sizeof(float));
  for (int k = 0; k < Lmax; ++k) m.lv[k].flags = take((size_t)nflags[k]);
  m.part = take((size_t)P * 8); m.done = take((size_t)U * sizeof(unsigned));
  const size_t clear1 = o;
  const size_t NC = (size_t)ccells[0];
  m.u = take(NC * 8); m.bl = take(NC * 8); m.uw = any_warm ? take(NC * 8) : 0; m.r64 = take(NC * 8);
  m.red = take((size_t)U * 8); m.sc = take((size_t)U * S_N * 8);
  m.scale = take((size_t)U * 8); m.run = take((size_t)U * 8);
  m.x = take(NC * 4); m.r = take(NC * 4); m.z = take(NC * 4); m.q = take(NC * 4);
  // The search direction lies where the FP64 residual does: k_mg_scale reads that
  // for the last time before a run's first k_cg_apply, which reads no direction, and
  // k_mg_residual64 writes it anew after the run. (A call then needs 45 bytes a
  // cell and channel of level 0.)
  m.p[0] = m.r64; m.p[1] = m.r64 + NC * 4;
  for (Inst &I : m.in) {
    if (I.dev) continue;
    const size_t n = (size_t)I.W * I.H, nc = n * I.C;
    I.in = take(nc * 2 * 4); I.mask = take(n * 4); I.guess = I.warm ? take(nc * 4) : 0; I.out = take(nc * 4);
  }
  if (!ctx->reserve(o)) return mfail(ctx, PT_OOM, "device arena allocation failed");
  m.base = static_cast<char *>(ctx->arena);
  cudaEventRecord(ctx->ev[0], m.st);

  // the tails (they hold addresses in the arena)
  blob.b.resize(m.tails);
  for (const Inst &I : m.in) {
    Tail T{};
    T.C = I.C; T.unit0 = I.unit0; T.n = I.L - I.k0;
    T.pow2 = I.lambda == 0.0;
    size_t cells_all = 0;
    for (int l = 0; l < T.n; ++l) {
      const int k = I.k0 + l;
      T.w[l] = I.w[k]; T.h[l] = I.h[k]; T.P[l] = pitch(I.w[k]);
      T.o[l] = I.o[k];
      T.act[l] = m.at<uint8_t>(m.lv[k].act);
      T.s[l] = level_s(k);
      T.d[l] = 4.0f * T.s[l] + (float)I.lambda;
      cells_all += (size_t)I.w[k] * I.h[k];
    }
    T.rhs = (I.k0 ? m.at<float>(m.lv[I.k0].rhs) : m.at<float>(m.r)) + I.oc[I.k0];
    T.e = (I.k0 ? m.at<float>(m.lv[I.k0].eu) : m.at<float>(m.z)) + I.oc[I.k0];
    blob.put(&T, sizeof(T));
    m.tail_smem = std::max(m.tail_smem, tail_bytes(cells_all, (size_t)I.w[I.k0] * I.h[I.k0]));
  }
  static_assert(sizeof(Tail) % 16 == 0, "the tails lie one after another");

  // tables and inputs
  cudaError_t ce = cudaSuccess;
  if (!ctx->mg_prepared) {  // once a context
    ce = cudaFuncSetAttribute(k_mg_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailSmem);
    ctx->mg_prepared = ce == cudaSuccess;
  }
  if (ce == cudaSuccess)
    ce = cudaMemcpyAsync(m.base + m.tab, blob.b.data(), blob.b.size(), cudaMemcpyHostToDevice, m.st);
  if (ce == cudaSuccess) ce = cudaMemsetAsync(m.base + clear0, 0, clear1 - clear0, m.st);
  std::vector<Io> io(m.in.size());
  for (size_t k = 0; k < m.in.size() && ce == cudaSuccess; ++k) {
    const Inst &I = m.in[k];
    const pt_problem &p = ps[I.idx];
    const size_t n = (size_t)I.W * I.H, nc = n * I.C;
    if (I.dev) {
      io[k] = Io{p.source_or_guidance, p.target_or_anchor, p.mask, I.warm ? p.initial_guess : nullptr, outs[I.idx]};
      continue;
    }
    float *in = m.at<float>(I.in);
    ce = cudaMemcpyAsync(in, p.source_or_guidance, nc * 4, cudaMemcpyHostToDevice, m.st);
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(in + nc, p.target_or_anchor, nc * 4, cudaMemcpyHostToDevice, m.st);
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(m.at<float>(I.mask), p.mask, n * 4, cudaMemcpyHostToDevice, m.st);
    if (ce == cudaSuccess && I.warm)
      ce = cudaMemcpyAsync(m.at<float>(I.guess), p.initial_guess, nc * 4, cudaMemcpyHostToDevice, m.st);
    io[k] = Io{in, in + nc, m.at<float>(I.mask), I.warm ? m.at<float>(I.guess) : nullptr, m.at<float>(I.out)};
  }
  if (ce == cudaSuccess)
    ce = cudaMemcpyAsync(m.base + m.io, io.data(), io.size() * sizeof(Io), cudaMemcpyHostToDevice, m.st);
  if (ce != cudaSuccess) return mfail(ctx, PT_LAUNCH_FAILED, std::string("input upload: ") + cudaGetErrorString(ce));

  const Io *iod = m.at<Io>(m.io);
  const Launch &A = m.tiles0, &S0 = m.strips0;
  const Geo *g0 = m.geo(S0);
  const int4 *b0 = m.bmap(S0);
  const dim3 gs = m.grid(S0, m.Cmax);
  uint8_t *act0 = m.at<uint8_t>(m.lv[0].act);
  const uint8_t *fl0 = m.at<uint8_t>(m.lv[0].flags);
  double *u = m.at<double>(m.u), *bl = m.at<double>(m.bl), *r64 = m.at<double>(m.r64), *red = m.at<double>(m.red),
         *sc = m.at<double>(m.sc), *scale = m.at<double>(m.scale), *run = m.at<double>(m.run);
  float *x = m.at<float>(m.x), *r = m.at<float>(m.r), *z = m.at<float>(m.z);
  float *pp[2] = {m.at<float>(m.p[0]), m.at<float>(m.p[1])};
  const Sums sums{m.at<double>(m.part), m.at<unsigned>(m.done), sc};
  k_mg_assemble<<<m.grid(A, 1), kBlock2, 0, m.st>>>(m.geo(A), m.bmap(A), A.one, iod, act0, m.at<uint8_t>(m.lv[0].flags), u, bl,
                                                     any_warm ? m.at<double>(m.uw) : nullptr);
  m.launches = 1;
  for (int k = 0; k < Lmax; ++k) {
    const Launch &K = m.coarsen[k];
    if (!K.n) continue;
    k_mg_coarsen<<<m.grid(K, 1), kBlock2, 0, m.st>>>(m.geo(K), m.bmap(K), K.one, m.at<uint8_t>(m.lv[k].act),
                                                     m.at<uint8_t>(m.lv[k + 1].act), m.at<uint8_t>(m.lv[k + 1].flags));
    ++m.launches;
  }
  cudaEventRecord(ctx->ev[1], m.st);

  // per-unit facts
  std::vector<int> uinst(U), maxit(U);
  std::vector<double> tol(U);
  for (size_t k = 0; k < m.in.size(); ++k)
    for (int c = 0; c < m.in[k].C; ++c) {
      const int un = m.in[k].unit0 + c;
      uinst[un] = (int)k;
      tol[un] = ps[m.in[k].idx].tolerance;
      maxit[un] = (int)ps[m.in[k].idx].max_iterations;
    }

  // FP64 residual norms per unit of the current u -> host
  std::vector<double> nrm(U);
  auto residual = [&](const double *uu) -> cudaError_t {
    k_mg_residual64<<<gs, kStrip, 0, m.st>>>(g0, b0, S0.one, fl0, act0, uu, bl, r64, sums, red);
    ++m.launches;
    cudaError_t e = cudaMemcpyAsync(nrm.data(), red, (size_t)U * 8, cudaMemcpyDeviceToHost, m.st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m.st);
    for (double &v : nrm) v = std::sqrt(v);
    return e;
  };
  ce = residual(u);
  if (ce != cudaSuccess) return mfail(ctx, PT_LAUNCH_FAILED, std::string("residual: ") + cudaGetErrorString(ce));
  const std::vector<double> r0 = nrm;  // ||r(anchor)|| per unit: the bar is tolerance * r0
  std::vector<int> warm_used(U, 0);
  if (any_warm) {
    double *uw = m.at<double>(m.uw);
    ce = residual(uw);
    if (ce != cudaSuccess) return mfail(ctx, PT_LAUNCH_FAILED, std::string("residual: ") + cudaGetErrorString(ce));
    // a guess is used per channel only if its residual is finite and below the anchor's
    for (int un = 0; un < U; ++un) {
      const Inst &I = m.in[uinst[un]];
      if (!I.warm || !(std::isfinite(nrm[un]) && nrm[un] < r0[un])) continue;
      warm_used[un] = 1;
      const size_t n = (size_t)pitch(I.W) * I.H, off = (size_t)I.oc[0] + (size_t)(un - I.unit0) * n;
      cudaMemcpyAsync(u + off, uw + off, n * 8, cudaMemcpyDeviceToDevice, m.st);
    }
    ce = residual(u);
    if (ce != cudaSuccess) return mfail(ctx, PT_LAUNCH_FAILED, std::string("residual: ") + cudaGetErrorString(ce));
  }

  // per-unit state
  std::vector<int> its(U, 0), stop(U, -1), refines(U, 0);
  std::vector<double> cur = nrm;  // FP64 ||r|| of the current u
  std::vector<std::vector<double>> hist(U);
  std::vector<double> hscale(U, 0.0), hrun(U, 0.0), rr(U);
  bool poisoned = false;
  for (int un = 0; un < U; ++un) {
    if (r0[un] == 0.0) stop[un] = PT_STOP_CONVERGED;  // poisson.rs:178-185
    else if (!std::isfinite(cur[un])) {  // (before the bar: inf <= tol * inf would pass it)
      // a NaN or infinity reached the system: its residual can never improve,
      // which the reference ends by its stall rule with the region's cells
      // non-finite; here at once, with the interior set to NaN
      stop[un] = PT_STOP_STALLED;
      hscale[un] = std::nan("");
      poisoned = true;
    } else if (cur[un] <= tol[un] * r0[un]) stop[un] = PT_STOP_CONVERGED;
    else if (maxit[un] == 0) stop[un] = PT_STOP_MAX_ITERATIONS;
  }
  if (poisoned) {  // u = fma(NaN, 0, u) = NaN at interior cells of those units
    cudaMemcpyAsync(scale, hscale.data(), (size_t)U * 8, cudaMemcpyHostToDevice, m.st);
    k_mg_update<<<gs, kStrip, 0, m.st>>>(g0, b0, S0.one, fl0, act0, nullptr, scale, u);
    ++m.launches;
    std::fill(hscale.begin(), hscale.end(), 0.0);
  }
  // One CG iteration: V-cycle z = M r, rho = r.z, p = z + beta p, q = A p,
  // alpha = rho / p.q, x += alpha p, r -= alpha q, ||r||^2 (to `red`). Its
  // launches depend only on the group's shapes and the arena, so they are
  // captured once into three CUDA graphs (first iteration, later odd and even
  // ones) cached on the context and replayed while shapes and arena stay the same.
  long long per_iteration = 0;
  // kind 0: the first iteration; 1, 2: the later ones, which take p from one
  // array to the other
  auto enqueue_iteration = [&](int kind) -> cudaError_t {
    const long long l0 = m.launches;
    float *p = pp[kind == 1 ? 0 : 1], *pn = pp[kind == 1 ? 1 : 0];
    const int first = kind == 0;
    vcycle(m, first);
    k_cg_apply<<<gs, kStrip, 0, m.st>>>(g0, b0, S0.one, fl0, act0, z, p, pn, run, sums, first);
    k_cg_step<<<gs, kStrip, 0, m.st>>>(g0, b0, S0.one, fl0, act0, pn, x, r, run, sums, red);
    m.launches += 2;
    per_iteration = m.launches - l0;
    return cudaGetLastError();
  };
  if (ctx->graphs) {
    // the graphs' arguments are arena offsets and the tables' contents
    std::string key(reinterpret_cast<const char *>(&m.base), sizeof(m.base));
    std::vector<size_t> offs = {o, m.tab, m.tails, m.part, m.done, m.red, m.sc, m.run, m.x, m.r, m.z, m.p[0], m.p[1], m.q,
                                (size_t)m.Cmax, (size_t)U};
    for (const LevelArr &v : m.lv) offs.insert(offs.end(), {v.act, v.flags, v.e, v.eu, v.rhs});
    key.append(reinterpret_cast<const char *>(offs.data()), offs.size() * sizeof(size_t));
    key.append(reinterpret_cast<const char *>(blob.b.data()), blob.b.size());
    if (key != ctx->mgkey || !ctx->mgexec[0] || !ctx->mgexec[1] || !ctx->mgexec[2]) {
      for (auto &ge : ctx->mgexec)
        if (ge) { cudaGraphExecDestroy(ge); ge = nullptr; }
      ctx->mgkey.clear();
      const long long saved = m.launches;
      for (int g = 0; g < 3 && ce == cudaSuccess; ++g) {
        cudaGraph_t graph = nullptr;
        ce = cudaStreamBeginCapture(m.st, cudaStreamCaptureModeThreadLocal);
        if (ce == cudaSuccess) {
          const cudaError_t e1 = enqueue_iteration(g);
          ce = cudaStreamEndCapture(m.st, &graph);
          if (e1 != cudaSuccess) ce = e1;
        }
        if (ce == cudaSuccess) ce = cudaGraphInstantiate(&ctx->mgexec[g], graph, 0);
        if (graph) cudaGraphDestroy(graph);
      }
      m.launches = saved;
      ctx->mgnodes = per_iteration;
      if (ce != cudaSuccess) {
        for (auto &ge : ctx->mgexec)
          if (ge) { cudaGraphExecDestroy(ge); ge = nullptr; }
        return mfail(ctx, PT_LAUNCH_FAILED, std::string("graph capture: ") + cudaGetErrorString(ce));
      }
      ctx->mgkey = std::move(key);
    }
  }
  int outer = 0;
  while (std::any_of(stop.begin(), stop.end(), [](int s) { return s < 0; })) {
    // scale this outer step's residual to unit norm; units that stopped get 0
    for (int un = 0; un < U; ++un) {
      hscale[un] = stop[un] < 0 ? cur[un] : 0.0;
      hrun[un] = stop[un] < 0 ? 1.0 : 0.0;
    }
    cudaMemcpyAsync(scale, hscale.data(), (size_t)U * 8, cudaMemcpyHostToDevice, m.st);
    cudaMemcpyAsync(run, hrun.data(), (size_t)U * 8, cudaMemcpyHostToDevice, m.st);
    cudaMemsetAsync(sc, 0, (size_t)U * S_N * 8, m.st);
    k_mg_scale<<<gs, kStrip, 0, m.st>>>(g0, b0, S0.one, fl0, r64, scale, r, x);
    m.launches += 1;
    // inner target: a quarter of the remaining bar, at most as deep as FP32
    // goes from a unit residual; a run whose residual stops falling (less than
    // 30% over 4 iterations: the FP32 floor) hands over to the next outer step
    std::vector<double> target(U), rel(U, 1.0);
    std::vector<std::vector<double>> seen(U);
    std::vector<int> going(U);
    for (int un = 0; un < U; ++un) {
      going[un] = stop[un] < 0;
      target[un] = going[un] ? std::max(0.25 * tol[un] * r0[un] / cur[un], kInnerFloor) : 1.0;
    }
    for (int it = 0;; ++it) {
      const int g = it == 0 ? 0 : 2 - (it & 1);
      if (ctx->mgexec[g]) {
        ce = cudaGraphLaunch(ctx->mgexec[g], m.st);
        m.launches += ctx->mgnodes;
      } else {
        ce = enqueue_iteration(g);
      }
      if (ce != cudaSuccess) return mfail(ctx, PT_LAUNCH_FAILED, std::string("cg: ") + cudaGetErrorString(ce));
      ce = cudaMemcpyAsync(rr.data(), red, (size_t)U * 8, cudaMemcpyDeviceToHost, m.st);
      if (ce == cudaSuccess) ce = cudaStreamSynchronize(m.st);
      if (ce != cudaSuccess) return mfail(ctx, PT_LAUNCH_FAILED, std::string("cg: ") + cudaGetErrorString(ce));
      bool any = false, changed = false;
      for (int un = 0; un < U; ++un) {
        if (!going[un]) continue;
        its[un] += 1;
        rel[un] = std::sqrt(rr[un]);  // relative to this outer step's unit residual
        hist[un].push_back(rel[un] * cur[un] / r0[un]);
        seen[un].push_back(rel[un]);
        const size_t n = seen[un].size();
        const bool stuck = n > 4 && seen[un][n - 1] > 0.7 * seen[un][n - 5];
        if (rel[un] <= target[un] || stuck || its[un] >= maxit[un] || !std::isfinite(rel[un])) {
          going[un] = 0;
          hrun[un] = 0.0;
          changed = true;
        }
        any |= going[un] != 0;
      }
      if (!any) break;
      if (changed) cudaMemcpyAsync(run, hrun.data(), (size_t)U * 8, cudaMemcpyHostToDevice, m.st);
    }
    // u += scale * x, then the FP64 residual decides
    k_mg_update<<<gs, kStrip, 0, m.st>>>(g0, b0, S0.one, fl0, act0, x, scale, u);
    ++m.launches;
    const std::vector<double> prev = cur;
    ce = residual(u);
    if (ce != cudaSuccess) return mfail(ctx, PT_LAUNCH_FAILED, std::string("residual: ") + cudaGetErrorString(ce));
    for (int un = 0; un < U; ++un) {
      if (stop[un] >= 0) continue;
      cur[un] = nrm[un];
      if (!hist[un].empty()) hist[un].back() = cur[un] / r0[un];
      if (outer > 0) refines[un] += 1;
      if (cur[un] <= tol[un] * r0[un]) stop[un] = PT_STOP_CONVERGED;
      else if (its[un] >= maxit[un]) stop[un] = PT_STOP_MAX_ITERATIONS;
      else if (!(cur[un] < prev[un] * (1.0 - 1e-12))) stop[un] = PT_STOP_STALLED;
    }
    ++outer;
  }
  cudaEventRecord(ctx->ev[2], m.st);
  k_mg_emit<<<m.grid(A, 1), kBlock2, 0, m.st>>>(m.geo(A), m.bmap(A), A.one, iod, act0, u);
  ++m.launches;
  ce = cudaSuccess;
  for (size_t k = 0; k < m.in.size() && ce == cudaSuccess; ++k) {
    const Inst &I = m.in[k];
    if (!I.dev)
      ce = cudaMemcpyAsync(outs[I.idx], m.at<float>(I.out), (size_t)I.W * I.H * I.C * 4, cudaMemcpyDeviceToHost,
                           m.st);
    double *hp = histories ? histories[I.idx] : nullptr;
    if (!hp) continue;
    const uint32_t cap = ps[I.idx].max_iterations;
    for (int c = 0; c < I.C && ce == cudaSuccess; ++c) {
      const std::vector<double> &h = hist[I.unit0 + c];
      const size_t n = std::min<size_t>(h.size(), cap);
      if (!n) continue;
      ce = cudaMemcpyAsync(hp + (size_t)c * cap, h.data(), n * 8,
                           I.dev ? cudaMemcpyHostToDevice : cudaMemcpyHostToHost, m.st);
    }
  }
  if (ce == cudaSuccess) ce = cudaEventRecord(ctx->ev[3], m.st);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(m.st);
  if (ce != cudaSuccess) return mfail(ctx, PT_LAUNCH_FAILED, std::string("result download: ") + cudaGetErrorString(ce));
  {
    float a = 0.f, b = 0.f;
    if (cudaEventElapsedTime(&a, ctx->ev[1], ctx->ev[2]) != cudaSuccess) a = -1.f;
    if (cudaEventElapsedTime(&b, ctx->ev[0], ctx->ev[3]) != cudaSuccess) b = -1.f;
    cudaGetLastError();
    solve_ms += a;
    call_ms += b;
    launches += m.launches;
  }
  for (const Inst &I : m.in) {
    pt_report *reps = reports[I.idx];
    const pt_problem &p = ps[I.idx];
    int worst = -1;
    for (int c = 0; c < I.C; ++c) {
      const int un = I.unit0 + c;
      pt_report rep{};
      rep.iterations = (uint32_t)its[un];
      rep.stop_reason = stop[un];
      rep.converged = stop[un] == PT_STOP_CONVERGED;
      rep.tolerance = p.tolerance;
      rep.final_residual = r0[un] == 0.0 ? cur[un] : cur[un] / r0[un];
      rep.history_len = (uint32_t)std::min<size_t>(hist[un].size(), p.max_iterations);
      rep.omega_used = kSmoothOmega;
      rep.refinements = (uint32_t)refines[un];
      rep.channel = c;
      rep.initial_residual = r0[un];
      rep.warm_start = warm_used[un];
      reps[c] = rep;
      // worse_of (poisson_blend.rs:240-246)
      if (worst < 0) worst = c;
      else {
        const pt_report &a = reps[worst];
        const bool b_worse = (rep.iterations != a.iterations) ? (rep.iterations > a.iterations)
                                                              : (rep.final_residual > a.final_residual);
        if (b_worse) worst = c;
      }
    }
    reps[I.C] = reps[worst];
  }
  return PT_OK;
}

}  // namespace

// Problems with PT_FLAG_MULTIGRID (pt_poisson_solve, pt_poisson_solve_batch):
// all of a call's instances share each launch, in groups of at most
// kGroupTiles level-0 tiles.
pt_status ptk_solve_mg_batch(pt_ctx *ctx, const pt_problem *ps, uint32_t n, float *const *outs,
                             pt_report *const *reports, double *const *histories) {
  std::lock_guard<std::mutex> lock(ctx->mu);
  cudaError_t ce = cudaSetDevice(ctx->device);
  if (ce != cudaSuccess) return mfail(ctx, PT_NO_DEVICE, cudaGetErrorString(ce));
  for (auto &e : ctx->ev)
    if (!e && cudaEventCreate(&e) != cudaSuccess) return mfail(ctx, PT_LAUNCH_FAILED, "event create");
  double solve_ms = 0.0, call_ms = 0.0;
  long long launches = 0, tiles = 0, units = 0;
  bool ran = false;
  std::vector<int> ids;
  auto flush = [&]() -> pt_status {
    if (ids.empty()) return PT_OK;
    const pt_status s = solve_group(ctx, ps, ids, outs, reports, histories, solve_ms, call_ms, launches);
    ids.clear();
    tiles = units = 0;
    ran = true;
    return s;
  };
  for (uint32_t i = 0; i < n; ++i) {
    const pt_problem &p = ps[i];
    if (p.channels == 0) {
      pt_report r{};
      r.converged = 1; r.stop_reason = PT_STOP_CONVERGED; r.tolerance = p.tolerance; r.channel = -1;
      reports[i][0] = r;
      continue;
    }
    const long long t = bands((int)p.width, (int)p.height);
    if (!ids.empty() && (tiles + t > kGroupTiles || units + p.channels > kGroupTiles)) {
      const pt_status s = flush();
      if (s != PT_OK) return s;
    }
    ids.push_back((int)i);
    tiles += t;
    units += p.channels;
  }
  const pt_status s = flush();
  if (s != PT_OK) return s;
  if (ran) {
    ctx->last_solve_ms = solve_ms;
    ctx->last_call_ms = call_ms;
    ctx->last_launches = launches;
    ctx->last_h2d = ctx->last_d2h = 0;  // not counted on this path
  }
  return PT_OK;
}
