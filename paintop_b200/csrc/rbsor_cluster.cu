// rbsor_cluster.cu -- the whole SOR solve of a region that fits one
// thread-block cluster (sm_100a).
//
// k_solve (rbsor_kernels.cu) streams tiles through shared memory: every step
// of S sweeps claims a tile, loads it with its halo, stores it, and meets the
// system's other tiles at an arrival counter. For a region of a few tiles that
// is a chain of global-memory round trips a step, with most of the GPU idle.
// Here a system's region stays on the chip from its first sweep to its last: a
// cluster of n blocks holds the bounding box of its interior cells, a band of
// rows each. A thread owns a patch of 8 columns x R rows (both colours) whose
// correction lives in its registers, and the right-hand side of two-row patches
// too (four-row ones keep it in shared memory of their own); otherwise shared
// memory carries only what other threads read, a patch's first and last rows and
// one value a row for the patch beside it. A band's first and last rows also go into the
// neighbour block's shared memory, by stores that count their bytes off a
// barrier there (st.async): a block waits for its two neighbours' rows, not for
// the cluster, and nobody for a fence. No cell is swept twice (there are no
// overlapped halos).
//
// One warp a block keeps the books: it adds up the block's sums of squares,
// exchanges them with the other blocks, and takes the system's state machine
// forward, while the other warps already run the next block of sweeps. They
// learn the decision on a block one block later; when it is not to carry on
// (rare: a residual correction, or the end), the block begun meanwhile is void
// and they go back to where it started, which every thread has stored.
//
// The arithmetic of every cell and residual is k_solve's, operand for operand,
// and so is the state machine (step_state): blocks of S sweeps, the residual
// correction at the same sweeps, the same stop rule. The FP64 sums of squares
// are taken in this kernel's own fixed order.
//
// Bound by: the latency of a half-sweep's instructions and, with many patches
// an SM, the FP32 -> FP64 conversions of the FP64 residual (their unit takes 16
// a cycle and SM; a patch of four rows needs 60 for 16 cells, where separate
// groups of four need 21 for four). Every block of a cluster takes the same
// steps, decided from the same sums by the same code; every wait for another
// warp's or block's data is bounded (bar_wait). The wall budget is tested by
// the first block once a step and passed on with its sums; it counts from the
// call's start (call_start), for clusters that run one after another and for
// k_solve after them alike.
#include "rbsor.cuh"
#include "rbsor_device.cuh"
#include "rbsor_launch.h"

#include <algorithm>
#include <climits>

namespace ptk {

namespace {

constexpr int kMaxS = 4;       // sweeps per step of any tile configuration
constexpr int kSlot = kMaxS + 1;

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// Every thread of every block of the cluster that has not returned.
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ unsigned remote(unsigned smem_addr, unsigned rank) {
  unsigned a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr), "r"(rank));
  return a;
}
__device__ __forceinline__ void st_remote(unsigned addr, const float4 &v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}
// Stores that count their bytes off a barrier beside their destination, so that
// the reader waits for exactly these and nobody for a fence.
__device__ __forceinline__ void st_async(unsigned addr, const float4 &v, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
               "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async(unsigned addr, double v, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(addr), "d"(v), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void bar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bar_arrive(unsigned bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// The same, ordering the thread's (and, after a __syncwarp, its warp's) stores
// before what other blocks do after they have seen it.
__device__ __forceinline__ void bar_arrive_cluster(unsigned bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool bar_try(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Wait for a barrier's phase, at most P.wait_ns (the clock is read every 4096
// tries); a block whose wait gave up raises the kernel's error word, the call's
// word of that and its own flag and waits no more, and others give up on the
// call's word, or on the block.
__device__ __forceinline__ void bar_wait(unsigned bar, unsigned parity, volatile int *gave_up, const KParams &P) {
  unsigned long long t0 = 0;
  for (unsigned k = 1; !bar_try(bar, parity); ++k) {
    if (k & 4095u) continue;
    if (*gave_up) return;
    const unsigned long long now = gtimer();
    if (!t0) t0 = now;
    if (*reinterpret_cast<volatile unsigned *>(P.bar + kBarGaveUp) != 0 || now - t0 > P.wait_ns) {
      *gave_up = 1;
      atomicCAS(P.err, 0, KERR_STALLED);
      atomicExch(P.bar + kBarGaveUp, 1u);
      return;
    }
  }
}

// The end of every thread: the only hardware barrier of the cluster after the
// first, so that it pairs with nothing else wherever a block gave up, and nobody
// leaves while another block may still store into its shared memory. After a wait
// gave up asynchronous stores may be under way that nobody waited for: every block
// stays for kSettleNs more, a thousand times what one takes.
constexpr unsigned long long kSettleNs = 1000000ull;
__device__ __forceinline__ void leave(const KParams &P) {
  cluster_sync();
  if (*reinterpret_cast<volatile unsigned *>(P.bar + kBarGaveUp) == 0) return;
  const unsigned long long t0 = gtimer();
  while (gtimer() - t0 < kSettleNs) __nanosleep(1000);
}

__device__ __forceinline__ double residual(float l, float r, float u, float dn, float e, float g, double dd) {
  const double ns = (((double)l + (double)r) + (double)u) + (double)dn;
  return fma(-dd, (double)e, ns) - (double)g;
}

// A patch's state in registers: e (and g) by colour and row, four cells each;
// bit 16 h + 4 r + i of fl: cell i of colour h in row r is interior.
template <int R>
struct Patch {
  float4 e[2][R];
  float4 g[R == 2 ? 2 : 1][R == 2 ? 2 : 1];  // two-row patches: the right-hand side
  uint32_t fl;
  unsigned ag;                               // four-row ones: its address in shared memory (rhs_row)
};

// The shared-memory windows of a block. TOP(h, j), BOT(h, j): colour h of the
// first and last rows of the patches; patch row j's first row is at TOP j, its
// last at BOT j + 1; BOT 0 and TOP m are the neighbour blocks'. RIGHT(h, j, v):
// the values of patch (j, v) that the patch to its right reads (the last of
// each row whose cells sit one column right), LEFT the ones for its left.
// (As shared-memory addresses, ROWS and EDGES bytes apart by colour.)
template <int T>
struct Windows {
  static constexpr int ROWS = win_rows(T), EDGES = win_edges(T);
  static constexpr int TOP = 0, BOT = 2 * ROWS, RIGHT = 4 * ROWS, LEFT = 4 * ROWS + 2 * EDGES, G = 4 * ROWS + 4 * EDGES;
};

__device__ __forceinline__ void st_win(unsigned a, const float4 &v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void st_win(unsigned a, const float2 &v) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ float4 ld_rows(unsigned a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float2 ld_edge(unsigned a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}

// What a half-sweep reads of the other colour beside the patch's own rows: the
// rows above and below, and one value a row of the patches beside.
struct Near {
  float4 up, dn;
  float2 lf, rt;
};

// The left and right neighbours of a row's four cells: l = n[0..3], r = n[1..4].
// Every row's parity is static: the box starts on an even row.
template <int H, int R>
__device__ __forceinline__ void row_neighbours(const Patch<R> &p, const Near &b, int r, float (&n)[5]) {
  const float4 ct = p.e[1 - H][r];
  if ((H + r) & 1) {  // the row's cells of this colour sit one column right of the other's
    n[0] = ct.x; n[1] = ct.y; n[2] = ct.z; n[3] = ct.w; n[4] = r < 2 ? b.rt.x : b.rt.y;
  } else {
    n[0] = r < 2 ? b.lf.x : b.lf.y; n[1] = ct.x; n[2] = ct.y; n[3] = ct.z; n[4] = ct.w;
  }
}

// Row r of colour H's right-hand side; in shared memory a warp's groups of four
// lie side by side.
template <int H, int T, int R>
__device__ __forceinline__ float4 rhs_row(const Patch<R> &p, int r) {
  if constexpr (R == 2) return p.g[H][r];
  else return ld_rows(p.ag + (unsigned)((H * R + r) * 16 * T));
}

// One half-sweep of colour H over the thread's patch. FULL: every cell of the
// warp's patches is interior, and no flag is tested.
template <int H, bool FULL, int T, int R>
__device__ __forceinline__ void relax(Patch<R> &p, const Near &b, float w, float inv) {
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float4 up = r == 0 ? b.up : p.e[1 - H][r - 1], dn = r == R - 1 ? b.dn : p.e[1 - H][r + 1];
    float n[5];
    row_neighbours<H>(p, b, r, n);
    const float4 g = rhs_row<H, T>(p, r), e = p.e[H][r];
    const uint32_t f = p.fl >> (16 * H + 4 * r);
    float4 ne = e;
    if (FULL || (f & 1u)) ne.x = fmaf(w, ((((n[0] + n[1]) + up.x) + dn.x) - g.x) * inv - e.x, e.x);
    if (FULL || (f & 2u)) ne.y = fmaf(w, ((((n[1] + n[2]) + up.y) + dn.y) - g.y) * inv - e.y, e.y);
    if (FULL || (f & 4u)) ne.z = fmaf(w, ((((n[2] + n[3]) + up.z) + dn.z) - g.z) * inv - e.z, e.z);
    if (FULL || (f & 8u)) ne.w = fmaf(w, ((((n[3] + n[4]) + up.w) + dn.w) - g.w) * inv - e.w, e.w);
    p.e[H][r] = ne;
  }
}

// The sum of squares of the FP64 residual at colour H's interior cells, whose
// values are e[].
template <int H, bool FULL, int T, int R>
__device__ __forceinline__ double squares(const Patch<R> &p, const float4 (&e)[R], const Near &b, double dd) {
  double part = 0.0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float4 up = r == 0 ? b.up : p.e[1 - H][r - 1], dn = r == R - 1 ? b.dn : p.e[1 - H][r + 1];
    float n[5];
    row_neighbours<H>(p, b, r, n);
    const float4 g = rhs_row<H, T>(p, r);
    const uint32_t f = p.fl >> (16 * H + 4 * r);
    const double x0 = residual(n[0], n[1], up.x, dn.x, e[r].x, g.x, dd), x1 = residual(n[1], n[2], up.y, dn.y, e[r].y, g.y, dd),
                 x2 = residual(n[2], n[3], up.z, dn.z, e[r].z, g.z, dd), x3 = residual(n[3], n[4], up.w, dn.w, e[r].w, g.w, dd);
    if (FULL || (f & 1u)) part = fma(x0, x0, part);
    if (FULL || (f & 2u)) part = fma(x1, x1, part);
    if (FULL || (f & 4u)) part = fma(x2, x2, part);
    if (FULL || (f & 8u)) part = fma(x3, x3, part);
  }
  return part;
}

// What colour H's cells of the patch show their neighbours: of each row the
// last value (rows whose cells sit one column right) or the first.
template <int R, int H>
__device__ __forceinline__ void edges(const Patch<R> &p, float2 &right, float2 &left) {
  constexpr int A = 1 - H, B = H;  // the first row that shows its last value, its first value
  right = make_float2(p.e[H][A].w, R == 4 ? p.e[H][(A + 2) % R].w : 0.f);
  left = make_float2(p.e[H][B].x, R == 4 ? p.e[H][(B + 2) % R].x : 0.f);
}

// A block's shared variables. bars: the rows of colours 0, 1 from the block
// above (0, 1) and below (2, 3); the cluster's sums, by the exchange's parity
// (4, 5); the warps' meetings (6); the block's sums and the decisions, by the
// step's parity (7, 8 and 9, 10); the cluster's meetings: the block's warps have
// come (11), all blocks' have, by the meeting's parity (12, 13).
enum Bar { B_UP = 0, B_DN = 2, B_SLOT = 4, B_MEET = 6, B_SUMS = 7, B_DECIDED = 9, B_HERE = 11, B_ALL = 12, B_COUNT = 14 };
struct Shared {
  SysDesc d;
  SysState st;
  unsigned long long bars[B_COUNT];
  double slot[2][kClusterMax][kSlot];
  double sums[2][kMaxS][kClusterMost / 32];
  int mode[2], s[2];  // the decisions
  int gave_up;
};

// The number of sweeps of the block after one of s sweeps that ends at
// iteration `it`, if the solve carries on.
__device__ __forceinline__ int next_block(const KParams &P, const Shared &sh, int it) {
  return min(P.S, sh.d.max_it - it);
}

// The warp that keeps the books.
__device__ __forceinline__ void keep_books(const KParams &P, Shared &sh, unsigned bar0, const int n, const int nwa,
                                           const unsigned rank) {
  const int lane = threadIdx.x & 31;
  const unsigned long long t_start = *call_start(P);
  const unsigned slot0 = (unsigned)__cvta_generic_to_shared(&sh.slot[0][rank][0]);
  int mode = sh.st.mode, s = sh.st.s, it = 0;
  unsigned x = 0, dc = 0, meets = 0;  // exchanges, decisions and cluster meetings so far
  auto cluster_meet = [&]() {  // the block's warps have come: tell every block
    bar_wait(bar0 + 8u * B_HERE, meets & 1u, &sh.gave_up, P);
    __syncwarp();
    if (lane < n) bar_arrive_cluster(remote(bar0 + 8u * (B_ALL + (meets & 1u)), lane));
    ++meets;
  };
  for (unsigned t = 0; mode != M_DONE; ++t) {
    if (mode != M_SWEEP) {  // a re-run's start, or the fold: before and after the other warps show it
      cluster_meet();
      cluster_meet();
    }
    bar_wait(bar0 + 8u * (B_SUMS + (t & 1u)), (t >> 1) & 1u, &sh.gave_up, P);
    const int nsum = mode == M_SWEEP ? s : (mode == M_FOLD ? 1 : 0);  // (a fold step ends with the new residual)
    double nrm[kMaxS], rel[kMaxS];
    bool late = false;
    if (nsum) {
      const unsigned to = slot0 + (x & 1u) * (unsigned)sizeof(sh.slot[0]), bar = bar0 + 8u * (B_SLOT + (x & 1u));
      double mine[kMaxS];
#pragma unroll
      for (int j = 0; j < kMaxS; ++j) mine[j] = lane < nwa && j < nsum ? sh.sums[t & 1u][j][lane] : 0.0;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1)
#pragma unroll
        for (int j = 0; j < kMaxS; ++j) mine[j] += __shfl_xor_sync(0xffffffffu, mine[j], o);
      if (lane < n && !(P.silent && (int)rank == n - 1)) {
        const unsigned rto = remote(to, lane), rbar = remote(bar, lane);
#pragma unroll
        for (int j = 0; j < kMaxS; ++j)
          if (j < nsum) st_async(rto + 8u * (unsigned)j, mine[j], rbar);
        if (rank == 0)
          st_async(rto + 8u * kMaxS, ld_vol(P.err) != 0 || over_budget(P, t_start) ? 1.0 : 0.0, rbar);
      }
      if (lane == 0) bar_expect(bar, 8u * (unsigned)(n * nsum + 1));
      __syncwarp();
      bar_wait(bar, (x >> 1) & 1u, &sh.gave_up, P);
      __syncwarp();
#pragma unroll
      for (int j = 0; j < kMaxS; ++j) mine[j] = lane < n && j < nsum ? sh.slot[x & 1u][lane][j] : 0.0;
      late = sh.gave_up || sh.slot[x & 1u][0][kMaxS] != 0.0;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1)
#pragma unroll
        for (int j = 0; j < kMaxS; ++j) mine[j] += __shfl_xor_sync(0xffffffffu, mine[j], o);
      // the norms and their ratios to r0, one a lane at once
      double v = mine[0];
#pragma unroll
      for (int j = 1; j < kMaxS; ++j) v = lane == j ? mine[j] : v;
      v = sqrt(v);
      const double q = v / sh.st.r0;
#pragma unroll
      for (int j = 0; j < kMaxS; ++j) {
        nrm[j] = __shfl_sync(0xffffffffu, v, j);
        rel[j] = __shfl_sync(0xffffffffu, q, j);
      }
      ++x;
    }
    __syncwarp();
    if (lane == 0) {
      double *hist = rank == 0 ? P.hist + sh.d.hist_off : nullptr;
      if (late) {
        if (rank == 0) atomicCAS(P.err, 0, KERR_DEADLINE);
        sh.st.mode = M_DONE;
        sh.st.status = -1;
      } else {
        step_state(sh.d, sh.st, mode, nrm, rel, hist, P.S);
        if (mode == M_FOLD) step_state(sh.d, sh.st, M_RESID, nrm, rel, hist, P.S);
      }
      sh.mode[dc & 1u] = sh.st.mode;
      sh.s[dc & 1u] = sh.st.s;
      bar_arrive(bar0 + 8u * (B_DECIDED + (dc & 1u)));
    }
    __syncwarp();
    ++dc;
    const int next = sh.st.mode;
    if (mode == M_SWEEP) {
      it += s;
      if (next != M_SWEEP && next != M_DONE && next_block(P, sh, it) > 0) {
        ++t;  // the block of sweeps begun meanwhile is void
        bar_wait(bar0 + 8u * (B_SUMS + (t & 1u)), (t >> 1) & 1u, &sh.gave_up, P);
      }
    }
    it = sh.st.iterations;
    mode = next;
    s = sh.st.s;
    __syncwarp();
  }
}

template <int R, int T>
__device__ __forceinline__ void solve_region(const KParams &P, const Route &rt, Shared &sh, const int sys,
                                             const unsigned rank, const int TW, const int TH, unsigned char *smem) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n = rt.n, nq = rt.nq, m = rt.m;
  const int jr = tid / nq, v = tid - jr * nq;             // the thread's patch
  const int j0 = (int)rank * m, mr = min(m, rt.bm - j0);  // the block's patch rows
  const int nwa = (mr * nq + 31) / 32;                    // its warps that hold patches
  const bool books = warp == (int)(blockDim.x >> 5) - 1, mine = !books && jr < mr;
  const int py = rt.y0 + (j0 + jr) * R, gi = (rt.x0 >> 1) + 4 * v;  // its first row, its plane index
  const bool to_up = mine && jr == 0 && rank > 0, to_dn = mine && jr == mr - 1 && (int)rank + 1 < n;

  for (int k = tid; k < win_bytes(T) / 4; k += blockDim.x) reinterpret_cast<float *>(smem)[k] = 0.0f;
  const unsigned bar0 = (unsigned)__cvta_generic_to_shared(sh.bars);
  const unsigned row_bytes = 16u * (unsigned)nq;
  if (tid == 0) {
    sh.d = P.sys[sys];
    sh.st = load_sys_state(P.st + sys);
    sh.gave_up = 0;
    for (int k = 0; k < B_COUNT; ++k)
      bar_init(bar0 + 8u * k, k == B_MEET || k == B_SUMS || k == B_SUMS + 1 || k == B_HERE ? (unsigned)nwa
                              : k == B_ALL || k == B_ALL + 1                              ? (unsigned)n
                                                                                          : 1u);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int k = 0; k < 2; ++k) {
      if (rank > 0) bar_expect(bar0 + 8u * (B_UP + k), row_bytes);
      if ((int)rank + 1 < n) bar_expect(bar0 + 8u * (B_DN + k), row_bytes);
    }
  }
  __syncthreads();
  const SysDesc &d = sh.d;
  const long long at = d.off + (long long)py * d.pw + gi;  // the patch in plane 0 of the cell pools
  auto pool = [&](int h, int r) { return at + (long long)h * d.plane + (long long)r * d.pw; };

  // ---- the patch: interior flags and the right-hand side; e = 0. Tiles
  // without interior cells were not assembled: their cells are not interior.
  using W = Windows<T>;
  Patch<R> p;
  p.fl = 0;
  p.ag = (unsigned)__cvta_generic_to_shared(smem) + W::G + 16u * (unsigned)min(tid, T - 1);
  auto set_rhs = [&](int h, int r, const float4 &v) {
    if constexpr (R == 2) p.g[h][r] = v;
    else if (!books) st_win(p.ag + (unsigned)((h * R + r) * 16 * T), v);
  };
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
      p.e[h][r] = z;
      float4 g = z;
      const int y = py + r;
      if (mine && y < d.H && gi < d.pw && P.tcount[d.tile0 + (y / TH) * d.ntx + (2 * gi) / TW] > 0) {
        const uint32_t c = *reinterpret_cast<const uint32_t *>(P.cell + pool(h, r));
        const uint32_t f = (c & 1u) | ((c >> 7) & 2u) | ((c >> 14) & 4u) | ((c >> 21) & 8u);
        p.fl |= f << (16 * h + 4 * r);
        if (f) g = __ldcg(reinterpret_cast<const float4 *>(P.g + pool(h, r)));
      }
      set_rhs(h, r, g);
    }
  cluster_sync();  // every block's windows are zeroed and its barriers set before a neighbour stores
  if (books) {
    keep_books(P, sh, bar0, n, nwa, rank);
    if (rank == 0 && lane == 0) P.st[sys] = sh.st;
    leave(P);
    return;
  }
  if (warp >= nwa) return;  // (the cluster's barriers count the threads that stay)

  const unsigned base = (unsigned)__cvta_generic_to_shared(smem);
  const unsigned bars_up = to_up ? remote(bar0, rank - 1) : 0u, bars_dn = to_dn ? remote(bar0, rank + 1) : 0u;
  // the patch in the windows: its rows; its edges (rows of nq + 2, a zero
  // column either side); the neighbour blocks' halo rows: the block above has m
  // full rows of patches, the one below starts at 0
  const unsigned aw = base + 16u * (unsigned)(jr * nq + v), ae = base + 8u * (unsigned)(jr * (nq + 2) + v + 1);
  const unsigned below = 16u * (unsigned)nq;
  const unsigned to_top = to_up ? remote(base, rank - 1) + 16u * (unsigned)(m * nq + v) : 0u;
  const unsigned to_bot = to_dn ? remote(base, rank + 1) + 16u * (unsigned)v : 0u;
  // what the neighbours read of colour h (a constant after inlining); async:
  // the rows for other blocks count off their barriers (in a half-sweep; else
  // the blocks meet before and after)
  auto show = [&](int h, bool async) {
    const float4 a = p.e[h][0], b = p.e[h][R - 1];
    float2 right, left;
    if (h) edges<R, 1>(p, right, left);
    else edges<R, 0>(p, right, left);
    st_win(aw + W::TOP + h * W::ROWS, a);
    st_win(aw + below + W::BOT + h * W::ROWS, b);
    st_win(ae + W::RIGHT + h * W::EDGES, right);
    st_win(ae + W::LEFT + h * W::EDGES, left);
    if (to_up) {
      if (async) st_async(to_top + W::TOP + h * W::ROWS, a, bars_up + 8u * (B_DN + h));
      else st_remote(to_top + W::TOP + h * W::ROWS, a);
    }
    if (to_dn) {
      if (async) st_async(to_bot + W::BOT + h * W::ROWS, b, bars_dn + 8u * (B_UP + h));
      else st_remote(to_bot + W::BOT + h * W::ROWS, b);
    }
  };
  // bit h: the parity of colour h's rows; bit 2: of the meetings; bits 3, 4: of
  // the even and odd decisions; from bit 5 on: cluster meetings so far
  unsigned phase = 0;
  // the other blocks' rows of colour h, by the threads that read them; the
  // first of a row arms the barrier's next phase
  auto wait_rows = [&](int h) {
    const unsigned par = (phase >> h) & 1u;
    if (to_up) {
      bar_wait(bar0 + 8u * (B_UP + h), par, &sh.gave_up, P);
      if (v == 0) bar_expect(bar0 + 8u * (B_UP + h), row_bytes);
    }
    if (to_dn) {
      bar_wait(bar0 + 8u * (B_DN + h), par, &sh.gave_up, P);
      if (v == 0) bar_expect(bar0 + 8u * (B_DN + h), row_bytes);
    }
    phase ^= 1u << h;
  };
  // the warps meet after each half-sweep, arriving before the residual and
  // waiting after it
  auto arrive = [&](int bar) {
    __syncwarp();
    if (lane == 0) bar_arrive(bar0 + 8u * bar);
  };
  auto meet_wait = [&]() {
    bar_wait(bar0 + 8u * B_MEET, (phase >> 2) & 1u, &sh.gave_up, P);
    phase ^= 4u;
  };
  // All blocks' warps meet, around rows shown by plain stores. Before them, since
  // an asynchronous store of an earlier half-sweep to the same row may still be on
  // its way: its sender waits for its neighbours' rows, never for its own to
  // arrive, and a later plain store of the same thread is not ordered behind it.
  // Every block has waited for all rows sent to it when it comes here. And after
  // them, before the rows are read. Two barriers in turn: a block comes to the
  // meeting after next only when all have passed this one.
  auto cluster_meet = [&]() {
    __syncwarp();
    if (lane == 0) bar_arrive_cluster(bar0 + 8u * B_HERE);
    bar_wait(bar0 + 8u * (B_ALL + ((phase >> 5) & 1u)), (phase >> 6) & 1u, &sh.gave_up, P);
    phase += 32u;
  };
  auto near = [&](int o) {
    return Near{ld_rows(aw + W::BOT + o * W::ROWS), ld_rows(aw + below + W::TOP + o * W::ROWS),
                ld_edge(ae - 8 + W::RIGHT + o * W::EDGES), ld_edge(ae + 8 + W::LEFT + o * W::EDGES)};
  };

  const float w = d.omega, inv = d.inv_denom;
  const double dd = 4.0 + d.lambda;
  const bool red_any = (p.fl & 0xffffu) != 0, black_any = (p.fl >> 16) != 0;
  const bool full = __all_sync(0xffffffffu, p.fl == (R == 4 ? 0xffffffffu : 0x00ff00ffu));
  // a block of sweeps' start, stored by the step's parity and taken back
  auto store = [&](unsigned t) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int r = 0; r < R; ++r)
        if ((p.fl >> (16 * h + 4 * r)) & 15u)
          __stcg(reinterpret_cast<float4 *>((t & 1u ? P.e1 : P.e0) + pool(h, r)), p.e[h][r]);
  };
  auto restore = [&](unsigned t) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int r = 0; r < R; ++r)
        if ((p.fl >> (16 * h + 4 * r)) & 15u)
          p.e[h][r] = __ldcg(reinterpret_cast<const float4 *>((t & 1u ? P.e1 : P.e0) + pool(h, r)));
  };
  // s sweeps; the sums of squares after each of them. Half-sweeps: wait for
  // the other colour's rows, relax, show the result, arrive; the residual's
  // sum of squares follows while the others catch up (it is the longer part),
  // from values the thread already holds.
  // (a warp's sum goes to the books as soon as it is known.)
  auto give = [&](unsigned t, int j, double x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) sh.sums[t & 1u][j][warp] = x;
  };
  auto sweeps = [&](const unsigned t, const int s, const bool redo) {
    double carry = 0.0;  // black's sum of the state before
#pragma unroll 1
    for (int j = 0; j <= s; ++j) {
      const bool last = j == s;
      Near b{};
      if (j > 0) {
        meet_wait();
        wait_rows(1);
      }
      if (last && redo) break;
      if (red_any) b = near(1);
      float4 old[R];
#pragma unroll
      for (int r = 0; r < R; ++r) old[r] = p.e[0][r];
      if (!last) {
        if (full) relax<0, true, T>(p, b, w, inv);
        else if (red_any) relax<0, false, T>(p, b, w, inv);
        if (mine) show(0, true);
        arrive(B_MEET);
      }
      if (j > 0) {
        if (full) carry += squares<0, true, T>(p, old, b, dd);
        else if (red_any) carry += squares<0, false, T>(p, old, b, dd);
        give(t, j - 1, carry);
      }
      if (last) break;
      meet_wait();
      wait_rows(0);
      carry = 0.0;
      if (black_any) b = near(0);
      if (full) relax<1, true, T>(p, b, w, inv);
      else if (black_any) relax<1, false, T>(p, b, w, inv);
      if (mine) show(1, true);
      arrive(B_MEET);
      if (full) carry = squares<1, true, T>(p, p.e[1], b, dd);
      else if (black_any) carry = squares<1, false, T>(p, p.e[1], b, dd);
    }
    arrive(B_SUMS + (int)(t & 1u));
  };
  unsigned dc = 0;  // decisions taken note of
  int mode = sh.st.mode, s = sh.st.s;
  auto decision = [&]() {
    const unsigned k = dc & 1u;
    bar_wait(bar0 + 8u * (B_DECIDED + k), (phase >> (3 + k)) & 1u, &sh.gave_up, P);
    phase ^= 8u << k;
    ++dc;
    if (sh.gave_up) { mode = M_DONE; return; }
    mode = sh.mode[k];
    s = sh.s[k];
  };

  int it = 0;      // sweeps that count so far
  unsigned t = 0;  // the step
  while (mode != M_DONE) {
    if (mode == M_SWEEP) {
      // blocks of sweeps, each begun before the decision on the one before
      store(t);
      sweeps(t, s, false);
      it += s;
      for (;;) {
        const int ahead = next_block(P, sh, it);
        if (ahead > 0) {
          store(t + 1);
          sweeps(t + 1, ahead, false);
        }
        decision();  // on step t
        if (mode != M_SWEEP) {
          if (mode == M_FOLD && ahead > 0) restore(t + 1);  // step t's end
          if (mode == M_REDO) restore(t);
          t += ahead > 0 ? 2u : 1u;
          break;
        }
        ++t;
        it += ahead;
      }
    } else if (mode == M_REDO) {  // step t - 1 or t - 2 again from its start, with fewer sweeps
      cluster_meet();
      if (mine) {
        show(0, false);
        show(1, false);
      }
      cluster_meet();
      sweeps(t++, s, true);
      decision();
    } else {  // M_FOLD: u += e on interior cells, e = 0; then g = -r(u), r in FP64 exactly as residual_l2 (poisson.rs:315-321)
      cluster_meet();
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const uint32_t f = (p.fl >> (16 * h + 4 * r)) & 15u;
          if (!f) continue;
          const float4 e = p.e[h][r];
          double2 *u = reinterpret_cast<double2 *>(P.u + pool(h, r));
          double2 a = __ldcg(u), b = __ldcg(u + 1);
          if (f & 1u) a.x += (double)e.x;
          if (f & 2u) a.y += (double)e.y;
          if (f & 4u) b.x += (double)e.z;
          if (f & 8u) b.y += (double)e.w;
          u[0] = a;
          u[1] = b;
          p.e[h][r] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
      if (mine) {
        show(0, false);
        show(1, false);
      }
      __threadfence();
      cluster_meet();
      const double lam4 = d.lambda + 4.0;
      double a = 0.0;
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const uint32_t f = (p.fl >> (16 * h + 4 * r)) & 15u;
          if (!f) continue;
          const long long o = pool(h, r), oo = pool(1 - h, r);
          const int q = (h + r) & 1;
          float g[4] = {0.f, 0.f, 0.f, 0.f};  // (a cell that is not interior: not read)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (!(f & (1u << i))) continue;
            const double L = __ldcg(P.u + oo + i - 1 + q), Rr = __ldcg(P.u + oo + i + q);
            const double U = __ldcg(P.u + oo + i - d.pw), D = __ldcg(P.u + oo + i + d.pw);
            const double res = fma(lam4, -__ldcg(P.u + o + i), ((L + Rr) + U) + D) - __ldg(P.bp + o + i);
            g[i] = (float)(-res);
            a = fma(res, res, a);
          }
          set_rhs(h, r, make_float4(g[0], g[1], g[2], g[3]));
        }
      give(t, 0, a);
      arrive(B_SUMS + (int)(t & 1u));
      ++t;
      decision();
      it = sh.st.iterations;
    }
  }
  leave(P);
}

}  // namespace

// A class of systems whose regions may take patches of two rows, or of four;
// each launch's blocks take theirs.
template <int R, int T>
__global__ void __launch_bounds__(T + 32, T == kClusterLeast ? 2 : 1) k_cluster_solve(KParams P,
                                                                                     const int *__restrict__ list,
                                                                                     int TW, int TH) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ Shared sh;
  const unsigned rank = cluster_rank();
  const int sys = list[blockIdx.x / cluster_size()];
  const Route rt = P.route[sys];
  if ((int)rank >= rt.n || rt.rows != R) return;  // (the cluster's barriers count the threads that stay)
  solve_region<R, T>(P, rt, sh, sys, rank, TW, TH, smem);
}

namespace {
// f(kernel, rows, limit) for each instance, until one fails
template <class F>
cudaError_t each_instance(F f) {
  cudaError_t e = f(k_cluster_solve<2, kClusterLeast>, 2, kClusterLeast);
  if (e == cudaSuccess) e = f(k_cluster_solve<4, kClusterLeast>, 4, kClusterLeast);
  if (e == cudaSuccess) e = f(k_cluster_solve<2, kClusterMost>, 2, kClusterMost);
  if (e == cudaSuccess) e = f(k_cluster_solve<4, kClusterMost>, 4, kClusterMost);
  return e;
}

// The launch of `count` clusters of `blocks` blocks; `at` is its storage.
cudaLaunchConfig_t cluster_config(int limit, int blocks, int count, int smem, cudaStream_t stream,
                                  cudaLaunchAttribute *at) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)count * (unsigned)blocks);
  cfg.blockDim = dim3((unsigned)limit + 32u);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = (unsigned)blocks;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}
}  // namespace

cudaError_t prepare_cluster(int *room) {
  static_assert(kClusterAlone >= cluster_smem(4, kClusterMost) && cluster_smem(4, kClusterLeast) <= 110 * 1024,
                "shared memory of the blocks");
  *room = INT_MAX;
  return each_instance([room](auto k, int, int limit) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kClusterAlone);
    cudaLaunchAttribute at{};
    cudaLaunchConfig_t cfg = cluster_config(limit, kClusterMax, 1, kClusterAlone, nullptr, &at);
    int fit = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&fit, k, &cfg);
    *room = std::min(*room, fit);
    return e;
  });
}

cudaError_t launch_cluster(const KParams &P, const TileConfig &tc, const ClusterClass &k, const int *list,
                           cudaStream_t stream) {
  if (k.count == 0) return cudaSuccess;
  return each_instance([&](auto kernel, int rows, int limit) {
    if (limit != k.limit || !(rows == 2 ? k.rows2 : k.rows4)) return cudaSuccess;
    cudaLaunchAttribute at{};
    const cudaLaunchConfig_t cfg =
        cluster_config(limit, k.blocks, k.count, k.alone ? kClusterAlone : cluster_smem(rows, limit), stream, &at);
    return cudaLaunchKernelEx(&cfg, kernel, P, list + k.first, tc.tw, tc.th);
  });
}

}  // namespace ptk
