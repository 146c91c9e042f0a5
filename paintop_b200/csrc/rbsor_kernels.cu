// rbsor_kernels.cu -- device kernels of the red-black SOR solver (sm_100a).
// See rbsor.cuh for the method, the HBM layout and the control scheme.
#include "rbsor.cuh"
#include "rbsor_device.cuh"
#include "rbsor_launch.h"

#include <cmath>
#include <cstdio>

namespace ptk {

// Asynchronous global -> shared copies (Ampere+ cp.async). `in == false` copies
// no bytes and zero-fills the destination.
__device__ __forceinline__ void cp_async16(void *smem_dst, const void *gmem_src, bool in) {
  const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(gmem_src),
               "r"(in ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem_dst, const void *gmem_src, bool in) {
  const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(gmem_src),
               "r"(in ? 4 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// ----------------------------------------------------------------------------
// geometry of one tile configuration
// ----------------------------------------------------------------------------
template <int S, int TH>
struct Geo {
  static constexpr int H = halo_y(S);
  static constexpr int HX = halo_x(S);
  static constexpr int TW = tile_w(S);
  static constexpr int LH = TH + 2 * H;
  static constexpr int PLANE = LH * kPWL;  // elements per shared plane
  static constexpr int XOFF = HX - H;      // unused loaded columns on each side
  // Rows 1..LH-2 in quads, two rows a half-warp, three (or two) quads a warp.
  static constexpr int QUADS = (LH - 2) / 4, NW = 8, NT = 32 * NW;
  static_assert((LH - 2) % 4 == 0 && QUADS % NW == 0, "rows 1..LH-2 must split evenly over the warps");
  static_assert(H % 2 == 1 && TH % 2 == 0, "loaded row 0 is odd, and a half-warp's two rows are owned alike");
  static_assert(HX >= H, "x halo must cover the sweep halo");
  static_assert(TW > 0 && TW % 8 == 0, "tile width must keep plane loads 16-byte aligned");
  static constexpr size_t kSmem = (size_t)2 * PLANE * sizeof(float)   // e
                                  + (size_t)2 * PLANE * sizeof(float) // g
                                  + (size_t)2 * PLANE                 // cell
                                  + NW * sizeof(double);              // reduction scratch
};

// ----------------------------------------------------------------------------
// assembly kernels
// ----------------------------------------------------------------------------
__device__ __forceinline__ bool interior_at(const SysDesc &d, int x, int y) {
  if (d.W < 3 || d.H < 3) return false;                  // poisson.rs:342-345
  if (x < 1 || y < 1 || x > d.W - 2 || y > d.H - 2) return false;
  return d.mask[(long long)y * d.W + x] > 0.5f;           // poisson.rs:349 (strict >)
}

// Interior cells per tile (owned region only) and their bounding box. min/max
// are order-independent, so the box is deterministic.
// The channels of an image share its mask, so only channel 0's blocks count;
// they store the count and box for every channel's copy of the tile.
__global__ void k_tile_count(KParams P, int TW, int TH) {
  const Tile tl = P.tiles[blockIdx.x];
  const SysDesc d = P.sys[tl.sys];
  if (d.chan != 0) return;
  __shared__ int s[32];
  __shared__ int sb[4];
  if (threadIdx.x < 4) sb[threadIdx.x] = (threadIdx.x < 2) ? 0x7fffffff : -1;
  __syncthreads();
  int n = 0, x0m = 0x7fffffff, y0m = 0x7fffffff, x1m = -1, y1m = -1;
  const int x0 = tl.tx * TW, y0 = tl.ty * TH;
  for (int k = threadIdx.x; k < TW * TH; k += blockDim.x) {
    const int x = x0 + k % TW, y = y0 + k / TW;
    if (x < d.W && y < d.H && interior_at(d, x, y)) {
      ++n;
      x0m = min(x0m, x); y0m = min(y0m, y); x1m = max(x1m, x); y1m = max(y1m, y);
    }
  }
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = n;
  if (x1m >= 0) {
    atomicMin(&sb[0], x0m); atomicMin(&sb[1], y0m); atomicMax(&sb[2], x1m); atomicMax(&sb[3], y1m);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s[w];
    const int4 box = make_int4(sb[0], sb[1], sb[2], sb[3]);
    const int local = (int)blockIdx.x - d.tile0;  // the tile's index within its system
    for (int c = 0; c < d.C; ++c) {
      const int tt = P.sys[tl.sys + c].tile0 + local;
      P.tcount[tt] = t;
      P.tbox[tt] = box;
    }
  }
}

__device__ __forceinline__ bool tile_support(const KParams &P, const SysDesc &d, int tx, int ty) {
  for (int dy = -1; dy <= 1; ++dy)
    for (int dx = -1; dx <= 1; ++dx) {
      const int x = tx + dx, y = ty + dy;
      if (x < 0 || y < 0 || x >= d.ntx || y >= d.nty) continue;
      if (P.tcount[d.tile0 + y * d.ntx + x] > 0) return true;
    }
  return false;
}

// r(anchor) at an interior pixel: (4 + lambda) a - (sum of the four anchor
// neighbours) against b' (poisson.rs:315-321), in this operand order.
__device__ __forceinline__ double anchor_residual(const SysDesc &d, long long px, double a, double bp) {
  const int C = d.C, ch = d.chan;
  const double na = (((double)d.tgt[(px - 1) * C + ch] + (double)d.tgt[(px + 1) * C + ch]) +
                     (double)d.tgt[(px - d.W) * C + ch]) + (double)d.tgt[(px + d.W) * C + ch];
  return fma(d.lambda + 4.0, -a, na) - bp;
}

// Assemble one tile of one system (owned cells only). Writes cell, bp, u, g and
// zeroes e0/e1; accumulates ||r(anchor)||^2 and ||r(u_init)||^2 partials.
// Arithmetic of b and r follows poisson.rs:364-373 (guidance_laplacian) and
// poisson.rs:315-321 (residual), operand for operand.
__global__ void __launch_bounds__(kThreads) k_assemble(KParams P, int TW, int TH) {
  __shared__ double sred[kWarps];
  // Block order: within each image, its channels' copies of a tile come one
  // after another, so the interleaved source and target pixels a tile reads
  // are still in L2 for the other channels' blocks. The tiles of an image are
  // channel 0's, then channel 1's, ...; block b of the image takes channel
  // b % C's tile b / C.
  int t = blockIdx.x;
  {
    const SysDesc &d0 = P.sys[P.tiles[t].sys];
    const int base = d0.tile0 - d0.chan * d0.ntiles;  // the image's first tile
    const int local = t - base;
    t = base + (local % d0.C) * d0.ntiles + local / d0.C;
  }
  const Tile tl = P.tiles[t];
  const SysDesc d = P.sys[tl.sys];
  if (!tile_support(P, d, tl.tx, tl.ty)) return;
  const int C = d.C, ch = d.chan;
  const double lam = d.lambda;
  double acc_a = 0.0, acc_u = 0.0;
  const int half = TW / 2;
  for (int k = threadIdx.x; k < 2 * TH * half; k += blockDim.x) {
    const int c = k / (TH * half);
    const int r = k - c * (TH * half);
    const int y = tl.ty * TH + r / half;
    const int i = tl.tx * half + r % half;
    if (y >= d.H || i >= d.pw) continue;
    const int x = 2 * i + ((c + y) & 1);
    const long long o = plane_index(d, c, y, i);
    P.e0[o] = 0.0f;
    P.e1[o] = 0.0f;
    if (x >= d.W) {  // padding column beyond the image
      P.cell[o] = 0; P.bp[o] = 0.0; P.u[o] = 0.0; P.g[o] = 0.0f;
      continue;
    }
    const long long px = (long long)y * d.W + x;
    const double a = (double)d.tgt[px * C + ch];
    if (!interior_at(d, x, y)) {
      P.cell[o] = 0; P.bp[o] = 0.0; P.u[o] = a; P.g[o] = 0.0f;
      continue;
    }
    // interior: all four neighbours are inside the image
    const long long pl = px - 1, pr = px + 1, pu = px - d.W, pd = px + d.W;
    const double sc = (double)d.src[px * C + ch];
    const double ns = (((double)d.src[pl * C + ch] + (double)d.src[pr * C + ch]) +
                       (double)d.src[pu * C + ch]) + (double)d.src[pd * C + ch];
    const double b = fma(4.0, -sc, ns);
    const double bp = fma(lam, -a, b);
    const double ra = anchor_residual(d, px, a, bp);
    acc_a = fma(ra, ra, acc_a);
    double uc = a, ru = ra;
    if (d.warm) {
      auto guess_or_anchor = [&](long long q, int qx, int qy) -> double {
        return interior_at(d, qx, qy) ? (double)d.guess[q * C + ch] : (double)d.tgt[q * C + ch];
      };
      uc = (double)d.guess[px * C + ch];
      const double nu = ((guess_or_anchor(pl, x - 1, y) + guess_or_anchor(pr, x + 1, y)) +
                         guess_or_anchor(pu, x, y - 1)) + guess_or_anchor(pd, x, y + 1);
      ru = fma(lam + 4.0, -uc, nu) - bp;
    }
    acc_u = fma(ru, ru, acc_u);
    P.cell[o] = 1;
    P.bp[o] = bp;
    P.u[o] = uc;
    P.g[o] = (float)(-ru);
  }
  acc_a = block_sum(acc_a, sred);
  acc_u = block_sum(acc_u, sred);
  if (threadIdx.x == 0) {
    P.fpart[t] = acc_a;
    P.fpart[P.ntiles + t] = acc_u;
  }
}

// ---- connected interior regions (automatic omega) --------------------------
// A union-find over the pixels of each labelled image (4-neighbour
// connectivity): every label points at itself (a root) or at a smaller index
// of the same region, so a root search walks strictly decreasing indices and
// ends; unions lower a root with atomicMin, so each retry sees a smaller
// label and ends too. The final labels are the regions' smallest pixel
// indices whatever the order of the unions, so the result is deterministic.
__device__ __forceinline__ int region_of(const KParams &P, long long gp) {
  int lo = 0, hi = P.nregions - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (P.regions[mid].lab_off <= gp) lo = mid; else hi = mid - 1;
  }
  return lo;
}
__device__ __forceinline__ int label_root(int *L, int x) {
  const volatile int *vl = L;
  const int x0 = x;
  for (int k = x; k >= 0; --k) {  // at most x + 1 steps: labels only decrease
    const int y = vl[x];
    if (y == x) break;
    x = y;
  }
  if (x != x0) atomicMin(&L[x0], x);  // shorten the chain; never raises a label
  return x;
}
__device__ void label_unite(int *L, int a, int b) {
  for (int k = a + b + 2; k > 0; --k) {  // each retry lowers a or b
    a = label_root(L, a);
    b = label_root(L, b);
    if (a == b) return;
    if (a < b) {
      const int old = atomicMin(&L[b], a);
      if (old == b) return;
      b = old;
    } else {
      const int old = atomicMin(&L[a], b);
      if (old == a) return;
      a = old;
    }
  }
}
__global__ void k_label_init(KParams P) {
  for (long long gp = blockIdx.x * (long long)blockDim.x + threadIdx.x; gp < P.rpix;
       gp += (long long)gridDim.x * blockDim.x) {
    const RegionDesc r = P.regions[region_of(P, gp)];
    const int p = (int)(gp - r.lab_off), y = p / r.W, x = p - y * r.W;
    P.label[gp] = interior_at(P.sys[r.sys0], x, y) ? p : -1;
  }
}
__global__ void k_label_link(KParams P) {
  for (long long gp = blockIdx.x * (long long)blockDim.x + threadIdx.x; gp < P.rpix;
       gp += (long long)gridDim.x * blockDim.x) {
    if (P.label[gp] < 0) continue;
    const RegionDesc r = P.regions[region_of(P, gp)];
    int *L = P.label + r.lab_off;
    const int p = (int)(gp - r.lab_off), y = p / r.W, x = p - y * r.W;
    if (x > 0 && L[p - 1] >= 0) label_unite(L, p, p - 1);
    if (y > 0 && L[p - r.W] >= 0) label_unite(L, p, p - r.W);
  }
}
__global__ void k_label_count(KParams P) {
  for (long long gp = blockIdx.x * (long long)blockDim.x + threadIdx.x; gp < P.rpix;
       gp += (long long)gridDim.x * blockDim.x) {
    if (P.label[gp] < 0) continue;
    const RegionDesc r = P.regions[region_of(P, gp)];
    const int root = label_root(P.label + r.lab_off, (int)(gp - r.lab_off));
    atomicAdd(&P.rsize[r.lab_off + root], 1);
  }
}
__global__ void k_label_max(KParams P) {
  for (long long gp = blockIdx.x * (long long)blockDim.x + threadIdx.x; gp < P.rpix;
       gp += (long long)gridDim.x * blockDim.x) {
    const int n = P.rsize[gp];
    if (n > 0) atomicMax(&P.rmax[region_of(P, gp)], n);
  }
}

// Per-system initial state from the assembly partials (tile order).
__global__ void k_init(KParams P) {
  __shared__ double sred[kWarps];
  const int sys = blockIdx.x;
  const SysDesc d = P.sys[sys];
  double sa = 0.0, su = 0.0;
  int nact = 0;
  for (int k = threadIdx.x; k < d.ntiles; k += blockDim.x) {
    const int t = d.tile0 + k;
    if (P.tcount[t] == 0) continue;
    sa += P.fpart[t];
    su += P.fpart[P.ntiles + t];
    ++nact;
  }
  sa = block_sum(sa, sred);
  su = block_sum(su, sred);
  for (int o = 16; o > 0; o >>= 1) nact += __shfl_xor_sync(0xffffffffu, nact, o);
  __shared__ int sn[kWarps];
  if ((threadIdx.x & 31) == 0) sn[threadIdx.x >> 5] = nact;
  // the region's bounding box, over the tiles (min and max do not depend on the order)
  __shared__ int sbox[4];
  if (threadIdx.x < 4) sbox[threadIdx.x] = threadIdx.x < 2 ? 0x7fffffff : -1;
  __syncthreads();
  for (int k = threadIdx.x; k < d.ntiles; k += blockDim.x) {
    if (P.tcount[d.tile0 + k] == 0) continue;
    const int4 b = P.tbox[d.tile0 + k];
    atomicMin(&sbox[0], b.x); atomicMin(&sbox[1], b.y); atomicMax(&sbox[2], b.z); atomicMax(&sbox[3], b.w);
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  if (sys == 0) *call_start(P) = gtimer();
  const int bx0 = sbox[0], by0 = sbox[1], bx1 = sbox[2], by1 = sbox[3];
  int n = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) n += sn[w];
  SysState s;
  s.mode = M_SWEEP; s.s = 0; s.iterations = 0; s.cur = 0;
  s.pending = P_NONE; s.status = -1; s.refinements = 0; s.since = 0;
  s.isince = 0; s.nact = n; s.out_anchor = 0; s.steps = 0;
  s.warm_used = 0; s.pad1 = 0;
  s.r0 = sqrt(sa); s.outer = sqrt(su);
  if (d.warm) {
    // The plain start is the fallback: a guess whose residual is not below the
    // anchor's (or not finite) is replaced by the anchor (k_warm_fallback).
    if (s.outer < s.r0) s.warm_used = 1;
    else s.outer = s.r0;
  }
  s.best = INFINITY; s.ibest = INFINITY; s.last = 1.0; s.ibase = s.outer;
  s.omega = d.omega;
  s.stall_window = (int)kStallWindow;  // poisson.rs:80
  s.pad2 = 0;
  if (d.omega < 0.0f) {
    // automatic SOR factor: Young's optimum for red-black SOR with the Jacobi
    // spectral radius of (4+lambda)I - N on the region's bounding box (a x b
    // cells including the boundary ring): (2cos(pi/a) + 2cos(pi/b)) / (4+lambda)
    double om = 1.0;
    if (bx1 >= 0) {
      const double a = (double)(bx1 - bx0 + 2), b = (double)(by1 - by0 + 2);
      const double pi = 3.141592653589793;
      double rho = (2.0 * cos(pi / a) + 2.0 * cos(pi / b)) / (4.0 + d.lambda);
      // Several regions share one box: bound the largest region's smallest
      // eigenvalue from its area instead (Faber-Krahn: no region of that area
      // has a smaller one than the disk, pi j0^2 / area), with the area grown
      // to (sqrt(n) + 1)^2 for the half-cell margin of the discrete boundary.
      // Both are upper bounds on the Jacobi spectral radius; take the smaller.
      if (d.region1 > 0) {
        const int nmax = P.rmax[d.region1 - 1];
        if (nmax > 0) {
          const double area = (sqrt((double)nmax) + 1.0) * (sqrt((double)nmax) + 1.0);
          const double j0 = 2.404825557695773;  // first zero of the Bessel function J0
          const double pij0sq = 3.141592653589793 * (j0 * j0);
          rho = fmin(rho, (4.0 - pij0sq / area) / (4.0 + d.lambda));
        }
      }
      rho = fmin(fmax(rho, 0.0), 1.0 - 1e-15);
      om = 2.0 / (1.0 + sqrt(1.0 - rho * rho));
    }
    s.omega = om;
    const_cast<SysDesc *>(P.sys)[sys].omega = (float)om;
    // Near the optimum the residual norm of red-black SOR rises and falls on a
    // time scale of 1/(2 - omega) sweeps (its asymptotic decay time) before it
    // settles; a window of twice that many sweeps keeps the stall rule a test
    // for lost progress rather than for that transient.
    s.stall_window = max((int)kStallWindow, (int)ceil(2.0 / fmax(2.0 - om, 1e-6)));
  }
  // poisson.rs:172-189: no unknowns or a satisfied system -> 0 iterations, converged.
  if (n == 0 || s.r0 == 0.0) {
    s.mode = M_DONE; s.status = STOP_CONVERGED; s.last = 0.0; s.out_anchor = 1;
    atomicAdd(P.bar + 2, 1u);
  } else if (d.max_it <= 0) {
    // poisson.rs:202: an empty sweep loop reports the cap with last_relative = 1.
    s.mode = M_DONE; s.status = STOP_MAX; s.last = 1.0; s.out_anchor = 1;
    atomicAdd(P.bar + 2, 1u);
  } else {
    s.s = d.max_it < P.S ? d.max_it : P.S;
  }
  // a region that one thread-block cluster can hold is k_cluster_solve's: for
  // k_solve it counts as done
  Route r{};
  if (P.route) {
    if (s.mode != M_DONE && cluster_route(bx0, by0, bx1, by1, P.many, &r)) atomicAdd(P.bar + 2, 1u);
    P.route[sys] = r;
  }
  P.st[sys] = s;
  P.arrive[sys] = 0;
  P.claim[sys] = (s.mode == M_DONE || r.n) ? (unsigned long long)kClaimDone : 0ull;
}

// Restore the anchor start (u = anchor, g = -r(anchor), as k_assemble writes
// without a guess) in the systems whose guess k_init rejected.
__global__ void __launch_bounds__(kThreads) k_warm_fallback(KParams P, int TW, int TH) {
  const int t = blockIdx.x;
  const Tile tl = P.tiles[t];
  const SysDesc d = P.sys[tl.sys];
  if (!d.warm || P.st[tl.sys].warm_used || !tile_support(P, d, tl.tx, tl.ty)) return;
  const int half = TW / 2;
  for (int k = threadIdx.x; k < 2 * TH * half; k += blockDim.x) {
    const int c = k / (TH * half);
    const int r = k - c * (TH * half);
    const int y = tl.ty * TH + r / half;
    const int i = tl.tx * half + r % half;
    if (y >= d.H || i >= d.pw) continue;
    const int x = 2 * i + ((c + y) & 1);
    if (x >= d.W || !interior_at(d, x, y)) continue;
    const long long o = plane_index(d, c, y, i);
    const long long px = (long long)y * d.W + x;
    const double a = (double)d.tgt[px * d.C + d.chan];
    P.u[o] = a;
    P.g[o] = (float)(-anchor_residual(d, px, a, P.bp[o]));
  }
}

// Per system, the tiles with interior cells in index order (one block per
// system; a block-wide exclusive scan keeps the order fixed).
__global__ void k_compact(KParams P) {
  __shared__ int sw[32];
  __shared__ int s_base;
  const SysDesc d = P.sys[blockIdx.x];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (threadIdx.x == 0) s_base = 0;
  __syncthreads();
  for (int k0 = 0; k0 < d.ntiles; k0 += blockDim.x) {
    const int k = k0 + threadIdx.x;
    const int flag = (k < d.ntiles && P.tcount[d.tile0 + k] > 0) ? 1 : 0;
    const unsigned m = __ballot_sync(0xffffffffu, flag);
    const int before = __popc(m & ((1u << lane) - 1u));
    if (lane == 0) sw[warp] = __popc(m);
    __syncthreads();
    int off = s_base;
    for (int w = 0; w < warp; ++w) off += sw[w];
    if (flag) P.act[d.tile0 + off + before] = d.tile0 + k;
    __syncthreads();
    if (threadIdx.x == 0) {
      int tot = 0;
      for (int w = 0; w < nw; ++w) tot += sw[w];
      s_base += tot;
    }
    __syncthreads();
  }
}

// Interleave the result: interior cells take (float)u (the reference's `as f32`,
// poisson_blend.rs:211-219); every other pixel copies the target bit for bit.
__global__ void k_emit(KParams P, const int *__restrict__ imgs, int nimg, int TW, int TH) {
  // image by image (blockIdx.y)
  for (int img = blockIdx.y; img < nimg; img += gridDim.y) {
    const int sys0 = imgs ? imgs[img] : 0;
    const SysDesc d0 = P.sys[sys0];
    const long long npx = (long long)d0.W * d0.H;
    const int C = d0.C;
    // four channels with 16-byte aligned images: one vector load and store per pixel
    const bool vec4 = C == 4 && ((reinterpret_cast<uintptr_t>(d0.tgt) | reinterpret_cast<uintptr_t>(d0.out)) & 15) == 0;
    for (long long px = blockIdx.x * (long long)blockDim.x + threadIdx.x; px < npx;
         px += (long long)gridDim.x * blockDim.x) {
      const int y = (int)(px / d0.W), x = (int)(px - (long long)y * d0.W);
      const int tx = x / TW, ty = y / TH;
      const int c = (x + y) & 1, i = x >> 1;
      // the channels share the tile counts (k_tile_count stores one per channel)
      const bool active = P.tcount[d0.tile0 + ty * d0.ntx + tx] > 0;
      if (vec4) {
        float4 v = *reinterpret_cast<const float4 *>(d0.tgt + px * 4);
        if (active) {
          float *vv = reinterpret_cast<float *>(&v);
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) {
            if (P.st[sys0 + ch].out_anchor) continue;
            const long long o = plane_index(P.sys[sys0 + ch], c, y, i);
            if (P.cell[o]) vv[ch] = (float)P.u[o];
          }
        }
        *reinterpret_cast<float4 *>(d0.out + px * 4) = v;
        continue;
      }
      for (int ch = 0; ch < C; ++ch) {
        const SysDesc &d = P.sys[sys0 + ch];
        float v = d.tgt[px * C + ch];
        if (active && !P.st[sys0 + ch].out_anchor) {
          const long long o = plane_index(d, c, y, i);
          if (P.cell[o]) v = (float)P.u[o];
        }
        d.out[px * C + ch] = v;
      }
    }
  }
}

// Per row band of tiles of image sys0: the first and last tile column holding
// interior cells, or -1, -1 when the band holds none (two ints per band). The
// solve reads the image's source and target only in those spans, one pixel
// and one row around; the rest of the output is the target, bit for bit
// (k_emit).
__global__ void k_band_flags(KParams P, int sys0, int *spans) {
  const SysDesc d = P.sys[sys0];
  for (int ty = threadIdx.x; ty < d.nty; ty += blockDim.x) {
    int lo = -1, hi = -1;
    for (int tx = 0; tx < d.ntx; ++tx)
      if (P.tcount[d.tile0 + ty * d.ntx + tx] > 0) {
        if (lo < 0) lo = tx;
        hi = tx;
      }
    spans[2 * ty] = lo;
    spans[2 * ty + 1] = hi;
  }
}

// ----------------------------------------------------------------------------
// the persistent solve kernel
// ----------------------------------------------------------------------------
// Cell-flag rows are stored in slot ly ^ ((ly >> 1) & 1): the two rows a warp
// reads (two apart, one per half-warp) then sit an odd number of 64-byte rows
// apart, in different shared-memory banks (rows two apart would share all 16).
__host__ __device__ constexpr int cell_slot(int ly) { return ly ^ ((ly >> 1) & 1); }

// A step of a tile: load it with its halo, s sweeps, store the owned cells.
//
// Bound by instructions and their latency (23 a cell and sweep with one row a
// lane, 54 % of the issue slots), first among them the FP32 -> FP64 conversions
// of the residual. So a lane takes two rows, which share the values between
// them: 34 conversions and 10 loads for eight cells, where single rows need 42
// and 12, and the rows' parity is static. Four warps a scheduler do
// then (8 warps a block, 128 registers): on 2048 x 2048 RGBA 3.55 ms with 16
// warps of single rows, 3.24 with 12 warps of two, 3.19 with 8, 3.40 with 6;
// 48 uneven images 57, 53, 50.5 and 52 ms. Four rows a lane convert less and
// have too few warps (3.38 to 3.75 ms), and a path without the tests of the
// cell flags costs more in code than it saves (3.35).
template <int S, int TH>
__device__ void sweep_tile(const KParams &P, const SysDesc &d, int t, const Tile &tl, int s,
                           int cur, float *sE, float *sG, uint8_t *sC, double *sred) {
  using G = Geo<S, TH>;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int X0 = tl.tx * G::TW - G::HX;  // loaded column 0, a multiple of 8
  const int Y0 = tl.ty * TH - G::H;
  const int gi0 = X0 >> 1;                // plane index of loaded column 0, a multiple of 4
  const float *__restrict__ ein = cur ? P.e1 : P.e0;
  float *__restrict__ eout = cur ? P.e0 : P.e1;

  // ---- load tile + halo straight into shared memory with cp.async (L2 only:
  // other blocks wrote these planes). Outside the image the copy reads nothing
  // and zero-fills, which is exactly a boundary cell (e = 0, g = 0, cell = 0).
  constexpr int V = kPWL / 4;
  for (int k = tid; k < 2 * G::LH * V; k += G::NT) {
    const int c = k / (G::LH * V);
    const int r = k - c * (G::LH * V);
    const int ly = r / V, v = r - ly * V;
    const int gy = Y0 + ly, gi = gi0 + 4 * v;
    const bool in = gy >= 0 && gy < d.H && gi >= 0 && gi < d.pw;
    const long long o = in ? plane_index(d, c, gy, gi) : d.off;  // a valid address either way
    const int so = c * G::PLANE + ly * kPWL + 4 * v;
    cp_async16(sE + so, ein + o, in);
    cp_async16(sG + so, P.g + o, in);
    cp_async4(sC + c * G::PLANE + cell_slot(ly) * kPWL + 4 * v, P.cell + o, in);
  }
  cp_async_wait_all();
  __syncthreads();

  const float w = d.omega, inv = d.inv_denom;
  const double dd = 4.0 + d.lambda;
  constexpr int OX0 = G::HX, OX1 = G::HX + G::TW;  // owned loaded columns
  constexpr int OY0 = G::H, OY1 = G::H + TH;       // owned loaded rows
  constexpr int RQ = kPWL / 4;                      // float4 per plane row (16 lanes)
  static_assert(OX0 % 8 == 0 && OX1 % 8 == 0, "owned columns come in whole lanes");
  static_assert(G::LH % 4 == 0 || G::LH % 4 == 2, "cell slots stay inside the plane");
  constexpr int LO = OX0 / 8, LE = OX1 / 8;         // lanes (l16) whose cells are owned
  // A lane takes four consecutive plane entries (four cells of one colour) of
  // two rows, a half-warp the rows' whole width. A row's parity is static: loaded
  // row 0 is odd in every tile and a quad begins at row 1 + 4 k. Every half-sweep
  // relaxes all rows 1..LH-2 and all columns: cells outside the window that a
  // whole-grid sweep would reproduce get values nobody reads (they never reach
  // the owned region before the tile is written back), which keeps the work of
  // every warp identical.
  const int hw = lane >> 4, l16 = lane & 15;
  const bool own_x = l16 >= LO && l16 < LE;
  double acc[S];
#pragma unroll
  for (int j = 0; j < S; ++j) acc[j] = 0.0;

  auto rval = [&](float l, float r, float u, float dn, float e, float g) -> double {
    const double ns = (((double)l + (double)r) + (double)u) + (double)dn;
    return fma(-dd, (double)e, ns) - (double)g;
  };
  // One half-sweep of colour h (constants after inlining): relax the cells, if
  // so asked, and return the sum of squares of the residual at the owned ones,
  // if so asked: of black's new values, of red's before.
  auto half_sweep = [&](const int h, const bool relax, const bool duty) -> double {
    float4 *Ec = reinterpret_cast<float4 *>(sE + h * G::PLANE);
    const float4 *Eo = reinterpret_cast<const float4 *>(sE + (1 - h) * G::PLANE);
    const float4 *Gc = reinterpret_cast<const float4 *>(sG + h * G::PLANE);
    const uint32_t *Cc = reinterpret_cast<const uint32_t *>(sC + h * G::PLANE);
    double part = 0.0;
#pragma unroll 1
    for (int k = warp; k < G::QUADS; k += G::NW) {
      const int ly = 1 + 4 * k + 2 * hw, r4 = ly * RQ + l16;
      const float4 o[4] = {Eo[r4 - RQ], Eo[r4], Eo[r4 + RQ], Eo[r4 + 2 * RQ]};
      float n[2][5];  // left and right neighbours: l = n[.][0..3], r = n[.][1..4]
      float4 e[2], g[2];
      uint32_t c[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float4 ct = o[1 + r];
        if (((h + r) & 1) == 0) {
          n[r][0] = __shfl_up_sync(0xffffffffu, ct.w, 1, 16);
          n[r][1] = ct.x; n[r][2] = ct.y; n[r][3] = ct.z; n[r][4] = ct.w;
        } else {
          n[r][0] = ct.x; n[r][1] = ct.y; n[r][2] = ct.z; n[r][3] = ct.w;
          n[r][4] = __shfl_down_sync(0xffffffffu, ct.x, 1, 16);
        }
        g[r] = Gc[r4 + r * RQ];
        e[r] = Ec[r4 + r * RQ];
        c[r] = Cc[cell_slot(ly + r) * RQ + l16];
      }
      float4 ne[2] = {e[0], e[1]};
      if (relax) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float4 up = o[r], dn = o[r + 2];
          if (c[r] & 0xffu) ne[r].x = fmaf(w, ((((n[r][0] + n[r][1]) + up.x) + dn.x) - g[r].x) * inv - e[r].x, e[r].x);
          if (c[r] & 0xff00u) ne[r].y = fmaf(w, ((((n[r][1] + n[r][2]) + up.y) + dn.y) - g[r].y) * inv - e[r].y, e[r].y);
          if (c[r] & 0xff0000u) ne[r].z = fmaf(w, ((((n[r][2] + n[r][3]) + up.z) + dn.z) - g[r].z) * inv - e[r].z, e[r].z);
          if (c[r] & 0xff000000u) ne[r].w = fmaf(w, ((((n[r][3] + n[r][4]) + up.w) + dn.w) - g[r].w) * inv - e[r].w, e[r].w);
          Ec[r4 + r * RQ] = ne[r];
        }
      }
      // a lane's eight residuals behind one lane-level test, so that their
      // conversion and FP64 chains interleave
      if (duty && own_x && ly >= OY0 && ly < OY1 && (c[0] | c[1]) != 0u) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float4 up = o[r], dn = o[r + 2], v = h ? ne[r] : e[r];
          const double x0 = rval(n[r][0], n[r][1], up.x, dn.x, v.x, g[r].x), x1 = rval(n[r][1], n[r][2], up.y, dn.y, v.y, g[r].y),
                       x2 = rval(n[r][2], n[r][3], up.z, dn.z, v.z, g[r].z), x3 = rval(n[r][3], n[r][4], up.w, dn.w, v.w, g[r].w);
          if (c[r] & 0xffu) part = fma(x0, x0, part);
          if (c[r] & 0xff00u) part = fma(x1, x1, part);
          if (c[r] & 0xff0000u) part = fma(x2, x2, part);
          if (c[r] & 0xff000000u) part = fma(x3, x3, part);
        }
      }
    }
    return part;
  };
#pragma unroll
  for (int j = 0; j < S; ++j) {
    if (j >= s) break;
    const double red = half_sweep(0, true, j > 0);  // (the residual of the sweep before)
    if (j > 0) acc[j > 0 ? j - 1 : 0] += red;
    __syncthreads();
    acc[j] += half_sweep(1, true, true);
    __syncthreads();
  }
  // red cells' residual of the final state
  {
    const double part = half_sweep(0, false, true);
#pragma unroll
    for (int j = 0; j < S; ++j)
      if (j == s - 1) acc[j] += part;
  }
  // The S tile partials in one pass, each with block_sum's order (a warp's
  // xor butterfly, then the warps in index order): one barrier instead of two
  // per sweep. The scratch is the black plane of g, which nothing reads after
  // the half-sweeps (the pass above reads only the red plane).
  {
    double *sr = reinterpret_cast<double *>(sG + G::PLANE);
#pragma unroll
    for (int j = 0; j < S; ++j) {
      if (j >= s) break;
      double v = acc[j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) sr[j * G::NW + warp] = v;
    }
    __syncthreads();
    if (tid < s) {
      double tot = 0.0;
      for (int w = 0; w < G::NW; ++w) tot += sr[tid * G::NW + w];
      P.partial[(long long)tid * P.ntiles + t] = tot;
    }
  }

  // ---- write the owned cells
  constexpr int OV = G::TW / 8;  // float4 per owned plane row
  for (int k = tid; k < 2 * TH * OV; k += G::NT) {
    const int c = k / (TH * OV);
    const int r = k - c * (TH * OV);
    const int ly = G::H + r / OV, v = G::HX / 8 + r % OV;
    const int gy = Y0 + ly, gi = gi0 + 4 * v;
    if (gy < d.H && gi < d.pw) {
      const int so = c * G::PLANE + ly * kPWL + 4 * v;
      *reinterpret_cast<float4 *>(eout + plane_index(d, c, gy, gi)) =
          *reinterpret_cast<const float4 *>(sE + so);
    }
  }
}

// u += e on interior cells; e = 0 (owned cells of the tile).
template <int S, int TH>
__device__ void fold_tile(const KParams &P, const SysDesc &d, const Tile &tl, int cur) {
  using G = Geo<S, TH>;
  float *ec = cur ? P.e1 : P.e0;
  constexpr int OV = G::TW / 8;
  for (int k = threadIdx.x; k < 2 * TH * OV; k += G::NT) {
    const int c = k / (TH * OV);
    const int r = k - c * (TH * OV);
    const int gy = tl.ty * TH + r / OV;
    const int gi = tl.tx * (G::TW / 2) + 4 * (r % OV);
    if (gy >= d.H || gi >= d.pw) continue;
    const long long o = plane_index(d, c, gy, gi);
    const float4 e = __ldcg(reinterpret_cast<const float4 *>(ec + o));
    const uint32_t cv = __ldg(reinterpret_cast<const uint32_t *>(P.cell + o));
    double2 u01 = __ldcg(reinterpret_cast<const double2 *>(P.u + o));
    double2 u23 = __ldcg(reinterpret_cast<const double2 *>(P.u + o + 2));
    if (cv & 0xffu) u01.x += (double)e.x;
    if (cv & 0xff00u) u01.y += (double)e.y;
    if (cv & 0xff0000u) u23.x += (double)e.z;
    if (cv & 0xff000000u) u23.y += (double)e.w;
    *reinterpret_cast<double2 *>(P.u + o) = u01;
    *reinterpret_cast<double2 *>(P.u + o + 2) = u23;
    *reinterpret_cast<float4 *>(ec + o) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// g = -r(u) with r in FP64 exactly as residual_l2 (poisson.rs:315-321); partial ||r||^2.
template <int S, int TH>
__device__ void resid_tile(const KParams &P, const SysDesc &d, int t, const Tile &tl, double *sred) {
  using G = Geo<S, TH>;
  constexpr int half = G::TW / 2;
  const double lam4 = d.lambda + 4.0;
  double acc = 0.0;
  for (int k = threadIdx.x; k < 2 * TH * half; k += G::NT) {
    const int c = k / (TH * half);
    const int r = k - c * (TH * half);
    const int gy = tl.ty * TH + r / half;
    const int gi = tl.tx * half + r % half;
    if (gy >= d.H || gi >= d.pw) continue;
    const long long o = plane_index(d, c, gy, gi);
    if (!__ldg(P.cell + o)) continue;
    const int q = (c + gy) & 1;
    const long long oo = d.off + (long long)(1 - c) * d.plane;
    const double L = __ldcg(P.u + oo + (long long)gy * d.pw + gi - 1 + q);
    const double R = __ldcg(P.u + oo + (long long)gy * d.pw + gi + q);
    const double U = __ldcg(P.u + oo + (long long)(gy - 1) * d.pw + gi);
    const double D = __ldcg(P.u + oo + (long long)(gy + 1) * d.pw + gi);
    const double lhs = fma(lam4, -__ldcg(P.u + o), ((L + R) + U) + D);
    const double res = lhs - __ldg(P.bp + o);
    P.g[o] = (float)(-res);
    acc = fma(res, res, acc);
  }
  acc = block_sum(acc, sred);
  if (threadIdx.x == 0) P.partial[t] = acc;
}

// The state machine step run by the last tile of a system to finish a step
// (thread 0 only). sums[j] = sum of the tile partials of sweep j (tile order).
__device__ void advance(const KParams &P, const SysDesc &d, SysState *stp, int mode,
                        const double *sums) {
  SysState s = load_sys_state(stp);
  double nrms[4], rels[4];  // at most four sweeps a step (tile_config)
  const int n = mode == M_SWEEP ? s.s : (mode == M_RESID ? 1 : 0);
  for (int j = 0; j < 4; ++j)
    if (j < n) {
      nrms[j] = sqrt(sums[j]);
      rels[j] = nrms[j] / s.r0;
    }
  if (step_state(d, s, mode, nrms, rels, P.hist + d.hist_off, P.S)) atomicAdd(P.bar + 2, 1u);
  *stp = s;
}

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// Warp 0: claim the next open tile of any system, starting at system `rot`.
// Returns the system (or -1 when every system is done, an error was raised or
// the wait for work exceeded its bound), *idx and *gen in every lane.
//
// Bound by the latency of its loads: 32 systems are looked at together, where
// one thread after the other took a claim word's latency a system, and a call
// of many systems spends its end with most of them done. 48 uneven RGB images
// (144 systems): 50.5 ms with one thread, 40.0 with a warp; one
// of 2048 x 2048 RGBA 3.19 and 3.15.
__device__ int claim_tile(const KParams &P, int rot, int *idx, unsigned *gen,
                          unsigned long long t_start) {
  const int lane = threadIdx.x & 31;
  unsigned long long idle_from = 0;  // (lane 0's)
  for (;;) {
    // an error anywhere or the wall budget ends every block at its next claim
    int stop = 0;
    if (lane == 0) {
      stop = ld_vol(P.err) != 0;
      if (!stop && over_budget(P, t_start)) {
        atomicCAS(P.err, 0, KERR_DEADLINE);
        stop = 1;
      }
    }
    if (__shfl_sync(0xffffffffu, stop, 0)) return -1;
    for (int k = 0; k < P.nsys; k += 32) {
      int c = rot + k + lane;
      if (c >= P.nsys) c -= P.nsys;
      unsigned nact = 0;
      bool open = k + lane < P.nsys;
      if (open) {
        nact = (unsigned)__ldcg(&P.st[c].nact);
        open = (unsigned)ld_acquire_u64(P.claim + c) < nact;  // else the step is fully handed out
      }
      for (unsigned m = __ballot_sync(0xffffffffu, open); m; m &= m - 1) {
        const int at = __ffs((int)m) - 1;
        unsigned long long cw = 0;
        bool got = false;
        if (lane == at) {
          cw = atomicAdd(P.claim + c, 1ull);
          got = (unsigned)cw < nact;
          if (got) __threadfence();  // the claimed generation's state was published before its claim word
        }
        if (!__any_sync(0xffffffffu, got)) continue;
        cw = __shfl_sync(0xffffffffu, cw, at);
        *idx = (int)(unsigned)cw;
        *gen = (unsigned)(cw >> 32);
        return __shfl_sync(0xffffffffu, c, at);
      }
    }
    if (lane == 0) {
      if (ld_acquire(P.bar + 2) >= (unsigned)P.nsys) stop = 1;
      const unsigned long long now = gtimer();
      // every open step is handed out and being finished by other blocks; a
      // step takes milliseconds at most, so 20 s without work is a fault
      if (!idle_from) idle_from = now;
      else if (!stop && now - idle_from > 20ull * 1000000000ull) {
        atomicCAS(P.err, 0, KERR_STALLED);
        stop = 1;
      }
    }
    if (__shfl_sync(0xffffffffu, stop, 0)) return -1;
    __nanosleep(64);
  }
}

template <int S, int TH>
__global__ void __launch_bounds__((Geo<S, TH>::NT), 2) k_solve(KParams P) {
  using G = Geo<S, TH>;
  extern __shared__ __align__(16) unsigned char smem[];
  float *sE = reinterpret_cast<float *>(smem);
  float *sG = sE + 2 * G::PLANE;
  uint8_t *sC = reinterpret_cast<uint8_t *>(sG + 2 * G::PLANE);
  double *sred = reinterpret_cast<double *>(sC + 2 * G::PLANE);
  __shared__ int s_last, s_sys, s_idx;
  __shared__ unsigned s_gen;
  const unsigned long long t_start = *call_start(P);
  int rot = P.nsys > 0 ? (int)(blockIdx.x % (unsigned)P.nsys) : 0;

  for (;;) {
    if (threadIdx.x < 32) {
      int idx = 0;
      unsigned gen = 0;
      const int sys = claim_tile(P, rot, &idx, &gen, t_start);
      if (threadIdx.x == 0) {
        s_sys = sys;
        s_idx = idx;
        s_gen = gen;
      }
    }
    __syncthreads();
    const int sys = s_sys, idx = s_idx;
    const unsigned gen = s_gen;
    __syncthreads();
    if (sys < 0) break;
    rot = sys;
    const SysDesc d = P.sys[sys];
    const int t = __ldcg(P.act + d.tile0 + idx);
    const Tile tl = P.tiles[t];
    SysState *stp = P.st + sys;
    const int mode = __ldcg(&stp->mode);
    const int s = __ldcg(&stp->s);
    const int cur = __ldcg(&stp->cur);
    if (mode == M_SWEEP || mode == M_REDO) {
      sweep_tile<S, TH>(P, d, t, tl, s, cur, sE, sG, sC, sred);
    } else if (mode == M_FOLD) {
      fold_tile<S, TH>(P, d, tl, cur);
    } else {
      resid_tile<S, TH>(P, d, t, tl, sred);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      const unsigned a = atomicAdd(P.arrive + sys, 1u);
      s_last = (a == (unsigned)__ldcg(&stp->nact) - 1u);
      __threadfence();
    }
    __syncthreads();
    if (s_last) {
      // the system's step is complete: reduce its partials in tile order,
      // advance its state machine and open its next step
      double part[S];
#pragma unroll
      for (int j = 0; j < S; ++j) part[j] = 0.0;
      const int nsum = (mode == M_SWEEP) ? s : (mode == M_RESID ? 1 : 0);
      const int nact = __ldcg(&stp->nact);
      if (nsum > 0) {
        for (int k = threadIdx.x; k < nact; k += G::NT) {
          const int tk = __ldcg(P.act + d.tile0 + k);
#pragma unroll
          for (int j = 0; j < S; ++j)
            if (j < nsum) part[j] += __ldcg(P.partial + (long long)j * P.ntiles + tk);
        }
#pragma unroll
        for (int j = 0; j < S; ++j)
          if (j < nsum) part[j] = block_sum(part[j], sred);
      }
      if (threadIdx.x == 0) {
        advance(P, d, stp, mode, part);
        P.arrive[sys] = 0;
        __threadfence();
        const unsigned long long next = (unsigned long long)(gen + 1u) << 32;
        atomicExch(P.claim + sys, __ldcg(&stp->mode) == M_DONE ? (next | kClaimDone) : next);
      }
      __syncthreads();
    }
  }
}

// ----------------------------------------------------------------------------
// launch entry points (host)
// ----------------------------------------------------------------------------
template <int S, int TH>
static cudaError_t prepare_solve_t(const KParams &P, int sms, int *grid_out) {
  using G = Geo<S, TH>;
  cudaError_t e = cudaFuncSetAttribute(k_solve<S, TH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)G::kSmem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_solve<S, TH>, G::NT, G::kSmem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  int grid = per_sm * sms;
  if (grid > P.ntiles) grid = P.ntiles > 0 ? P.ntiles : 1;
  *grid_out = grid;
  return cudaSuccess;
}

template <int S, int TH>
static cudaError_t launch_prepared_t(const KParams &P, int grid, cudaStream_t stream) {
  using G = Geo<S, TH>;
  KParams Pc = P;
  Pc.S = S;
  // No block waits for a particular other block (work is claimed, never
  // assigned), so an ordinary launch suffices; the grid fills the GPU once.
  k_solve<S, TH><<<grid, G::NT, G::kSmem, stream>>>(Pc);
  return cudaGetLastError();
}

int tile_config_count() { return 5; }

// (sweeps per step S, owned tile height TH); every loaded height TH + 2(2S+1)
// leaves rows 1..LH-2 a multiple of 32.
TileConfig tile_config(int idx) {
  switch (idx) {
    case 0: return {1, 60, tile_w(1)};
    case 1: return {2, 88, tile_w(2)};
    case 2: return {3, 84, tile_w(3)};
    case 3: return {3, 52, tile_w(3)};
    default: return {4, 80, tile_w(4)};
  }
}

size_t tile_config_smem(int idx) {
  switch (idx) {
    case 0: return Geo<1, 60>::kSmem;
    case 1: return Geo<2, 88>::kSmem;
    case 2: return Geo<3, 84>::kSmem;
    case 3: return Geo<3, 52>::kSmem;
    default: return Geo<4, 80>::kSmem;
  }
}

cudaError_t launch_assembly(const KParams &P, const TileConfig &tc, cudaStream_t stream, bool any_warm) {
  if (P.ntiles <= 0) return cudaSuccess;
  if (P.nregions > 0) {
    cudaError_t e = cudaMemsetAsync(P.rsize, 0, P.rpix * sizeof(int), stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(P.rmax, 0, P.nregions * sizeof(int), stream);
    if (e != cudaSuccess) return e;
    long long nb = (P.rpix + 255) / 256;
    const unsigned blocks = (unsigned)(nb > 148 * 16 ? 148 * 16 : (nb < 1 ? 1 : nb));
    k_label_init<<<blocks, 256, 0, stream>>>(P);
    k_label_link<<<blocks, 256, 0, stream>>>(P);
    k_label_count<<<blocks, 256, 0, stream>>>(P);
    k_label_max<<<blocks, 256, 0, stream>>>(P);
  }
  k_tile_count<<<P.ntiles, 256, 0, stream>>>(P, tc.tw, tc.th);
  k_compact<<<P.nsys, 256, 0, stream>>>(P);
  k_assemble<<<P.ntiles, kThreads, 0, stream>>>(P, tc.tw, tc.th);
  k_init<<<P.nsys, 256, 0, stream>>>(P);
  if (any_warm) k_warm_fallback<<<P.ntiles, kThreads, 0, stream>>>(P, tc.tw, tc.th);
  return cudaGetLastError();
}

cudaError_t prepare_solve(const KParams &P, int cfg, int sms, int *grid) {
  switch (cfg) {
    case 0: return prepare_solve_t<1, 60>(P, sms, grid);
    case 1: return prepare_solve_t<2, 88>(P, sms, grid);
    case 2: return prepare_solve_t<3, 84>(P, sms, grid);
    case 3: return prepare_solve_t<3, 52>(P, sms, grid);
    default: return prepare_solve_t<4, 80>(P, sms, grid);
  }
}

cudaError_t launch_prepared(const KParams &P, int cfg, int grid, cudaStream_t stream) {
  switch (cfg) {
    case 0: return launch_prepared_t<1, 60>(P, grid, stream);
    case 1: return launch_prepared_t<2, 88>(P, grid, stream);
    case 2: return launch_prepared_t<3, 84>(P, grid, stream);
    case 3: return launch_prepared_t<3, 52>(P, grid, stream);
    default: return launch_prepared_t<4, 80>(P, grid, stream);
  }
}

cudaError_t launch_solve(const KParams &P, int cfg, int sms, cudaStream_t stream, int *grid) {
  cudaError_t e = prepare_solve(P, cfg, sms, grid);
  if (e != cudaSuccess) return e;
  return launch_prepared(P, cfg, *grid, stream);
}

cudaError_t launch_tile_count(const KParams &P, const TileConfig &tc, cudaStream_t stream) {
  if (P.ntiles <= 0) return cudaSuccess;
  k_tile_count<<<P.ntiles, 256, 0, stream>>>(P, tc.tw, tc.th);
  return cudaGetLastError();
}

cudaError_t launch_band_flags(const KParams &P, int sys0, int *spans, cudaStream_t stream) {
  k_band_flags<<<1, 256, 0, stream>>>(P, sys0, spans);
  return cudaGetLastError();
}

cudaError_t launch_emit(const KParams &P, const int *imgs, int nimg, const TileConfig &tc, long long npx,
                        cudaStream_t stream) {
  if (npx <= 0 || nimg <= 0) return cudaSuccess;
  long long blocks = (npx + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  // one launch for all images; their blocks fill the GPU a few times over
  const long long each = 148 * 32 / nimg > 16 ? 148 * 32 / nimg : 16;
  if (nimg > 1 && blocks > each) blocks = each;
  k_emit<<<dim3((unsigned)blocks, (unsigned)(nimg < 65535 ? nimg : 65535)), 256, 0, stream>>>(P, imgs, nimg, tc.tw, tc.th);
  return cudaGetLastError();
}

}  // namespace ptk
