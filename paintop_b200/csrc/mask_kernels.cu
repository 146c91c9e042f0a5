// mask_kernels.cu -- device rasterisers of the reference's two mask generators,
// so a mask made by a plan node never leaves the GPU before the solve reads it.
//
//   pt_mask_ellipse  mask.ellipse@1  crates/paintop-cpu/src/ellipse.rs
//                    coverage :168-201, feather :208-218, rasterize :545-565
//   pt_mask_polygon  mask.polygon@1  crates/paintop-cpu/src/mask_polygon.rs
//                    contains :161-196, rasterize :259-286 (4 x 4 subsamples, :77)
//
// Ellipse: one thread per pixel evaluates the reference's formula in fp64 with
// its fused multiply-adds; sin and cos of the angle come from the host's libm
// once per call, like the reference's sin_cos, and sqrt is correctly rounded on
// the device. Only hypot may differ from the host's in the last bit (the op is
// declared tolerance-bounded for exactly that reason).
//
// Most pixels lie far from the edge, where the feather saturates: a bound on the
// signed distance from (u/rx)^2 + (v/ry)^2 alone settles those without the
// square roots and divisions (4096 x 4096: 168 us with them for every pixel, 54 without).
//
// Polygon: the reference tests every edge at every one of the 16 subsamples of
// every pixel. A subsample row's crossing abscissa t = (y - y0) / (y1 - y0),
// c = fma(t, x1 - x0, x0) depends on the row and the edge only, and a
// subsample column x_q = (q + 0.5) / 4 lies left of c exactly when
// q < ceil(4c - 0.5), an integer computed exactly from c. So a warp owns a
// span of up to 2048 pixels of one pixel row: its lanes compute each (edge, subsample
// row)'s crossing once, turn it into that integer, add crossings right of the
// whole span to a span-wide winding, drop those left of it and keep the few
// inside it. Then each lane sums up one 128-pixel run of the span; a run without
// a crossing inside has one coverage and is stored as such. In the others the
// lanes look at a crossing each, and the pixels' 16 subsamples are resolved from
// those inside the run: up to seven one after the other, more by their sums over the
// run's columns. The arithmetic of every crossing is the reference's and winding sums
// and parities do not depend on the order crossings are visited in, so the mask is
// bit-identical to the reference's rasterize(). More than 256 edges: a block a
// span, edges in chunks.
//
// Bound by the stores of the plane where it is large (4096 x 4096: 67 MB) and by a
// warp's instructions, one after the other, where it is small. Kernel times in us, of a
// block a span with a barrier a row and every thread visiting every crossing; of a warp a
// span of 2048 pixels, every lane visiting every crossing; and of this one, whose
// spans get shorter on small images:
//   4096 x 4096, 12 vertices     62   22   23      256 vertices  186  133  111
//   1000 x  700, 12 vertices     11   12   12      256 vertices   26   80   25
//   2049 x   33, 12 vertices      7   15    8      256 vertices   15  131   13
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/paintop_cuda.h"
#include "ctx.h"
#include "abi_guard.h"

namespace {

constexpr int kSub = 4;                    // subsamples per axis (mask_polygon.rs:77)
constexpr int kRowThreads = 256;           // threads of a polygon block
constexpr int kPix = 4;                    // pixels per thread (one float4 store)
constexpr int kSpan = kRowThreads * kPix;  // pixels of a row per polygon block

__device__ __forceinline__ double feather(double sd, double half_width_px) {
  if (half_width_px <= 0.0) return sd <= 0.0 ? 1.0 : 0.0;
  double t = (sd + half_width_px) / (2.0 * half_width_px);
  t = t < 0.0 ? 0.0 : (t > 1.0 ? 1.0 : t);
  // rounded intrinsics: 1 - (t t) g must not contract into one fma
  const double smoothstep = __dmul_rn(__dmul_rn(t, t), fma(2.0, -t, 3.0));
  return __dsub_rn(1.0, smoothstep);
}

// far2: (u/rx)^2 + (v/ry)^2 above which the coverage is 0, near2: below which it
// is 1. The signed distance (f - 1) f / |grad| is at least |f - 1| min(rx, ry)
// in size, f = sqrt of that sum, so beyond half_width_px of the edge the feather
// is saturated; the limits keep a margin of 1e-9 for the rounding of both.
__global__ void k_mask_ellipse(int W, int H, double cx, double cy, double rx, double ry, double sn, double cs,
                               double half_width_px, double far2, double near2, float *out) {
  const double irx = 1.0 / rx, iry = 1.0 / ry;
  const long long n = (long long)W * H;
  const long long step = (long long)gridDim.x * blockDim.x;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += step) {
    const int j = (int)(p / W), i = (int)(p - (long long)j * W);
    const double off_x = ((double)i + 0.5) - cx, off_y = ((double)j + 0.5) - cy;
    const double local_u = fma(sn, off_y, cs * off_x);
    const double local_v = fma(cs, off_y, -sn * off_x);
    const double ax = local_u * irx, ay = local_v * iry, f2 = fma(ax, ax, ay * ay);
    double cov = 1.0;
    if (f2 > far2 && f2 < 1e200) {
      cov = 0.0;
    } else if (!(f2 < near2)) {
      const double norm_x = local_u / rx, norm_y = local_v / ry;
      const double f = sqrt(fma(norm_x, norm_x, norm_y * norm_y));
      if (f != 0.0) {
        const double grad = hypot(local_u / (rx * rx), local_v / (ry * ry));
        if (grad != 0.0) cov = feather((f - 1.0) * f / grad, half_width_px);
      }
    }
    out[p] = (float)cov;
  }
}

// Subsample columns q >= 0 (x_q = (q + 0.5) / 4) strictly left of c, i.e. the
// q with c > x_q: q < ceil(4c - 0.5). Exact: clamping c to [-1, W + 1] keeps
// every comparison with the row's subsamples, 4c is a power-of-two scaling,
// and 4c - 0.5 is representable for |4c| <= 2^31.
__device__ __forceinline__ int columns_left_of(double c, int W) {
  const double cc = fmin(fmax(c, -1.0), (double)W + 1.0);
  const double z = ceil(__dsub_rn(__dmul_rn(4.0, cc), 0.5));
  return (int)fmin(fmax(z, 0.0), 4.0 * (double)W);
}

// (k_mask_polygon_chunked) Winding of this thread's 4 x kPix subsamples of one
// subsample row, applied to the fill rule and added to inside[]: wt is shared by
// all its columns, w[l] holds crossings that fall inside its columns.
__device__ __forceinline__ void add_row(int wt, const int (&w)[kPix * kSub], bool partial, int even_odd,
                                        int (&inside)[kPix]) {
  if (!partial) {
    const int n = even_odd ? (wt & 1) : (wt != 0);
    for (int p = 0; p < kPix; ++p) inside[p] += kSub * n;
  } else {
    for (int p = 0; p < kPix; ++p)
      for (int s = 0; s < kSub; ++s) {
        const int v = wt + w[p * kSub + s];
        inside[p] += even_odd ? (v & 1) : (v != 0);
      }
  }
}

// edges[k] = (x0, y0, x1, y1) of the edge from vertex k to vertex (k + 1) % n.
__device__ __forceinline__ void store_row(float *out, int W, int j, int px, int vec4, float c0, float c1, float c2,
                                          float c3) {
  float *row = out + (long long)j * W + px;
  if (vec4 && px + kPix <= W) {
    *reinterpret_cast<float4 *>(row) = make_float4(c0, c1, c2, c3);
  } else {
    if (px < W) row[0] = c0;
    if (px + 1 < W) row[1] = c1;
    if (px + 2 < W) row[2] = c2;
    if (px + 3 < W) row[3] = c3;
  }
}

// Polygons of at most kRowThreads edges: a warp a unit of one row and one span of
// `span` runs; crossings inside the span by subsample row in shared memory
// (room for nedges each). MANY: more than kManyEdges edges; then a run's columns
// too, for a run of many crossings. (Of 12 vertices 4096 x 4096 takes 24 us that way, 22
// with every lane looking at every crossing.)
constexpr int kRun = 32 * kPix;               // pixels of a run: a float4 a lane
constexpr int kRuns = 16;                     // runs of a span at most
constexpr int kUnitWarps = kRowThreads / 32;  // warps per block at most
// Units an SM below which spans get shorter (1920 x 1080, 12 vertices: 12 us with 8, 14
// with 16, 19 with 32; of 256 vertices 45 with 16, 53 with 32, 65 with 4).
constexpr int kFewUnits = 8;
constexpr int kManyEdges = 32;                // more than one crossing a lane
size_t rows_smem(int nedges, int warps) {
  return (size_t)nedges * (sizeof(double4) + warps * kSub * sizeof(int2)) +
         (nedges > kManyEdges ? (size_t)warps * kRun * kSub * sizeof(int) : 0);
}

template <bool MANY>
__global__ void __launch_bounds__(kRowThreads, MANY ? 4 : 3) k_mask_polygon_rows(int W, int H, const double4 *__restrict__ edges,
                                                                  int nedges, int even_odd, double ymin, double ymax,
                                                                  int vec4, int span, int spans,
                                                                  float *__restrict__ out) {
  extern __shared__ __align__(32) unsigned char smem[];
  double4 *sedge = reinterpret_cast<double4 *>(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  int2 *cross = reinterpret_cast<int2 *>(sedge + nedges) + warp * kSub * nedges;  // [kSub][nedges] (column, direction)
  int *last = reinterpret_cast<int *>(reinterpret_cast<int2 *>(sedge + nedges) + warps * kSub * nedges) + warp * kRun * kSub;
  const double step = 1.0 / (double)kSub;
  for (int k = threadIdx.x; k < nedges; k += blockDim.x) sedge[k] = edges[k];
  __syncthreads();
  const long long units = (long long)H * spans;
  for (long long u = blockIdx.x * (long long)warps + warp; u < units; u += (long long)gridDim.x * warps) {
    const int j = units <= INT_MAX ? (int)u / spans : (int)(u / spans), x0 = (int)(u - (long long)j * spans) * (span * kRun);
    const int q0 = 4 * x0, q1 = 4 * min(x0 + span * kRun, W);
    int count[kSub], base[kSub];
#pragma unroll
    for (int t = 0; t < kSub; ++t) count[t] = base[t] = 0;
    const double ylo = fma(0.5, step, (double)j), yhi = fma((double)kSub - 0.5, step, (double)j);
    // a scanline below every vertex or at/above the highest one straddles no
    // edge (the half-open test compares y0 <= y and y1 <= y): coverage 0
    if (!(yhi < ymin || ylo >= ymax)) {
      __syncwarp();  // the last unit's crossings have been read
      for (int e0 = 0; e0 < nedges; e0 += 32) {
        const bool have = e0 + lane < nedges;
        const double4 E = have ? sedge[e0 + lane] : make_double4(0., 0., 0., 0.);
        // all its ends at or above the first subsample row, or below the last: no crossing
        if (MANY && __all_sync(0xffffffffu, fmax(E.y, E.w) <= ylo || fmin(E.y, E.w) > yhi)) continue;
        // two rows' crossings at a time without a branch between them, so that their
        // divisions' chains overlap (four would spill); where there is none the value is
        // not used (and its divisor is 1, as 0 takes all lanes through the division's
        // special cases)
#pragma unroll
        for (int t0 = 0; t0 < kSub; t0 += 2) {
          int qs[2], ds[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const double sy = fma((double)(t0 + i) + 0.5, step, (double)j);
            const bool below0 = E.y <= sy, below1 = E.w <= sy;
            const double tt = (sy - E.y) / (below0 == below1 ? 1.0 : E.w - E.y);
            qs[i] = columns_left_of(fma(tt, E.z - E.x, E.x), W);
            ds[i] = below0 == below1 ? 0 : (below0 ? 1 : -1);
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int t = t0 + i, qc = qs[i], d = ds[i];
            const bool right = d && qc >= q1, in = d && !right && qc > q0;  // (qc <= q0: no column of the span is left of it)
            base[t] += __popc(__ballot_sync(0xffffffffu, right && d > 0)) - __popc(__ballot_sync(0xffffffffu, right && d < 0));
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (in) cross[t * nedges + count[t] + __popc(m & ((1u << lane) - 1u))] = make_int2(qc, d);
            count[t] += __popc(m);
          }
        }
      }
      __syncwarp();
    }
    // lane r: run r's coverage, or -1 where a crossing lies inside it -- if the walk
    // over the span's crossings costs less than resolving its runs
    float run = -1.0f;
    if (lane < span && count[0] + count[1] + count[2] + count[3] <= 16 * (span - 1)) {
      const int r0 = q0 + lane * 4 * kRun, r1 = r0 + 4 * kRun;
      int n = 0;
      bool crossed = false;
#pragma unroll
      for (int t = 0; t < kSub; ++t) {
        int wt = base[t];
        for (int k = 0; k < count[t]; ++k) {
          const int2 c = cross[t * nedges + k];
          if (c.x >= r1) wt += c.y;
          else if (c.x > r0) crossed = true;
        }
        n += kSub * (even_odd ? (wt & 1) : (wt != 0));
      }
      run = crossed ? -1.0f : (float)n * (1.0f / (float)(kSub * kSub));  // k / 16, exact
    }
    const int runs = (min(x0 + span * kRun, W) - x0 + kRun - 1) / kRun;
    for (int r = 0; r < runs; ++r) {
      const float n = __shfl_sync(0xffffffffu, run, r);
      const int px = x0 + r * kRun + lane * kPix;
      if (n >= 0.0f) {
        store_row(out, W, j, px, vec4, n, n, n, n);
      } else {
        const int qp = 4 * px, r0 = q0 + r * 4 * kRun, r1 = r0 + 4 * kRun;
        int inside[kPix] = {0, 0, 0, 0};
#pragma unroll
        for (int t = 0; t < kSub; ++t) {
          int wt = base[t], within = 0;
          const int m = count[t];
          const int2 *list = cross + t * nedges;
          auto crossing = [&](int k) { return k < m ? list[k] : make_int2(r0, 0); };
          // the 16 columns' windings in a nibble each, 8 more than they are; up to
          // seven crossings leave every nibble in 1 .. 15
          constexpr unsigned long long kOnes = 0x1111111111111111ull;
          unsigned long long w = 8 * kOnes;
          auto count_one = [&](int x, int d) {
            if (x >= qp + kPix * kSub) {
              wt += d;
            } else if (x > qp) {  // columns qp .. x - 1 are left of it
              const unsigned long long left = kOnes >> (4 * (kPix * kSub - (x - qp)));
              w += d > 0 ? left : 0ull - left;
              if (!MANY) ++within;  // (the lane's)
            }
          };
          if (!MANY || m <= 7) {  // every lane looks at every crossing
            for (int k = 0; k < m; ++k) {
              const int2 c = list[k];
              count_one(c.x, c.y);
            }
          } else {
            // a crossing a lane: those right of the run count alike for all columns
            for (int k0 = 0; k0 < m; k0 += 32) {
              const int2 c = crossing(k0 + lane);
              wt += __popc(__ballot_sync(0xffffffffu, c.x >= r1 && c.y > 0)) - __popc(__ballot_sync(0xffffffffu, c.x >= r1 && c.y < 0));
              within += __popc(__ballot_sync(0xffffffffu, c.x > r0 && c.x < r1));
            }
            // ... and only those inside it one after the other
            for (int k0 = 0; k0 < m && within <= 7; k0 += 32) {
              const int2 c = crossing(k0 + lane);
              for (unsigned in = __ballot_sync(0xffffffffu, c.x > r0 && c.x < r1); in; in &= in - 1) {
                const int from = __ffs((int)in) - 1;
                count_one(__shfl_sync(0xffffffffu, c.x, from), __shfl_sync(0xffffffffu, c.y, from));
              }
            }
          }
          if (within <= 7) {
            unsigned long long in;  // a one in each covered column's nibble
            if (even_odd) {
              in = (w & kOnes) ^ ((wt & 1) ? kOnes : 0ull);
            } else if (wt > 7 || wt < -7) {
              in = kOnes;
            } else {
              const unsigned long long x = w ^ (kOnes * (unsigned long long)(8 - wt));  // 0 where the winding is 0
              in = (x | (x >> 1) | (x >> 2) | (x >> 3)) & kOnes;
            }
#pragma unroll
            for (int p = 0; p < kPix; ++p) inside[p] += __popc((unsigned)(in >> (16 * p)) & 0xffffu);
          } else if (!MANY) {  // column by column
#pragma unroll
            for (int p = 0; p < kPix; ++p)
              for (int l = p * kSub; l < (p + 1) * kSub; ++l) {
                int v = wt;
                for (int k = 0; k < m; ++k) {
                  const int2 c = list[k];
                  if (c.x > qp && c.x < qp + kPix * kSub && qp + l < c.x) v += c.y;
                }
                inside[p] += even_odd ? (v & 1) : (v != 0);
              }
          } else {
            // many: each at the last column left of it; a column's winding is the sum
            // from it to the run's end
            int4 *own = reinterpret_cast<int4 *>(last + lane * kPix * kSub);
#pragma unroll
            for (int p = 0; p < kPix; ++p) own[p] = make_int4(0, 0, 0, 0);
            __syncwarp();
            for (int k = lane; k < m; k += 32) {
              const int2 c = list[k];
              if (c.x > r0 && c.x < r1) atomicAdd(last + (c.x - r0 - 1), c.y);
            }
            __syncwarp();
            int sum = 0;
#pragma unroll
            for (int p = 0; p < kPix; ++p) {
              const int4 v = own[p];
              sum += v.x + v.y + v.z + v.w;
            }
            asm volatile("" ::: "memory");  // (they are read again below: held, they would spill)
            int from = sum;  // this lane's and all later lanes'
#pragma unroll
            for (int o = 1; o < 32; o *= 2) {
              const int x = __shfl_down_sync(0xffffffffu, from, o);
              if (lane + o < 32) from += x;
            }
            int acc = wt + from - sum;
            auto column = [&](int d) {
              acc += d;
              return even_odd ? (acc & 1) : (int)(acc != 0);
            };
#pragma unroll
            for (int p = kPix - 1; p >= 0; --p) {
              const int4 v = own[p];
              inside[p] += column(v.w);
              inside[p] += column(v.z);
              inside[p] += column(v.y);
              inside[p] += column(v.x);
            }
          }
        }
        constexpr float u = 1.0f / (float)(kSub * kSub);  // k / 16, exact
        store_row(out, W, j, px, vec4, (float)inside[0] * u, (float)inside[1] * u, (float)inside[2] * u, (float)inside[3] * u);
      }
    }
  }
}

// More than 256 edges: edges in chunks of 256, one per thread, and every
// subsample row's windings held across chunks.
// edges[k] = (x0, y0, x1, y1) of the edge from vertex k to vertex (k + 1) % n.
__global__ void __launch_bounds__(kRowThreads) k_mask_polygon_chunked(int W, int H,
                                                                     const double4 *__restrict__ edges, int nedges,
                                                                     int even_odd, double ymin, double ymax,
                                                                     int vec4, float *__restrict__ out) {
  __shared__ int cross_q[kSub][kRowThreads];        // crossings inside the span: columns left of them
  __shared__ signed char cross_dir[kSub][kRowThreads];
  __shared__ int count[kSub];
  __shared__ int span_base[kSub];                   // winding of crossings right of the whole span
  const int x0 = blockIdx.x * kSpan;
  const int q0 = 4 * x0, q1 = 4 * min(x0 + kSpan, W);
  const int px = x0 + threadIdx.x * kPix;           // this thread's first pixel
  const int qp = 4 * px;                            // and its first subsample column
  const double step = 1.0 / (double)kSub;
  for (int j = blockIdx.y; j < H; j += gridDim.y) {
    double sy[kSub];
    for (int t = 0; t < kSub; ++t) sy[t] = fma((double)t + 0.5, step, (double)j);
    int inside[kPix];
    for (int p = 0; p < kPix; ++p) inside[p] = 0;
    if (!(sy[kSub - 1] < ymin || sy[0] >= ymax)) {
      int wt[kSub];
      int w[kSub][kPix * kSub];
      bool partial[kSub];
      for (int t = 0; t < kSub; ++t) {
        wt[t] = 0;
        partial[t] = false;
        for (int l = 0; l < kPix * kSub; ++l) w[t][l] = 0;
      }
      if (threadIdx.x < kSub) span_base[threadIdx.x] = 0;
      for (int e0 = 0; e0 < nedges; e0 += kRowThreads) {
        if (threadIdx.x < kSub) count[threadIdx.x] = 0;
        __syncthreads();
        const int e = e0 + threadIdx.x;
        if (e < nedges) {
          const double4 E = edges[e];
          for (int t = 0; t < kSub; ++t) {
            const bool below0 = E.y <= sy[t], below1 = E.w <= sy[t];
            if (below0 == below1) continue;
            const double tt = (sy[t] - E.y) / (E.w - E.y);
            const int qc = columns_left_of(fma(tt, E.z - E.x, E.x), W);
            const int d = below0 ? 1 : -1;
            if (qc >= q1) {
              atomicAdd(&span_base[t], d);
            } else if (qc > q0) {  // (qc <= q0: no column of the span is left of it)
              const int k = atomicAdd(&count[t], 1);
              cross_q[t][k] = qc;
              cross_dir[t][k] = (signed char)d;
            }
          }
        }
        __syncthreads();
        for (int t = 0; t < kSub; ++t) {
          const int m = count[t];
          for (int k = 0; k < m; ++k) {
            const int qc = cross_q[t][k];
            const int d = cross_dir[t][k];
            if (qc >= qp + kPix * kSub) {
              wt[t] += d;
            } else if (qc > qp) {
              partial[t] = true;
              for (int l = 0; l < kPix * kSub; ++l) w[t][l] += qp + l < qc ? d : 0;
            }
          }
        }
        __syncthreads();
      }
      for (int t = 0; t < kSub; ++t) add_row(wt[t] + span_base[t], w[t], partial[t], even_odd, inside);
      __syncthreads();  // span_base is reset for the next row only after every read
    }
    constexpr float u = 1.0f / (float)(kSub * kSub);  // k / 16, exact
    store_row(out, W, j, px, vec4, (float)inside[0] * u, (float)inside[1] * u, (float)inside[2] * u, (float)inside[3] * u);
  }
}

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

pt_status mfail(pt_ctx *ctx, pt_status s, const std::string &msg) {
  if (ctx) ctx->last_error = msg;
  return s;
}

// Device output (the caller's, or the arena's first bytes for a host mask) and
// `extra` bytes of arena scratch after it.
pt_status mask_target(pt_ctx *ctx, size_t npx, bool device_out, float *mask, size_t extra, float **out,
                      char **scratch) {
  const size_t own = device_out ? 0 : align256(npx * sizeof(float));
  if (!ctx->reserve(own + align256(extra))) return mfail(ctx, PT_OOM, "device arena allocation failed");
  char *base = static_cast<char *>(ctx->arena);
  *out = device_out ? mask : reinterpret_cast<float *>(base);
  *scratch = base + own;
  return PT_OK;
}

// Events: ev[0] call start, ev[1]/ev[2] around the rasteriser, ev[3] call end
// (read back by pt_ctx_last_timing).
pt_status mask_begin(pt_ctx *ctx) {
  for (auto &e : ctx->ev)
    if (!e && cudaEventCreate(&e) != cudaSuccess) return mfail(ctx, PT_LAUNCH_FAILED, "event create");
  cudaEventRecord(ctx->ev[0], ctx->stream);
  return PT_OK;
}

pt_status mask_finish(pt_ctx *ctx, size_t npx, bool device_out, float *mask, const float *dev, int launches) {
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && !device_out)
    e = cudaMemcpyAsync(mask, dev, npx * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaEventRecord(ctx->ev[3], ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return mfail(ctx, PT_LAUNCH_FAILED, std::string("mask: ") + cudaGetErrorString(e));
  float a = 0.f, b = 0.f;
  if (cudaEventElapsedTime(&a, ctx->ev[1], ctx->ev[2]) != cudaSuccess) a = -1.f;
  if (cudaEventElapsedTime(&b, ctx->ev[0], ctx->ev[3]) != cudaSuccess) b = -1.f;
  cudaGetLastError();
  ctx->last_solve_ms = a;
  ctx->last_call_ms = b;
  ctx->last_launches = launches;
  ctx->last_h2d = ctx->last_d2h = 0;  // not counted on this path
  return PT_OK;
}

}  // namespace

extern "C" pt_status pt_mask_ellipse(pt_ctx *ctx, uint32_t width, uint32_t height, double center_x,
                                     double center_y, double radius_x, double radius_y, double angle_rad,
                                     double half_width_px, float *mask, uint32_t flags) {
  return abi_guard(ctx, [&]() -> pt_status {
    if (!ctx) return PT_INVALID_ARG;
    const size_t npx = (size_t)width * height;
    if (npx && !mask) return mfail(ctx, PT_INVALID_ARG, "null mask buffer");
    // the checks of EllipseGeometry::resolve (ellipse.rs:119-158)
    if (!std::isfinite(center_x) || !std::isfinite(center_y) || !std::isfinite(angle_rad))
      return mfail(ctx, PT_INVALID_ARG, "non-finite ellipse center or angle");
    if (!(std::isfinite(radius_x) && radius_x > 0.0) || !(std::isfinite(radius_y) && radius_y > 0.0))
      return mfail(ctx, PT_INVALID_ARG, "ellipse radii must be finite and > 0");
    if (!std::isfinite(half_width_px) || half_width_px < 0.0)
      return mfail(ctx, PT_INVALID_ARG, "feather half-width must be finite and >= 0");
    if (npx == 0) return PT_OK;
    if (npx > (size_t)INT32_MAX * 4) return mfail(ctx, PT_INVALID_ARG, "mask too large");
    std::lock_guard<std::mutex> lock(ctx->mu);
    cudaError_t ce = cudaSetDevice(ctx->device);
    if (ce != cudaSuccess) return mfail(ctx, PT_NO_DEVICE, cudaGetErrorString(ce));
    const bool dev = (flags & PT_FLAG_DEVICE_POINTERS) != 0;
    float *out = nullptr;
    char *scratch = nullptr;
    pt_status st = mask_target(ctx, npx, dev, mask, 0, &out, &scratch);
    if (st != PT_OK) return st;
    if ((st = mask_begin(ctx)) != PT_OK) return st;
    const double sn = std::sin(angle_rad), cs = std::cos(angle_rad);
    const long long blocks = std::min<long long>(((long long)npx + 255) / 256, (long long)ctx->sms * 16);
    // (radii whose squares leave the range of doubles take the formula everywhere)
    const double rmin = std::min(radius_x, radius_y), band = half_width_px / rmin;
    const bool plain = rmin >= 1e-100 && std::max(radius_x, radius_y) <= 1e100;
    const double far2 = plain ? (1.0 + band) * (1.0 + band) * (1.0 + 1e-9) : INFINITY;
    const double near2 = plain && band < 1.0 ? (1.0 - band) * (1.0 - band) * (1.0 - 1e-9) : -1.0;
    cudaEventRecord(ctx->ev[1], ctx->stream);
    k_mask_ellipse<<<(unsigned)blocks, 256, 0, ctx->stream>>>((int)width, (int)height, center_x, center_y,
                                                             radius_x, radius_y, sn, cs, half_width_px, far2, near2, out);
    cudaEventRecord(ctx->ev[2], ctx->stream);
    return mask_finish(ctx, npx, dev, mask, out, 1);
  });
}

extern "C" pt_status pt_mask_polygon(pt_ctx *ctx, uint32_t width, uint32_t height, const double *points_xy,
                                     uint32_t n_points, int32_t fill_rule, float *mask, uint32_t flags) {
  return abi_guard(ctx, [&]() -> pt_status {
    if (!ctx) return PT_INVALID_ARG;
    const size_t npx = (size_t)width * height;
    if (npx && !mask) return mfail(ctx, PT_INVALID_ARG, "null mask buffer");
    if (n_points && !points_xy) return mfail(ctx, PT_INVALID_ARG, "null points");
    if (fill_rule != PT_FILL_NONZERO && fill_rule != PT_FILL_EVEN_ODD)
      return mfail(ctx, PT_INVALID_ARG, "unknown fill rule");
    for (size_t k = 0; k < 2 * (size_t)n_points; ++k)
      if (!std::isfinite(points_xy[k])) return mfail(ctx, PT_INVALID_ARG, "non-finite polygon coordinate");
    if (npx == 0) return PT_OK;
    // subsample column indices (4 per pixel) are int32 in the kernel
    if (width > (1u << 28) || height > (uint32_t)INT32_MAX) return mfail(ctx, PT_INVALID_ARG, "mask too large");
    std::lock_guard<std::mutex> lock(ctx->mu);
    cudaError_t ce = cudaSetDevice(ctx->device);
    if (ce != cudaSuccess) return mfail(ctx, PT_NO_DEVICE, cudaGetErrorString(ce));
    const bool dev = (flags & PT_FLAG_DEVICE_POINTERS) != 0;
    float *out = nullptr;
    char *scratch = nullptr;
    pt_status st = mask_target(ctx, npx, dev, mask, (size_t)n_points * sizeof(double4), &out, &scratch);
    if (st != PT_OK) return st;
    if ((st = mask_begin(ctx)) != PT_OK) return st;
    if (n_points < 3) {  // contains() is false everywhere (mask_polygon.rs:162-165)
      cudaEventRecord(ctx->ev[1], ctx->stream);
      ce = cudaMemsetAsync(out, 0, npx * sizeof(float), ctx->stream);
      cudaEventRecord(ctx->ev[2], ctx->stream);
      if (ce != cudaSuccess) return mfail(ctx, PT_LAUNCH_FAILED, cudaGetErrorString(ce));
      return mask_finish(ctx, npx, dev, mask, out, 0);
    }
    std::vector<double4> edges(n_points);
    double ymin = points_xy[1], ymax = points_xy[1];
    for (uint32_t k = 0; k < n_points; ++k) {
      const uint32_t q = (k + 1) % n_points;
      edges[k] = make_double4(points_xy[2 * k], points_xy[2 * k + 1], points_xy[2 * q], points_xy[2 * q + 1]);
      ymin = std::min(ymin, points_xy[2 * k + 1]);
      ymax = std::max(ymax, points_xy[2 * k + 1]);
    }
    double4 *dedges = reinterpret_cast<double4 *>(scratch);
    ce = cudaMemcpyAsync(dedges, edges.data(), edges.size() * sizeof(double4), cudaMemcpyHostToDevice, ctx->stream);
    if (ce != cudaSuccess) return mfail(ctx, PT_LAUNCH_FAILED, cudaGetErrorString(ce));
    const uint32_t spans = (width + kSpan - 1) / kSpan;
    const int vec4 = (width % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) ? 1 : 0;
    const int even_odd = fill_rule == PT_FILL_EVEN_ODD ? 1 : 0;
    cudaEventRecord(ctx->ev[1], ctx->stream);
    if (n_points > (uint32_t)kRowThreads) {
      const dim3 grid(spans, std::min<uint32_t>(height, 65535u));
      k_mask_polygon_chunked<<<grid, kRowThreads, 0, ctx->stream>>>((int)width, (int)height, dedges,
                                                                    (int)n_points, even_odd, ymin, ymax, vec4, out);
    } else {
      // a unit a warp, at most eight blocks an SM; on images whose rows of whole
      // spans leave SMs idle, shorter spans (a warp goes through its crossings one after
      // the other) and smaller blocks
      int span = kRuns, warps = kUnitWarps;
      auto count = [&](int s) { return (long long)height * ((width + s * kRun - 1) / (s * kRun)); };
      const bool many = n_points > (uint32_t)kManyEdges;
      const int few = many ? 2 * kFewUnits : kFewUnits;  // (of many crossings each unit takes longer)
      while (span > 1 && count(span) < (long long)ctx->sms * few) span /= 2;
      const long long units = count(span);
      while (warps > 1 && units < (long long)ctx->sms * warps) warps /= 2;
      const unsigned blocks = (unsigned)std::min<long long>((units + warps - 1) / warps, (long long)ctx->sms * 8);
      const size_t smem = rows_smem((int)n_points, warps);
      if (smem > 48 * 1024) {  // (more than a launch may ask for unasked)
        ce = cudaFuncSetAttribute(k_mask_polygon_rows<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)rows_smem(kRowThreads, kUnitWarps));
        if (ce != cudaSuccess) return mfail(ctx, PT_LAUNCH_FAILED, cudaGetErrorString(ce));
      }
      (many ? k_mask_polygon_rows<true> : k_mask_polygon_rows<false>)<<<blocks, 32 * warps, smem, ctx->stream>>>(
          (int)width, (int)height, dedges, (int)n_points, even_odd, ymin, ymax, vec4, span,
          (int)((width + span * kRun - 1) / (span * kRun)), out);
    }
    cudaEventRecord(ctx->ev[2], ctx->stream);
    return mask_finish(ctx, npx, dev, mask, out, 1);
  });
}
