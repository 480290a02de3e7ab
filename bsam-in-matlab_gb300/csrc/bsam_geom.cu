// bsam_geom.cu -- device part of the diffuse-domain coefficient sampling:
// the squared distance from sample points to a closed polygon
// (DiffuseDomainBSAM/src/ddStarfishGeometry.m:140-177, exact point-to-
// segment distance).  The host keeps the O(n) parts (the radial sign test
// and the starting candidate, which need atan2/cos/sin); the device does the
// O(n x segments) minimum.  Per segment the arithmetic is the reference's
//   t  = ((x - ax) ex + (y - ay) ey) / |e|^2,  t = max(0, min(1, t))
//   dd = ((x - ax) - t ex)^2 + ((y - ay) - t ey)^2
// in that order (no contraction), and a minimum does not depend on the
// order of its terms, so the result equals the host's bit for bit.
//
// GB300 issues a warp's FP64 operation every 19 cycles per SM, so the search
// runs in FP32 with error bounds and only the segments that can hold the
// minimum are evaluated in FP64: a first pass over boxes of 64 and of 8
// segments finds the FP32 minimum, a second collects every segment within
// the bounds of it (one or two per point), and the lanes then evaluate their
// own candidates in step.  300,000 points against 2,999 segments: the kernel
// took 4.3 ms with FP64 boxes and segments, now 0.14.
#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>
#include <cstdint>
#include <string>

#include "bsam_dev.h"
#include "internal.h"

namespace {

constexpr int kThreads = 256;
constexpr int kGroup = 8;               // segments per box
constexpr int kSuper = 8;               // boxes per outer box (kGroup kSuper = 64: two warps)
constexpr int kKeep = 4;                // candidates a lane collects before it evaluates them

// the FP32 tables: per segment (ax, ay, ex, ey), per group and per outer
// group a box rounded outwards (minx, miny, maxx, maxy)
struct SegTables {
  float4 *seg, *box, *outer;
};

// one block per outer group, one thread per segment
__global__ void __launch_bounds__(kGroup *kSuper) k_segtables(const double *__restrict__ v, int ns, SegTables T) {
  const int t = threadIdx.x, i = blockIdx.x * (kGroup * kSuper) + t;
  float4 b = make_float4(INFINITY, INFINITY, -INFINITY, -INFINITY);
  if (i < ns) {
    const double ax = v[2 * i], ay = v[2 * i + 1], bx = v[2 * i + 2], by = v[2 * i + 3];
    T.seg[i] = make_float4((float)ax, (float)ay, (float)(bx - ax), (float)(by - ay));
    b = make_float4(fminf(__double2float_rd(ax), __double2float_rd(bx)),
                    fminf(__double2float_rd(ay), __double2float_rd(by)),
                    fmaxf(__double2float_ru(ax), __double2float_ru(bx)),
                    fmaxf(__double2float_ru(ay), __double2float_ru(by)));
  }
  auto join = [&](int off) {
    b.x = fminf(b.x, __shfl_xor_sync(0xffffffffu, b.x, off));
    b.y = fminf(b.y, __shfl_xor_sync(0xffffffffu, b.y, off));
    b.z = fmaxf(b.z, __shfl_xor_sync(0xffffffffu, b.z, off));
    b.w = fmaxf(b.w, __shfl_xor_sync(0xffffffffu, b.w, off));
  };
  for (int off = 1; off < kGroup; off *= 2) join(off);
  if (t % kGroup == 0 && i < ns) T.box[i / kGroup] = b;
  for (int off = kGroup; off < 32; off *= 2) join(off);
  __shared__ float4 half;
  if (t == 32) half = b;
  __syncthreads();
  if (t == 0) {
    b.x = fminf(b.x, half.x);
    b.y = fminf(b.y, half.y);
    b.z = fmaxf(b.z, half.z);
    b.w = fmaxf(b.w, half.w);
    T.outer[blockIdx.x] = b;
  }
}

// the reference's squared distance to segment g (FP64)
__device__ __forceinline__ double seg_dist2(const double *__restrict__ v, int g, double px, double py) {
  const double ax = v[2 * g], ay = v[2 * g + 1];
  const double ex = v[2 * (g + 1)] - ax, ey = v[2 * (g + 1) + 1] - ay;
  const double l2 = ex * ex + ey * ey;
  const double rx = px - ax, ry = py - ay;
  double t = (rx * ex + ry * ey) / l2;
  t = fmax(0.0, fmin(1.0, t));
  const double qx = rx - t * ex, qy = ry - t * ey;
  return qx * qx + qy * qy;
}

// FP32 error bound.  With u = 2^-24 and every coordinate at most M: the point
// relative to the segment's start is off by at most 5 u M per component, the
// projection along the segment by 27 u M, the residual vector by 24 u M, the
// length and its square's rounding by 12 u M more -- below 64 u M in all; the
// bound used is twice that.
constexpr float kTol = 128.0f / 16777216.0f;

// `scale`: largest vertex coordinate; a point for which FP32 has no room
// (coordinates beyond 1e15, below 1e-12, or not finite) takes every segment
// in FP64
__global__ void __launch_bounds__(kThreads) k_segdist(const double *__restrict__ v, int ns, SegTables T, double scale,
                                                      const double *__restrict__ x, const double *__restrict__ y,
                                                      double *__restrict__ best, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  // a NaN start stays: no distance compares below it
  const bool on = i < n && !isnan(best[i]);
  const double px = on ? x[i] : 0.0, py = on ? y[i] : 0.0;
  double b = on ? best[i] : 0.0;
  const double M = fmax(scale, fmax(fabs(px), fabs(py)));
  const bool fits = M <= 1e15 && scale >= 1e-12;
  if (on && !fits)
    for (int g = 0; g < ns; ++g) b = fmin(b, seg_dist2(v, g, px, py));
  const bool live = on && fits;
  if (__any_sync(0xffffffffu, live)) {
    const float xl = __double2float_rd(px), xh = __double2float_ru(px), yl = __double2float_rd(py),
                yh = __double2float_ru(py);
    const float xf = (float)px, yf = (float)py;
    // a lower bound on the squared distance to a box
    auto box2 = [&](const float4 B) {
      const float dx = fmaxf(fmaxf(__fsub_rd(B.x, xh), __fsub_rd(xl, B.z)), 0.0f);
      const float dy = fmaxf(fmaxf(__fsub_rd(B.y, yh), __fsub_rd(yl, B.w)), 0.0f);
      return __fadd_rd(__fmul_rd(dx, dx), __fmul_rd(dy, dy));
    };
    auto seg2 = [&](const float4 S) {
      const float rx = xf - S.x, ry = yf - S.y;
      const float t = fmaxf(0.0f, fminf(1.0f, (rx * S.z + ry * S.w) / (S.z * S.z + S.w * S.w)));
      const float qx = rx - t * S.z, qy = ry - t * S.w;
      return qx * qx + qy * qy;
    };
    const int ng = (ns + kGroup - 1) / kGroup, no = (ng + kSuper - 1) / kSuper;
    // first pass: the FP32 minimum.  A box is skipped only where its lower
    // bound is above the smallest value so far by more than the bounds, so
    // the minimum found is within them of the true one.
    float m = live ? __double2float_ru(b) : -1.0f;
    const float tol = kTol * (float)M;
    auto widen = [&](float d2) {          // (sqrt(d2) + 2 tol)^2, rounded up
      const float s = __fadd_ru(__fsqrt_ru(d2), 2.0f * tol);
      return __fmul_ru(__fmul_ru(s, s), 1.000001f);
    };
    float thr = live ? widen(m) : -1.0f;
    for (int o = 0; o < no; ++o) {
      if (!__any_sync(0xffffffffu, box2(T.outer[o]) <= thr)) continue;
      for (int g = o * kSuper; g < min(ng, (o + 1) * kSuper); ++g) {
        if (!__any_sync(0xffffffffu, box2(T.box[g]) <= thr)) continue;
        for (int j = g * kGroup; j < min(ns, (g + 1) * kGroup); ++j) m = fminf(m, seg2(T.seg[j]));
        if (live) thr = fminf(thr, widen(fmaxf(m, 0.0f)));
      }
    }
    // second pass: the segments that can hold the minimum
    int keep[kKeep], nk = 0;
#pragma unroll
    for (int c = 0; c < kKeep; ++c) keep[c] = 0;
    for (int o = 0; o < no; ++o) {
      if (!__any_sync(0xffffffffu, box2(T.outer[o]) <= thr)) continue;
      for (int g = o * kSuper; g < min(ng, (o + 1) * kSuper); ++g) {
        if (!__any_sync(0xffffffffu, box2(T.box[g]) <= thr)) continue;
        for (int j = g * kGroup; j < min(ns, (g + 1) * kGroup); ++j) {
          const bool in = seg2(T.seg[j]) <= thr;
          if (__any_sync(0xffffffffu, in && nk == kKeep)) {   // a lane is full: it evaluates this one at once
            if (in && nk == kKeep) b = fmin(b, seg_dist2(v, j, px, py));
          }
          if (in && nk < kKeep) {
#pragma unroll
            for (int c = 0; c < kKeep; ++c) keep[c] = c == nk ? j : keep[c];
            ++nk;
          }
        }
      }
    }
#pragma unroll
    for (int c = 0; c < kKeep; ++c)
      if (c < nk) b = fmin(b, seg_dist2(v, keep[c], px, py));
  }
  if (on) best[i] = b;
}

int gfail(int code, const std::string &m) { return bsam_internal_set_error(code, m); }

#define GCK(x)                                                                                      \
  do {                                                                                              \
    cudaError_t e_ = (x);                                                                           \
    if (e_ != cudaSuccess)                                                                          \
      return gfail(e_ == cudaErrorMemoryAllocation ? BSAM_ERR_NOMEM : BSAM_ERR_CUDA,                 \
                   std::string(#x) + ": " + cudaGetErrorString(e_));                                \
  } while (0)

}  // namespace

extern "C" int bsam_polygon_dist2(bsam_ctx ctx, const double *verts, int nverts, const double *x, const double *y,
                                  double *best, int64_t n) {
  if (!ctx || !verts || nverts < 2 || n < 0 || (n && (!x || !y || !best)))
    return gfail(BSAM_ERR_ARG, "bsam_polygon_dist2: bad argument");
  if (n == 0) return BSAM_OK;
  GCK(cudaSetDevice(ctx->device));
  const int ns = nverts - 1, ng = (ns + kGroup - 1) / kGroup, no = (ng + kSuper - 1) / kSuper;
  const size_t nv = 2 * (size_t)nverts, nt = 2 * ((size_t)ns + ng + no);   // in doubles (the tables' float4s)
  const size_t need = sizeof(double) * (nt + nv + 3 * (size_t)n);
  if (need > ctx->scratch_bytes) {   // stream-ordered: no device-wide synchronisation
    if (ctx->scratch) cudaFreeAsync(ctx->scratch, ctx->stream);
    ctx->scratch = nullptr;
    ctx->scratch_bytes = 0;
    GCK(cudaMallocAsync(&ctx->scratch, need, ctx->stream));
    ctx->scratch_bytes = need;
  }
  double scale = 0;                  // a NaN or infinite vertex: every segment in FP64
  for (size_t k = 0; k < nv; ++k) {
    const double a = std::fabs(verts[k]);
    if (!(a <= scale)) scale = a <= DBL_MAX ? a : INFINITY;
    if (scale == INFINITY) break;
  }
  SegTables T;
  T.seg = (float4 *)ctx->scratch;
  T.box = T.seg + ns;
  T.outer = T.box + ng;
  double *dv = (double *)ctx->scratch + nt, *dx = dv + nv, *dy = dx + n, *db = dy + n;
  cudaStream_t s = ctx->stream;
  GCK(cudaMemcpyAsync(dv, verts, sizeof(double) * nv, cudaMemcpyHostToDevice, s));
  GCK(cudaMemcpyAsync(dx, x, sizeof(double) * n, cudaMemcpyHostToDevice, s));
  GCK(cudaMemcpyAsync(dy, y, sizeof(double) * n, cudaMemcpyHostToDevice, s));
  GCK(cudaMemcpyAsync(db, best, sizeof(double) * n, cudaMemcpyHostToDevice, s));
  k_segtables<<<no, kGroup * kSuper, 0, s>>>(dv, ns, T);
  const unsigned grid = (unsigned)((n + kThreads - 1) / kThreads);
  k_segdist<<<grid, kThreads, 0, s>>>(dv, ns, T, scale, dx, dy, db, n);
  GCK(cudaGetLastError());
  GCK(cudaMemcpyAsync(best, db, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
  GCK(cudaStreamSynchronize(s));
  return BSAM_OK;
}
