// Shared device helpers of the B200 HashPoint kernels.
//
// Arithmetic that decides which points a ray keeps is written with explicit
// round-to-nearest intrinsics (__fmaf_rn, __fmul_rn, ...) so nvcc cannot fuse
// or reorder it: every expression reproduces, bit for bit, the way the
// reference's kernels round (operand order and fused multiply-adds were
// established by diffing GPU outputs of the reference's expressions), and the
// CPU oracle restates the same sequence with fmaf.  CUDA's norm3df, rnorm3df
// and __expf are called exactly where the reference calls them.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../include/hashpoint_b200.h"

// Point counts above which torch's cuBLAS GEMMs of the reference projection
// (epcq/epcq.py:253 world->camera, :261 camera->image) used a fused
// multiply-add chain on B200 (torch 2.11, cuBLAS 12.8); at or below them each
// product was rounded separately.  Established by diffing torch outputs against
// both forms for every N in 2..2100 and every 8th N in 200000..260000; N = 1
// matched neither form for the world->camera product.
#ifndef HP_WORLD_FUSED_ABOVE
#define HP_WORLD_FUSED_ABOVE 1536
#endif
#ifndef HP_IMAGE_FUSED_ABOVE
#define HP_IMAGE_FUSED_ABOVE 233023
#endif

namespace hp {

constexpr int kKeptPerCell = 48;   // kept points per window cell (POINT_BUFFER_SIZE48)
constexpr int kBins = 128;         // t-histogram bins (MAX_SAMPLE_POINTS_NUM)
constexpr int kBallBuf = 8;        // ids gathered per sample (POINT_BUFFER_SIZE8)
constexpr int kQueryPerCell = 32;  // ids gathered per window cell by the ray query (POINT_BUFFER_SIZE)
constexpr int kMaxKernel = 5;      // largest window side of the sampling path (the reference's warps cover 32 cells)

// Camera as the kernels see it: c2w stays a device pointer (rows 0..2 read).
struct DevCamera {
  const float* c2w;
  float fx, fy, cx, cy;
  int width, height;
};

// Options as the kernels see them.
struct DevOptions {
  int k;
  float t_intvl;
  float radius;
  int S, P;
  int num_point_per_ray;
  float alpha_g, gamma;
};

struct Ray {
  float o[3];
  float d[3];
  float dd;  // dot(d, d), constant per ray
};

// dot3 as the reference's _dot3d (cuda_util.cuh:57) rounds under nvcc: fma(a2,b2, fma(a0,b0, a1*b1)).
__device__ __forceinline__ float dot3(float a0, float a1, float a2, float b0, float b1, float b2) {
  return __fmaf_rn(a2, b2, __fmaf_rn(a0, b0, __fmul_rn(a1, b1)));
}

// cam2world_ray (cuda_util.cuh:338-354): x = (u + 0.5 - cx) / fx in double,
// d_i = fma(c_i0, x, c_i1 * y) + c_i2, normalised with rnorm3df.
__device__ __forceinline__ void make_ray(const float* __restrict__ c2w, float fx, float fy, float cx, float cy, int u,
                                         int v, Ray& r) {
  const float x = (float)(((double)u + 0.5 - (double)cx) / (double)fx);
  const float y = (float)(((double)v + 0.5 - (double)cy) / (double)fy);
  float d[3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    d[i] = __fadd_rn(__fmaf_rn(c2w[4 * i + 0], x, __fmul_rn(c2w[4 * i + 1], y)), c2w[4 * i + 2]);
    r.o[i] = c2w[4 * i + 3];
  }
  const float rn = rnorm3df(d[0], d[1], d[2]);
#pragma unroll
  for (int i = 0; i < 3; i++) r.d[i] = __fmul_rn(d[i], rn);
  r.dd = dot3(r.d[0], r.d[1], r.d[2], r.d[0], r.d[1], r.d[2]);
}

// calculate_neighbor_uv (cuda_util.cuh:382-388) in exact integer form:
// offsets ceil((l+1)/k) - ceil(k/2) and l%k - (ceil(k/2)-1), clamped into the image.
__device__ __forceinline__ void window_cell(int v, int u, int k, int H, int W, int l, int& vv, int& uu) {
  const int koff = (k + 1) >> 1;
  const int a = v + (l + k) / k - koff;
  const int b = u + (l % k) - (koff - 1);
  vv = min(max(a, 0), H - 1);
  uu = min(max(b, 0), W - 1);
}

__device__ __forceinline__ float4 load_point(const float* __restrict__ xyz, int id) {
  const float* p = xyz + 3 * (size_t)id;
  return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), 0.f);
}

// The reference keeps a candidate when norm3df(e) < radius (e = point minus its
// projection on the ray).  The squared length e2 (three roundings) decides it
// without the square root whenever e2 is outside a band of relative width
// 2^-16 around radius^2 -- far wider than the few-ulp errors of e2 and
// norm3df -- and norm3df decides inside the band, so the result is identical.
// A radius of zero, below zero or NaN keeps nothing: norm3df decides all.
struct RadiusTest {
  float r, lo2, hi2;
  bool fast;  // else the band is everything
};

__host__ __device__ inline RadiusTest make_radius_test(float r) {
  RadiusTest rt;
  rt.r = r;
  const double r2 = (double)r * (double)r;
  rt.fast = r > 0.0f && r2 > 1e-30 && r2 < 1e30;
  rt.lo2 = rt.fast ? (float)(r2 * (1.0 - 1.0 / 65536.0)) : -1.0f;
  rt.hi2 = rt.fast ? (float)(r2 * (1.0 + 1.0 / 65536.0)) : INFINITY;
  return rt;
}

// q: the squared length of (e0, e1, e2).
__device__ __forceinline__ float squared(float e0, float e1, float e2) {
  return __fmaf_rn(e2, e2, __fmaf_rn(e1, e1, __fmul_rn(e0, e0)));
}

// For all lanes of the warp; the band is taken by a branch of the whole warp.
__device__ __forceinline__ bool within_radius(const RadiusTest& rt, bool in, float q, float e0, float e1, float e2) {
  bool kept = in && q < rt.lo2;
  const bool band = in && !(q < rt.lo2) && !(q > rt.hi2);
  if (__any_sync(0xffffffffu, band)) {
    const float n = norm3df(e0, e1, e2);
    if (band) kept = n < rt.r;
  }
  return kept;
}

// PointRayInterset (cuda_util.cuh:215-236): t = (p - o).d / d.d, the point's
// projection on the ray fma(t, d, o), its distance norm3df(p - projection).
// ray_t is t, the correctly rounded quotient, with inv_dd = RN(1 / d.d): a first
// quotient, its exact residual and one fused step (Markstein 1990).  d is
// normalised, so d.d is a few ulp from 1; for every d.d within 64 ulp of 1 and
// every numerator mantissa this equals the division, at 3 instructions for 10
// and without its branch.  (Numerators below 2^-100 and from 2^127 on, whose
// residual or quotient leaves the normal range, are not covered.)
__device__ __forceinline__ float ray_t(const Ray& r, float inv_dd, const float4& p) {
  const float num = dot3(__fsub_rn(p.x, r.o[0]), __fsub_rn(p.y, r.o[1]), __fsub_rn(p.z, r.o[2]), r.d[0], r.d[1], r.d[2]);
  const float q = __fmul_rn(num, inv_dd);
  return __fmaf_rn(__fmaf_rn(-q, r.dd, num), inv_dd, q);
}

// Clipped bucket range of a hash entry: [x, x + count) within [0, n_sorted).
__device__ __forceinline__ int2 bucket_range(int2 h, int n_sorted) {
  if (h.x < 0 || h.y <= 0 || h.x >= n_sorted) return make_int2(0, 0);
  return make_int2(h.x, h.x + min(h.y, n_sorted - h.x));
}

// Lanes [lo, hi) of a warp as a bit mask (0 <= lo <= hi <= 32).
__device__ __forceinline__ unsigned lane_span(int lo, int hi) {
  const unsigned below_hi = hi >= 32 ? 0xffffffffu : (1u << hi) - 1u;
  const unsigned below_lo = lo >= 32 ? 0xffffffffu : (1u << lo) - 1u;
  return below_hi & ~below_lo;
}

}  // namespace hp

// Host-side helpers shared by the entry points (defined in hp_api.cu).
namespace hp {
int32_t set_error(int32_t code, const char* fmt, ...);
int32_t check_launch(const char* what);
}  // namespace hp
