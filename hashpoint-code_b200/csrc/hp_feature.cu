// Downstream of sampling: the per-sample point-attribute gather and the
// volume-rendering composite.
//
// hp_feature_query replaces FeatureQuery.forward (epcq/epcq.py:345-387).  The
// reference selects the valid samples with boolean indexing, gathers xyz /
// rgb / dir / feat of every selected point id with four torch.gather calls,
// scatters them into zero-filled canvases, and builds the per-pixel ray
// directions (generate_rays, epcq.py:333-341) for the whole image before
// selecting them.  Here the valid samples are numbered by an exclusive scan of
// the mask (hp_mask_scan) and one kernel writes, for each valid sample, its
// sample point, its ray direction, its P validity flags and the P gathered
// attribute rows -- each output element once, point rows read with coalesced
// warp loads.
//
// hp_clamp_t and hp_render replace clamp_t and render (epcq.py:508-529): per
// ray, the sample spacing with out-of-range gaps replaced by vsize, opacity
// 1 - exp(-sigma * delta), transmittance as the running product of
// (1 - opacity + 1e-10), and the weighted colour sum plus the background
// times the transmittance in front of the last sample.  One thread walks one
// ray's samples in order; hp_render can take t values instead of spacings and
// apply clamp_t on the fly.
#include <cuda_fp16.h>

#include "hp_common.cuh"

namespace hp {

constexpr int kScanThreads = 256;
constexpr int kScanPerThread = 16;  // mask bytes per thread (one 16-byte load)
constexpr int kScanTile = kScanThreads * kScanPerThread;

__device__ __forceinline__ int count_bytes(uint4 w) {
  // mask bytes are 0 or 1 (bool); count the nonzero ones
  auto c = [](unsigned x) { return __popc(__vcmpne4(x, 0u) & 0x01010101u); };
  return c(w.x) + c(w.y) + c(w.z) + c(w.w);
}

// Per tile of kScanTile mask bytes: its count.
__global__ void __launch_bounds__(kScanThreads) k_mask_tile_counts(const uint8_t* __restrict__ mask, int64_t n,
                                                                   int* __restrict__ tile_counts) {
  __shared__ int warp_sum[kScanThreads / 32];
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanPerThread;
  int c = 0;
  if (base + kScanPerThread <= n && ((uintptr_t)(mask + base) & 15) == 0) {
    c = count_bytes(*reinterpret_cast<const uint4*>(mask + base));
  } else {
    for (int q = 0; q < kScanPerThread; q++)
      if (base + q < n) c += mask[base + q] != 0;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int w = 0; w < kScanThreads / 32; w++) t += warp_sum[w];
    tile_counts[blockIdx.x] = t;
  }
}

// Exclusive scan of the tile counts in place (one block), total to *count.
__global__ void __launch_bounds__(1024) k_mask_scan_tiles(int* __restrict__ tile_counts, int n_tiles,
                                                          int* __restrict__ count) {
  __shared__ int warp_sum[32];
  const int per = (n_tiles + blockDim.x - 1) / blockDim.x;
  const int b0 = threadIdx.x * per, b1 = min(n_tiles, b0 + per);
  int local = 0;
  for (int i = b0; i < b1; i++) local += tile_counts[i];
  int incl = local;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  int off = 0;
  for (int w = 0; w < warp; w++) off += warp_sum[w];
  int run = off + incl - local;
  for (int i = b0; i < b1; i++) {
    const int c = tile_counts[i];
    tile_counts[i] = run;
    run += c;
  }
  if (threadIdx.x == blockDim.x - 1) *count = run;
}

// offsets[i] = valid samples before i (tile base + block-local exclusive scan).
// kSum: `tile` holds the tiles' counts, and each block adds up those before its
// own (a few loads a thread while there are at most kSumTiles, and one launch
// less: FeatureQuery over 5.1M samples went from 299 us to 293, with wider feature stores); the
// last block writes the total.  Else `tile` holds their scan.
constexpr int kSumTiles = 4096;
template <bool kSum>
__global__ void __launch_bounds__(kScanThreads) k_mask_offsets(const uint8_t* __restrict__ mask, int64_t n,
                                                               const int* __restrict__ tile, int* __restrict__ offsets,
                                                               int* __restrict__ count) {
  int tile_base = 0;
  if constexpr (kSum) {
    __shared__ int part[kScanThreads / 32];
    int sum = 0;
    for (int q = threadIdx.x; q < (int)blockIdx.x; q += kScanThreads) sum += __ldg(tile + q);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sum;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; w++) tile_base += part[w];
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *count = tile_base + __ldg(tile + blockIdx.x);
  } else {
    tile_base = __ldg(tile + blockIdx.x);
  }
  // A warp takes 512 mask bytes in four passes of 128 (four a lane), so that each
  // load and store instruction covers whole lines.  A pass counts at most 128:
  // the four passes' counts scan as the bytes of one word.
  constexpr int kPasses = kScanPerThread / 4;
  static_assert(kPasses == 4, "a byte per pass");
  __shared__ int warp_sum[kScanThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t base = (int64_t)blockIdx.x * kScanTile + warp * (32 * kScanPerThread) + 4 * lane;
  const bool aligned = (((uintptr_t)mask & 3) | ((uintptr_t)offsets & 15)) == 0;
  unsigned w[kPasses], local = 0;
#pragma unroll
  for (int k = 0; k < kPasses; k++) {
    const int64_t i = base + 128 * k;
    w[k] = 0;
    if (aligned && i + 4 <= n) {
      w[k] = __vcmpne4(__ldg(reinterpret_cast<const unsigned*>(mask + i)), 0u) & 0x01010101u;
    } else {
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (i + q < n) w[k] |= (unsigned)(mask[i + q] != 0) << (8 * q);
    }
    local |= (unsigned)__popc(w[k]) << (8 * k);
  }
  unsigned incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  const unsigned total = __shfl_sync(0xffffffffu, incl, 31);
  auto byte = [](unsigned x, int k) { return (int)((x >> (8 * k)) & 0xffu); };
  if (lane == 0) warp_sum[warp] = byte(total, 0) + byte(total, 1) + byte(total, 2) + byte(total, 3);
  __syncthreads();
  int run = tile_base;
#pragma unroll
  for (int v = 0; v < kScanThreads / 32; v++)
    if (v < warp) run += warp_sum[v];
  incl -= local;  // exclusive, byte by byte: no borrow
#pragma unroll
  for (int k = 0; k < kPasses; k++) {
    const int64_t i = base + 128 * k;
    const int o0 = run + byte(incl, k), o1 = o0 + (int)(w[k] & 1u);
    const int o2 = o1 + (int)((w[k] >> 8) & 1u), o3 = o2 + (int)((w[k] >> 16) & 1u);
    if (aligned && i + 4 <= n) {
      *reinterpret_cast<int4*>(offsets + i) = make_int4(o0, o1, o2, o3);
    } else {
      if (i < n) offsets[i] = o0;
      if (i + 1 < n) offsets[i + 1] = o1;
      if (i + 2 < n) offsets[i + 2] = o2;
      if (i + 3 < n) offsets[i + 3] = o3;
    }
    run += byte(total, k);
  }
}

struct FeatArgs {
  const float* xyz;
  const float* rgb;
  const float* dir;
  const void* feat;
  int feat_dim, feat_half;
  int n_points;
  const float* sp_xyz;
  const int* pc_idx;
  const uint8_t* mask;
  const int* offsets;
  int64_t n_samples;  // rays * S
  int S, P;
  const float* c2w;
  float fx, fy, cx, cy;
  int width;
  const int* ray_uv;  // [rays, 2] (u, v) or null: ray r is pixel (r % width, r / width)
  float* o_xyz;
  float* o_rgb;
  float* o_dir;
  float* o_feat;
  float* o_sp;
  uint8_t* o_valid;
  float* o_rays;
};

// One warp per 32 consecutive samples; the warp serves their valid ones in
// turn, spreading each sample's outputs over its lanes.
__global__ void __launch_bounds__(256) k_feature_query(FeatArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t i0 = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * 32;
  if (i0 >= a.n_samples) return;
  const int64_t my = i0 + lane;
  const bool valid = my < a.n_samples && a.mask[my] != 0;
  unsigned todo = __ballot_sync(0xffffffffu, valid);
  const int my_off = valid ? a.offsets[my] : 0;
  const int P = a.P, F = a.feat_dim;
  while (todo) {
    const int l = __ffs(todo) - 1;
    todo &= todo - 1;
    const int64_t i = i0 + l;
    const int64_t m = __shfl_sync(0xffffffffu, my_off, l);
    const unsigned ray = (unsigned)i / (unsigned)a.S;  // sample counts are below 2^31: 32-bit division
    // sample point and ray direction (generate_rays: ((u - cx) / fx, (v - cy) / fy, 1) rotated by c2w)
    if (lane < 3) a.o_sp[m * 3 + lane] = a.sp_xyz[i * 3 + lane];
    if (lane >= 3 && lane < 6) {
      const int c = lane - 3;
      int u, v;
      if (a.ray_uv) {
        u = a.ray_uv[2 * (int64_t)ray];
        v = a.ray_uv[2 * (int64_t)ray + 1];
      } else {
        v = (int)(ray / (unsigned)a.width);
        u = (int)(ray - (unsigned)v * (unsigned)a.width);
      }
      const float dx = __fdiv_rn(__fsub_rn((float)u, a.cx), a.fx);
      const float dy = __fdiv_rn(__fsub_rn((float)v, a.cy), a.fy);
      const float* R = a.c2w + 4 * c;
      a.o_rays[m * 3 + c] = __fadd_rn(__fadd_rn(__fmul_rn(dx, R[0]), __fmul_rn(dy, R[1])), R[2]);
    }
    // validity flags and xyz / rgb / dir rows: lane = (point, component) over 3 * P lanes per pass
    const int* ids = a.pc_idx + i * P;
    for (int e = lane; e < 3 * P; e += 32) {
      const int p = e / 3, c = e - 3 * p;
      const int id = ids[p];
      const bool ok = (unsigned)id < (unsigned)a.n_points;
      if (c == 0) a.o_valid[m * P + p] = ok;
      const int64_t o = (m * P + p) * 3 + c;
      a.o_xyz[o] = ok ? a.xyz[(int64_t)id * 3 + c] : 0.0f;
      a.o_rgb[o] = ok ? a.rgb[(int64_t)id * 3 + c] : 0.0f;
      a.o_dir[o] = ok ? a.dir[(int64_t)id * 3 + c] : 0.0f;
    }
    // feature rows: P * F consecutive floats
    float* of = a.o_feat + m * P * F;
    for (int e = lane; e < P * F; e += 32) {
      const int p = e / F, f = e - p * F;
      const int id = ids[p];
      float val = 0.0f;
      if ((unsigned)id < (unsigned)a.n_points) {
        if (a.feat_half)
          val = __half2float(reinterpret_cast<const __half*>(a.feat)[(int64_t)id * F + f]);
        else
          val = reinterpret_cast<const float*>(a.feat)[(int64_t)id * F + f];
      }
      of[e] = val;
    }
  }
}

// Four features, as the gather moves them: one float4 out.
template <int kHalf>
struct FeatPiece {
  using type = float4;
};
template <>
struct FeatPiece<1> {
  using type = uint2;
};

// The same gather with 16-byte stores, for feature rows whose bytes are a
// multiple of 16 (F = 32 fp16 or fp32 features, the Aggregator's width).
//
// Bound by how many gathers are in flight.  A block lists the valid ones of its
// 128 samples, so that its warps share them evenly however the mask clumps, and
// eight lanes serve a sample: nine words of the point attributes and kPieces
// feature pieces a lane are loaded before any is stored (at P = 8 and F = 32 one
// round each; the fp16 pieces are 8-byte loads, whose widened stores fill whole
// lines).  What a sample has one of (position, ray direction with its divisions)
// is done by a thread a sample beforehand.  The outputs are stored past the L2's
// table (streaming).  613k samples of 8 points with 32 fp16 features from 1M
// points, the whole call: 304 us when a warp served its own 32 samples in pairs
// with both halves' loads two deep, 256 with 16 lanes a sample, 252 so;
// one lane a word, or ids fetched a sample ahead, made it 310 to 357 (less in
// flight, fewer warps).
constexpr int kVecBlock = 128;
template <int kHalf>
__global__ void __launch_bounds__(kVecBlock, 12) k_feature_query_vec(FeatArgs a) {
  using Piece = typename FeatPiece<kHalf>::type;
  constexpr int kPieces = kHalf ? 8 : 4;  // 16 registers either way
  __shared__ uint8_t list[kVecBlock];  // the block's valid samples in order
  __shared__ int rows[kVecBlock];     // and their output rows
  __shared__ int counts[kVecBlock / 32];
  const int lane = threadIdx.x & 31, hl = lane & 7, warp = threadIdx.x >> 5;
  const int64_t i0 = (int64_t)blockIdx.x * kVecBlock;
  const bool valid = i0 + threadIdx.x < a.n_samples && a.mask[i0 + threadIdx.x] != 0;
  const unsigned votes = __ballot_sync(0xffffffffu, valid);
  if (lane == 0) counts[warp] = __popc(votes);
  __syncthreads();
  int before = 0, n_valid = 0;
#pragma unroll
  for (int w = 0; w < kVecBlock / 32; w++) {
    if (w < warp) before += counts[w];
    n_valid += counts[w];
  }
  if (valid) {  // what a sample has one of: a thread each, the warp's together
    const int k = before + __popc(votes & ((1u << lane) - 1));
    list[k] = (uint8_t)threadIdx.x;
    const int64_t i = i0 + threadIdx.x, m = a.offsets[i];
    rows[k] = (int)m;
    const unsigned ray = (unsigned)i / (unsigned)a.S;  // sample counts are below 2^31: 32-bit division
    int u, v;
    if (a.ray_uv) {
      u = a.ray_uv[2 * (int64_t)ray];
      v = a.ray_uv[2 * (int64_t)ray + 1];
    } else {
      v = (int)(ray / (unsigned)a.width);
      u = (int)(ray - (unsigned)v * (unsigned)a.width);
    }
    const float dx = __fdiv_rn(__fsub_rn((float)u, a.cx), a.fx);
    const float dy = __fdiv_rn(__fsub_rn((float)v, a.cy), a.fy);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const float* R = a.c2w + 4 * c;
      a.o_rays[m * 3 + c] = __fadd_rn(__fadd_rn(__fmul_rn(dx, R[0]), __fmul_rn(dy, R[1])), R[2]);
      a.o_sp[m * 3 + c] = a.sp_xyz[i * 3 + c];
    }
  }
  __syncthreads();
  const int P = a.P, F = a.feat_dim;
  const int cpp = F / 4;  // pieces (four features) per feature row
  const int cshift = (cpp & (cpp - 1)) == 0 ? __ffs(cpp) - 1 : -1;  // log2(cpp) when a power of two
  const int nch = P * cpp;
  const char* feat = reinterpret_cast<const char*>(a.feat);
  for (int k = threadIdx.x >> 3; k < n_valid; k += kVecBlock / 8) {
    const int64_t m = rows[k], i = i0 + list[k];
    const int* ids = a.pc_idx + i * P;  // the same few words for the eight lanes (L1)
    // xyz / rgb / dir rows: element e = (point, component), three per lane per pass
    for (int e = hl; e < 3 * P; e += 24) {
      float x[3], g[3], d[3];
      bool ok[3];
#pragma unroll
      for (int h = 0; h < 3; h++) {
        const int ee = e + 8 * h;
        x[h] = g[h] = d[h] = 0.0f;
        ok[h] = false;
        if (ee < 3 * P) {
          const int p = ee / 3, c = ee - 3 * p;
          const int id = ids[p];
          ok[h] = (unsigned)id < (unsigned)a.n_points;
          if (ok[h]) {
            x[h] = a.xyz[(int64_t)id * 3 + c];
            g[h] = a.rgb[(int64_t)id * 3 + c];
            d[h] = a.dir[(int64_t)id * 3 + c];
          }
        }
      }
#pragma unroll
      for (int h = 0; h < 3; h++) {
        const int ee = e + 8 * h;
        if (ee < 3 * P) {
          const int p = ee / 3, c = ee - 3 * p;
          if (c == 0) a.o_valid[m * P + p] = ok[h];
          const int64_t o = (m * P + p) * 3 + c;
          __stcs(a.o_xyz + o, x[h]);
          __stcs(a.o_rgb + o, g[h]);
          __stcs(a.o_dir + o, d[h]);
        }
      }
    }
    // feature rows: piece q of point p, kPieces per lane in flight; each store instruction covers whole lines
    float* of = a.o_feat + m * P * F;
    for (int c = hl; c < nch; c += 8 * kPieces) {
      Piece v[kPieces];
#pragma unroll
      for (int h = 0; h < kPieces; h++) {
        const int cc = c + 8 * h;
        v[h] = Piece{};
        if (cc < nch) {
          const int p = cshift >= 0 ? cc >> cshift : cc / cpp, q = cc - p * cpp;
          const int id = ids[p];
          if ((unsigned)id < (unsigned)a.n_points)
            v[h] = __ldg(reinterpret_cast<const Piece*>(feat) + ((int64_t)id * cpp + q));
        }
      }
#pragma unroll
      for (int h = 0; h < kPieces; h++) {
        const int cc = c + 8 * h;
        if (cc < nch) {  // piece cc of the sample's rows is its floats 4 cc .. + 3
          if constexpr (kHalf) {
            const __half2* hh = reinterpret_cast<const __half2*>(&v[h]);
            const float2 f0 = __half22float2(hh[0]), f1 = __half22float2(hh[1]);
            __stcs(reinterpret_cast<float4*>(of) + cc, make_float4(f0.x, f0.y, f1.x, f1.y));
          } else {
            __stcs(reinterpret_cast<float4*>(of) + cc, v[h]);
          }
        }
      }
    }
  }
}

// clamp_t: gaps outside (1e-8, 2 vsize], and the last sample's, become vsize.
__device__ __forceinline__ float clamp_gap(float d, float vsize) {
  const float m = (d < 1e-8f || d > __fmul_rn(2.0f, vsize)) ? 1.0f : 0.0f;
  return __fadd_rn(__fmul_rn(d, __fsub_rn(1.0f, m)), __fmul_rn(m, vsize));
}

__device__ __forceinline__ float clamped_gap(const float* t, int s, int S, float vsize) {
  return clamp_gap(s + 1 < S ? __fsub_rn(t[s + 1], t[s]) : vsize, vsize);
}

// Four consecutive elements per thread, whatever S: one 16-byte load (the
// element after them comes from the next lane, lane 31 loads its own) and one
// 16-byte store.  Unaligned arrays (kVec 0) go one by one, 256 apart.  HBM
// bounds it: 640,000 x 8 (41 MB) in 11 us as ncu times the launch, 18.5 us with
// one element and one modulo a thread.
template <int kVec>
__global__ void __launch_bounds__(256) k_clamp_t(const float* __restrict__ t_val, int64_t n, int S, float vsize,
                                                 float* __restrict__ out) {
  const int64_t block0 = (int64_t)blockIdx.x * 1024;
  const int64_t i = block0 + (kVec ? threadIdx.x * 4 : threadIdx.x);
  auto slot = [&](int64_t e) { return e < 0x7fffffff ? (int)((unsigned)e % (unsigned)S) : (int)(e % S); };
  if constexpr (kVec) {
    const bool whole = i + 4 <= n;
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    if (whole) t = *reinterpret_cast<const float4*>(t_val + i);
    float next = __shfl_down_sync(0xffffffffu, t.x, 1);
    const bool next_whole = __shfl_down_sync(0xffffffffu, whole, 1);
    if (i >= n) return;
    int s = slot(i);
    if (whole) {
      if (((threadIdx.x & 31) == 31 || !next_whole) && i + 4 < n) next = t_val[i + 4];
      const float v[5] = {t.x, t.y, t.z, t.w, next};
      float g[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        g[q] = clamp_gap(s + 1 < S ? __fsub_rn(v[q + 1], v[q]) : vsize, vsize);
        s = s + 1 < S ? s + 1 : 0;
      }
      *reinterpret_cast<float4*>(out + i) = make_float4(g[0], g[1], g[2], g[3]);
    } else {
      for (int64_t e = i; e < n; e++) {
        out[e] = clamped_gap(t_val + (e - s), s, S, vsize);
        s = s + 1 < S ? s + 1 : 0;
      }
    }
  } else {
    for (int64_t e = i; e < n && e < block0 + 1024; e += 256) {
      const int s = slot(e);
      out[e] = clamped_gap(t_val + (e - s), s, S, vsize);
    }
  }
}

// render (with the deltas given, or derived from t_val by clamp_t when deltas is null)
__global__ void k_render(const float* __restrict__ deltas, const float* __restrict__ t_val, float vsize,
                         const float* __restrict__ sigmas, const float* __restrict__ rgbs, int64_t rays, int S,
                         int white_bg, float* __restrict__ color) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rays) return;
  float trans = 1.0f;  // transmittance before this sample
  float bg_trans = 1.0f;  // the background sees the transmittance before the last sample
  float c0 = 0.0f, c1 = 0.0f, c2 = 0.0f;
  for (int s = 0; s < S; s++) {
    bg_trans = trans;
    const float d = deltas ? deltas[r * S + s] : clamped_gap(t_val + r * S, s, S, vsize);
    const float opacity = __fsub_rn(1.0f, expf(__fmul_rn(-sigmas[r * S + s], d)));
    const float w = __fmul_rn(opacity, trans);
    const float* c = rgbs + (r * S + s) * 3;
    c0 = __fadd_rn(c0, __fmul_rn(w, c[0]));
    c1 = __fadd_rn(c1, __fmul_rn(w, c[1]));
    c2 = __fadd_rn(c2, __fmul_rn(w, c[2]));
    trans = __fmul_rn(trans, __fadd_rn(__fsub_rn(1.0f, opacity), 1e-10f));
  }
  const float bg = white_bg ? 1.0f : 0.0f;
  color[r * 3 + 0] = __fadd_rn(c0, __fmul_rn(bg_trans, bg));
  color[r * 3 + 1] = __fadd_rn(c1, __fmul_rn(bg_trans, bg));
  color[r * 3 + 2] = __fadd_rn(c2, __fmul_rn(bg_trans, bg));
}

// The same for S = kS (a multiple of 4) with 16-byte aligned bases: a ray's
// sigma, t (or delta) and rgb rows are loaded as 16-byte vectors before any
// arithmetic, so a thread waits on one round of loads instead of one per
// sample; the arithmetic and its order are k_render's.
template <int kS>
__global__ void __launch_bounds__(256) k_render_vec(const float* __restrict__ deltas, const float* __restrict__ t_val,
                                                    float vsize, const float* __restrict__ sigmas,
                                                    const float* __restrict__ rgbs, int64_t rays, int white_bg,
                                                    float* __restrict__ color) {
  static_assert(kS % 4 == 0, "kS must be a multiple of 4");
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rays) return;
  float sg[kS], tv[kS], cl[3 * kS];
  const float4* s4 = reinterpret_cast<const float4*>(sigmas + r * kS);
  const float4* t4 = reinterpret_cast<const float4*>((deltas ? deltas : t_val) + r * kS);
  const float4* c4 = reinterpret_cast<const float4*>(rgbs + r * kS * 3);
#pragma unroll
  for (int q = 0; q < kS / 4; q++) {
    const float4 x = __ldg(s4 + q), y = __ldg(t4 + q);
    sg[4 * q] = x.x, sg[4 * q + 1] = x.y, sg[4 * q + 2] = x.z, sg[4 * q + 3] = x.w;
    tv[4 * q] = y.x, tv[4 * q + 1] = y.y, tv[4 * q + 2] = y.z, tv[4 * q + 3] = y.w;
  }
#pragma unroll
  for (int q = 0; q < 3 * kS / 4; q++) {
    const float4 x = __ldg(c4 + q);
    cl[4 * q] = x.x, cl[4 * q + 1] = x.y, cl[4 * q + 2] = x.z, cl[4 * q + 3] = x.w;
  }
  float trans = 1.0f, bg_trans = 1.0f;
  float c0 = 0.0f, c1 = 0.0f, c2 = 0.0f;
#pragma unroll
  for (int s = 0; s < kS; s++) {
    bg_trans = trans;
    const float d = deltas ? tv[s] : clamped_gap(tv, s, kS, vsize);
    const float opacity = __fsub_rn(1.0f, expf(__fmul_rn(-sg[s], d)));
    const float w = __fmul_rn(opacity, trans);
    c0 = __fadd_rn(c0, __fmul_rn(w, cl[3 * s]));
    c1 = __fadd_rn(c1, __fmul_rn(w, cl[3 * s + 1]));
    c2 = __fadd_rn(c2, __fmul_rn(w, cl[3 * s + 2]));
    trans = __fmul_rn(trans, __fadd_rn(__fsub_rn(1.0f, opacity), 1e-10f));
  }
  const float bg = white_bg ? 1.0f : 0.0f;
  color[r * 3 + 0] = __fadd_rn(c0, __fmul_rn(bg_trans, bg));
  color[r * 3 + 1] = __fadd_rn(c1, __fmul_rn(bg_trans, bg));
  color[r * 3 + 2] = __fadd_rn(c2, __fmul_rn(bg_trans, bg));
}

}  // namespace hp

using namespace hp;

static size_t mask_tiles(int64_t n) { return (size_t)((n + kScanTile - 1) / kScanTile); }

extern "C" size_t hp_mask_scan_workspace_size(int64_t n) {
  if (n < 0) return 0;
  return ((mask_tiles(n) + 1) * sizeof(int) + 255) & ~(size_t)255;
}

extern "C" int32_t hp_mask_scan(const uint8_t* mask, int64_t n, int32_t* offsets, int32_t* count, void* workspace,
                                size_t workspace_bytes, hp_stream_t stream) {
  if (n < 0 || n >= (1ll << 31)) return set_error(HP_ERR_INVALID_ARGUMENT, "hp_mask_scan: n out of range");
  if ((n > 0 && (!mask || !offsets)) || !count)
    return set_error(HP_ERR_INVALID_ARGUMENT, "hp_mask_scan: null pointer");
  if (!workspace || workspace_bytes < hp_mask_scan_workspace_size(n))
    return set_error(HP_ERR_WORKSPACE, "hp_mask_scan: workspace needs %zu bytes", hp_mask_scan_workspace_size(n));
  cudaStream_t st = (cudaStream_t)stream;
  const int tiles = (int)mask_tiles(n);
  int* tile = (int*)workspace;
  if (tiles == 0) {
    if (cudaMemsetAsync(count, 0, sizeof(int32_t), st) != cudaSuccess)
      return set_error(HP_ERR_CUDA, "hp_mask_scan: memset failed");
    return HP_OK;
  }
  k_mask_tile_counts<<<tiles, kScanThreads, 0, st>>>(mask, n, tile);
  if (int32_t rc = check_launch("k_mask_tile_counts")) return rc;
  if (tiles <= kSumTiles) {
    k_mask_offsets<true><<<tiles, kScanThreads, 0, st>>>(mask, n, tile, offsets, count);
    return check_launch("k_mask_offsets");
  }
  k_mask_scan_tiles<<<1, 1024, 0, st>>>(tile, tiles, count);
  if (int32_t rc = check_launch("k_mask_scan_tiles")) return rc;
  k_mask_offsets<false><<<tiles, kScanThreads, 0, st>>>(mask, n, tile, offsets, count);
  return check_launch("k_mask_offsets");
}

extern "C" int32_t hp_feature_query(const hp_point_attrs* pts, const float* sp_xyz, const int32_t* pc_idx,
                                    const uint8_t* mask, int64_t n_rays, int32_t S, int32_t P,
                                    const int32_t* offsets, const hp_camera* cam, const int32_t* ray_uv,
                                    float* pc_xyz, float* pc_rgb, float* pc_dir, float* pc_feat, float* out_sp_xyz,
                                    uint8_t* valid, float* rays_d, hp_stream_t stream) {
  static const char* who = "hp_feature_query";
  if (!pts || !cam) return set_error(HP_ERR_INVALID_ARGUMENT, "%s: null pointer", who);
  if (n_rays < 0 || S < 1 || P < 1 || n_rays * S >= (1ll << 31) || pts->n_points < 0 || pts->n_points >= (1ll << 31) ||
      pts->feat_dim < 0)
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: sizes out of range", who);
  if (!cam->c2w || (!ray_uv && cam->width <= 0) || !(cam->fx != 0.0f) || !(cam->fy != 0.0f))
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: bad camera", who);
  if (n_rays == 0) return HP_OK;
  if (!sp_xyz || !pc_idx || !mask || !offsets || !pc_xyz || !pc_rgb || !pc_dir || !out_sp_xyz || !valid || !rays_d ||
      (pts->feat_dim > 0 && (!pc_feat || !pts->feat)) || (pts->n_points > 0 && (!pts->xyz || !pts->rgb || !pts->dir)))
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: null pointer", who);
  FeatArgs a;
  a.xyz = pts->xyz;
  a.rgb = pts->rgb;
  a.dir = pts->dir;
  a.feat = pts->feat;
  a.feat_dim = pts->feat_dim;
  a.feat_half = pts->feat_half;
  a.n_points = (int)pts->n_points;
  a.sp_xyz = sp_xyz;
  a.pc_idx = pc_idx;
  a.mask = mask;
  a.offsets = offsets;
  a.n_samples = n_rays * S;
  a.S = S;
  a.P = P;
  a.c2w = cam->c2w;
  a.fx = cam->fx;
  a.fy = cam->fy;
  a.cx = cam->cx;
  a.cy = cam->cy;
  a.width = cam->width;
  a.ray_uv = ray_uv;
  a.o_xyz = pc_xyz;
  a.o_rgb = pc_rgb;
  a.o_dir = pc_dir;
  a.o_feat = pc_feat;
  a.o_sp = out_sp_xyz;
  a.o_valid = valid;
  a.o_rays = rays_d;
  const int64_t warps = (a.n_samples + 31) / 32;
  const int esz = a.feat_half ? 2 : 4;
  // 16-byte moves when the rows and both base addresses allow them
  const bool vec = a.feat_dim > 0 && (a.feat_dim * esz) % 16 == 0 && ((uintptr_t)a.feat & 15) == 0 &&
                   ((uintptr_t)a.o_feat & 15) == 0;
  if (vec && a.feat_half)
    k_feature_query_vec<1><<<(unsigned)((a.n_samples + kVecBlock - 1) / kVecBlock), kVecBlock, 0, (cudaStream_t)stream>>>(a);
  else if (vec)
    k_feature_query_vec<0><<<(unsigned)((a.n_samples + kVecBlock - 1) / kVecBlock), kVecBlock, 0, (cudaStream_t)stream>>>(a);
  else
    k_feature_query<<<(unsigned)((warps + 7) / 8), 256, 0, (cudaStream_t)stream>>>(a);
  return check_launch("k_feature_query");
}

extern "C" int32_t hp_clamp_t(const float* t_val, int64_t n_rays, int32_t S, float vsize, float* t_dist,
                              hp_stream_t stream) {
  if (n_rays < 0 || S < 1 || n_rays * S >= (1ll << 39))
    return set_error(HP_ERR_INVALID_ARGUMENT, "hp_clamp_t: sizes out of range");
  if (n_rays == 0) return HP_OK;
  if (!t_val || !t_dist) return set_error(HP_ERR_INVALID_ARGUMENT, "hp_clamp_t: null pointer");
  const unsigned blocks = (unsigned)((n_rays * S + 1023) / 1024);
  if ((((uintptr_t)t_val | (uintptr_t)t_dist) & 15) == 0)
    k_clamp_t<1><<<blocks, 256, 0, (cudaStream_t)stream>>>(t_val, n_rays * S, S, vsize, t_dist);
  else
    k_clamp_t<0><<<blocks, 256, 0, (cudaStream_t)stream>>>(t_val, n_rays * S, S, vsize, t_dist);
  return check_launch("k_clamp_t");
}

extern "C" int32_t hp_render(const float* deltas, const float* t_val, float vsize, const float* sigmas,
                             const float* rgbs, int64_t n_rays, int32_t S, int32_t white_bg, float* color,
                             hp_stream_t stream) {
  if (n_rays < 0 || S < 1) return set_error(HP_ERR_INVALID_ARGUMENT, "hp_render: sizes out of range");
  if (n_rays == 0) return HP_OK;
  if ((!deltas && !t_val) || !sigmas || !rgbs || !color)
    return set_error(HP_ERR_INVALID_ARGUMENT, "hp_render: null pointer");
  const unsigned blocks = (unsigned)((n_rays + 255) / 256);
  cudaStream_t st = (cudaStream_t)stream;
  const bool aligned = (((uintptr_t)(deltas ? deltas : t_val) | (uintptr_t)sigmas | (uintptr_t)rgbs) & 15) == 0;
  if (aligned && S == 8)
    k_render_vec<8><<<blocks, 256, 0, st>>>(deltas, t_val, vsize, sigmas, rgbs, n_rays, white_bg, color);
  else if (aligned && S == 16)
    k_render_vec<16><<<blocks, 256, 0, st>>>(deltas, t_val, vsize, sigmas, rgbs, n_rays, white_bg, color);
  else if (aligned && S == 4)
    k_render_vec<4><<<blocks, 256, 0, st>>>(deltas, t_val, vsize, sigmas, rgbs, n_rays, white_bg, color);
  else
    k_render<<<blocks, 256, 0, st>>>(deltas, t_val, vsize, sigmas, rgbs, n_rays, S, white_bg, color);
  return check_launch("k_render");
}
