// Window search, primary-surface selection, K-sample emission and per-sample
// point selection.
//
// Replaces _C.quick_sampling (epcq/csrc/epcq_render_topk.cu:341-417), which
// zero-fills all four outputs, runs quick_sampling_kernel (:82-220, one warp
// per ray, one lane per window cell, a 128-bin shared-memory histogram built
// with float atomics and a serial walk on lane 0) and then
// quick_search_nearby_pc (:10-81, one thread per (ray, sample slot) re-walking
// the window).  Here a launch is two kernels:
//
//   k_ray_list        one block per 256-pixel tile: each ray's window candidate
//                count from the hash table; rays without any get their default
//                outputs (coalesced runs), the others go into a list with
//                their directions, a tile's rays ordered by count
//   k_quick_sampling  persistent warps take rays from the list.  A ray with few
//                candidates is served by 8 lanes (four rays a warp), a heavy
//                one by the whole warp; lanes stand for candidates (what the
//                fast arithmetic cannot decide is done again by serve_exact, a
//                ray whose list overflows by sample_ray_warp):
//
//   pass A  every candidate of the window (rows of cells are runs of the
//           sorted ids) is tested against the ray once; those within the
//           radius -- at most 48 per window cell -- are "kept" and give tmin.
//           The kept ones, and the few just outside the radius or beyond a
//           cell's 48, are listed (indices, in window order) in shared memory:
//           no later pass looks at any other candidate
//   bins    int((t - tmin) / t_intvl) of the kept entries: a histogram in
//           shared memory of counts and quantised distance sums
//   walk    bins with >= 2 points in ascending order: alpha = gamma *
//           exp(-mean_dist / alpha_g), emit when alpha * T > 1e-3, T -= alpha,
//           stop when T < 1e-3 or S samples are out
//   ball    per sample, the reference's 8-entry id buffer over the listed
//           candidates, with its quirk that, while the buffer fills, the
//           tracked "farthest" entry is the nearest one.  The hits go to shared
//           memory in order; 8 lanes hold the buffer in ascending distance, so
//           a replacement is one ballot and one shift
//
// The candidates the ball query can take are within the radius of a point of
// the ray, so they are within the radius of the ray up to float error, and the
// list's margin (see near_limit) is orders of magnitude above that: each
// buffer sees exactly the sequence of the full window walk.
//
// What bounds it is instruction issue, then the latency of the candidates'
// first touch.  One thread per ray (tiles staged in shared memory, 32 rays of a
// window-size class a warp) left half the lanes idle -- every window row and
// buffer replacement waited for the longest lane -- and its blocks idle at
// each tile's end; with lanes as candidates 30 of 32 lanes are active and there
// is no barrier.  1M points, 800 x 800, radius 0.008: 1000 us -> 418 us (446 M
// -> 337 M warp instructions, 54% -> 73% of the issue slots); 4M points at
// 512 x 512: 4470 -> 1103 us; 100k points, 3 x 3 window: 193 -> 57 us.  Measured
// and not kept: the listed candidates themselves in shared memory (20 bytes an
// entry leave too little L1: 780-1010 us on the first view), re-walking the
// window in every pass instead of a list (760-850 us), copies of the code per
// lane count (instruction-cache misses: 560-620 us), two samples a ball pass
// (registers: 662-730 us).
//
// Bin sums are accumulated in window-cell then bucket order; the reference
// adds them with shared-memory atomics in an unspecified order, so a bin's
// mean distance can differ from the reference's in the last bit -- which moves
// an output only if alpha * T or T sits within that bit of 1e-3.
#include <cmath>
#include <cstdio>
#include <mutex>

#include "hp_common.cuh"

namespace hp {

constexpr int kTeReg = 4;        // emitted sample depths kept in registers (sample_ray_warp)
constexpr int kBallPass = 2;     // samples served by one ball-query walk
constexpr int kHeavyWindow = 240;  // default: rays with more window candidates get a whole warp (8 lanes hold 240 to 256)
constexpr int kMaxHeavyWindow = 4096;  // largest tunable threshold
constexpr int kWalkBatch = 4;    // bins whose sums one walk pass of sample_ray_warp gathers
constexpr int kClasses = 64;     // window-size classes a tile's rays are ordered by
constexpr int kThreads = 256;    // pixels of a tile, threads per block of the list kernels
constexpr int kWarps = kThreads / 32;
constexpr int kServeThreads = 128;  // threads per block of the serving kernels
constexpr int kServeWarps = kServeThreads / 32;
constexpr int64_t kMaxTilesPerView = 1 << 21;
constexpr int kHistWords = 512;  // per warp: the rays' bin histograms, then their ball hits

// t-bin index int((t - tmin) / t_intvl) of a kept candidate (x = t - tmin >= 0).
// y = x * RN(1 / t_intvl) is within 3.1 * 2^-24 * q of the quotient q and of
// its rounding RN(q), so when y widened by 2^-21 relative on both sides
// truncates to one integer, that integer is int(RN(q)); otherwise (a bin
// edge within a few ulps) the division is done exactly.
struct BinDiv {
  float intvl, inv;
  bool fast;
};

struct SampleArgs {
  const float* __restrict__ xyz;
  const int* __restrict__ sidx;
  const float4* __restrict__ pts;  // sorted_point_idx packed: (x, y, z, id as int bits; -1 = invalid)
  const int2* __restrict__ hash;
  int n_points;  // ids outside [0, n_points) are skipped
  int n_sorted;  // bucket ranges are clipped to [0, n_sorted)
  DevCamera cam;
  DevOptions opt;
  float* __restrict__ sp_xyz;
  int* __restrict__ pc_idx;
  float* __restrict__ sp_t;
  uint8_t* __restrict__ mask;
  // derived from the options once per launch (derive_args)
  RadiusTest rt;
  BinDiv bins;
  float near0;   // near_limit's constant part
  float quanta;  // 1 / radius
  unsigned inv_idx, inv_xyz, inv_t;  // inverse_of the words a ray has in pc_idx, sp_xyz and sp_t
  float eps;     // relative error of alpha from a mean distance off by one part of the radius (serve_rays)
};

// The rays to serve, each as (ray, direction bits): those of 8 lanes in units
// of four from the front (a tile's last unit is filled up with ray -1), those
// of a whole warp from the back.
struct RayList {
  int4* rays;
  long long cap;
  unsigned* counts;  // [4]: front entries, back entries, next front unit, next back entry to serve
  int* front_view;   // batched launches: view of each front unit
  int* back_view;    // and of each back entry
  int light;         // rays with more window candidates than this are served by a whole warp
};

// Stage configurations: a block's warps hold kStage listed candidates on chip
// (a quarter of a warp's per ray served by 8 lanes) at kBlocks blocks of
// kServeThreads per SM, and the ray list is built over kTileH x kTileW pixel
// tiles.  Registers per thread follow from the resident threads (64, 80, 96):
// fewer warps spill less but hide less of the candidates' latency.  960 entries
// a warp: with 640, 4M-point views at 512 x 512 lose 22% to rays whose list
// overflows; shapes and sphere views are level, the 3M-point clustered view
// gains 5% (less shared memory leaves more L1).
template <int kStage_, int kBlocks_, int kTileH_, int kTileW_, class Index_ = int>
struct StageCfg {
  using Index = Index_;  // numbers the candidates of a window in the general walk
  static constexpr int kStage = kStage_;
  static constexpr int kBlocks = kBlocks_;
  static constexpr int kTileH = kTileH_;
  static constexpr int kTileW = kTileW_;
  static constexpr int kEntries = kStage / kServeWarps;  // per warp
  static constexpr int kWarpBytes = kEntries * 4 + kHistWords * 4;
  static constexpr int kSmem = kServeWarps * kWarpBytes;
  static_assert(kTileH * kTileW == kThreads && kEntries % 32 == 0 && kEntries <= 1024 && kBlocks * (kSmem + 1024) <= 227 * 1024, "stage");
};
using Cfg1 = StageCfg<3840, 8, 8, 32>;
using Cfg2 = StageCfg<3968, 6, 8, 32>;
using Cfg3 = StageCfg<4096, 5, 8, 32>;
using Cfg4 = StageCfg<3840, 8, 16, 16>;
using Cfg5 = StageCfg<3968, 6, 16, 16>;
constexpr int kStageConfigs = 5;  // hp_tuning.stage_config 1..5 (0 = the default)
constexpr int kDefaultStageConfig = 4;
// Clamped window cells repeat a bucket (and tables may overlap), so a window's
// 25 cells can hold 25 times the id list: up to 2^26 ids an int numbers them,
// beyond that the default configuration with a walk in 64-bit indices serves
// the view.  (Called from the same kernel, that walk cost the other rays 3%.)
#ifdef HP_TESTING
constexpr int64_t kIntIds = 40;
#else
constexpr int64_t kIntIds = 1 << 26;
#endif
using CfgWide = StageCfg<Cfg4::kStage, Cfg4::kBlocks, Cfg4::kTileH, Cfg4::kTileW, long long>;
constexpr int kWideConfig = kStageConfigs + 1;

__device__ __forceinline__ int2 cell_range(const SampleArgs& a, int vv, int uu) {
  return bucket_range(__ldg(a.hash + (size_t)vv * a.cam.width + uu), a.n_sorted);
}

// Pack the candidates once per launch: pts[j] = (xyz of sorted_point_idx[j],
// its id), or id -1 when the id is outside [0, n_points).  Every later fetch
// of candidate j is then one 16-byte load instead of
// an id load and a dependent point gather.
__device__ __forceinline__ float4 packed_point(const int* __restrict__ sidx, int j, const float* __restrict__ xyz,
                                               int n_points) {
  const int id = __ldg(sidx + j);
  float4 p = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
  if ((unsigned)id < (unsigned)n_points) {
    const float4 q = load_point(xyz, id);
    p = make_float4(q.x, q.y, q.z, __int_as_float(id));
  }
  return p;
}

constexpr int kPackPerBlock = 4 * kThreads;

// Candidates [block * kPackPerBlock, + kPackPerBlock) packed by one block, four per thread in flight.
__device__ __forceinline__ void pack_block(const SampleArgs& a, long long block) {
  const long long j0 = block * kPackPerBlock + threadIdx.x;
  float4 p[4];
#pragma unroll
  for (int q = 0; q < 4; q++)
    if (j0 + kThreads * q < a.n_sorted) p[q] = packed_point(a.sidx, (int)(j0 + kThreads * q), a.xyz, a.n_points);
#pragma unroll
  for (int q = 0; q < 4; q++)
    if (j0 + kThreads * q < a.n_sorted) const_cast<float4*>(a.pts)[j0 + kThreads * q] = p[q];
}

__host__ __device__ inline BinDiv make_bin_div(float intvl) {
  BinDiv bd;
  bd.intvl = intvl;
  bd.inv = 1.0f / intvl;
  bd.fast = intvl > 0.0f && bd.inv < 0x1p100f && intvl < 0x1p100f;
  return bd;
}

// ceil(2^32 / n): x / n is the high word of x times it for x <= 32 n; 0 where that does not hold.
__host__ __device__ inline unsigned inverse_of(int n) { return n < 2 || n > 8192 ? 0u : 0xffffffffu / (unsigned)n + 1u; }

__host__ __device__ inline void derive_args(SampleArgs& a) {
  a.inv_idx = a.opt.S <= 8192 && a.opt.P <= 8192 ? inverse_of(a.opt.S * a.opt.P) : 0u;
  a.inv_xyz = a.opt.S <= 8192 ? inverse_of(a.opt.S * 3) : 0u;
  a.inv_t = inverse_of(a.opt.S);
  a.rt = make_radius_test(a.opt.radius);
  a.bins = make_bin_div(a.opt.t_intvl);
  a.near0 = a.opt.radius * 1.001f;
  a.quanta = 1.0f / a.opt.radius;
  a.eps = fabsf(a.opt.radius / a.opt.alpha_g);
  // The reference's "farthest" buffer entry starts at 1e3, so eight entries beyond that leave slot 0 the one to
  // replace; the lanes' buffer does not know this: such radii are left to serve_exact.
  if (a.opt.radius > 1e3f) a.eps = INFINITY;
}

__device__ __forceinline__ int bin_index(const BinDiv& bd, float x) {
  if (bd.fast) {
    const float y = __fmul_rn(x, bd.inv);
    const int lo = __float2int_rz(__fmul_rn(y, 1.0f - 0x1p-21f));
    if (lo == __float2int_rz(__fmul_rn(y, 1.0f + 0x1p-21f))) return lo;
  }
  return __float2int_rz(__fdiv_rn(x, bd.intvl));
}

// The same for all lanes of the warp (those not `in` get any value); the exact
// division is taken by a branch of the whole warp.
__device__ __forceinline__ int bin_index(const BinDiv& bd, bool in, float x) {
  const float y = __fmul_rn(x, bd.inv);
  int b = __float2int_rz(__fmul_rn(y, 1.0f - 0x1p-21f));
  const bool edge = in && (!bd.fast || b != __float2int_rz(__fmul_rn(y, 1.0f + 0x1p-21f)));
  if (__any_sync(0xffffffffu, edge)) {
    const int e = __float2int_rz(__fdiv_rn(x, bd.intvl));
    if (edge) b = e;
  }
  return b;
}

// The general walk: a ray by a whole warp, with the reference's own arithmetic.
// The ray's k*k window cells (reference order: rows, then columns, clamped) are
// concatenated into one candidate sequence: lane c < k*k holds cell c's range
// (cbase, ccnt) and its exclusive prefix, and each chunk of 32 consecutive
// candidates is spread over the lanes, every lane finding its cell by a binary
// search over the prefixes (shuffles).  What depends on the order: the
// 48-per-cell cap from ballot ranks plus a per-cell carry, bin sums added one
// candidate at a time in sequence order, and the 8-entry ball buffers fed hits
// in sequence order.  J numbers the candidates (see kIntIds).
template <class J>
__device__ __noinline__ void sample_ray_warp(const SampleArgs& a, int v, int u, unsigned* wbuf) {
  const unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int W = a.cam.width, H = a.cam.height, k = a.opt.k;
  const int lo = ((k + 1) >> 1) - 1;
  // lane c < k*k: cell c's first index and count
  int cbase = 0, ccnt = 0;
  if (lane < k * k) {
    const int q = lane / k;
    const int vv = min(max(v + q - lo, 0), H - 1), uu = min(max(u + (lane - q * k) - lo, 0), W - 1);
    const int2 rg = cell_range(a, vv, uu);
    cbase = rg.x;
    ccnt = rg.y - rg.x;
  }
  const int ray = v * W + u;
  const int S = a.opt.S, P = a.opt.P;
  const float radius = a.opt.radius;
  Ray r;
  make_ray(a.cam.c2w, a.cam.fx, a.cam.fy, a.cam.cx, a.cam.cy, u, v, r);
  const float inv_dd = __frcp_rn(r.dd);
  const RadiusTest& rt = a.rt;

  J cpre = ccnt;  // exclusive prefix over cells
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const J t = __shfl_up_sync(kAll, cpre, o);
    if (lane >= o) cpre += t;
  }
  const J total = __shfl_sync(kAll, cpre, 31);
  cpre -= ccnt;
  auto span = [](J x) { return (int)min(max(x, J(0)), J(32)); };
  const bool capped = __any_sync(kAll, ccnt > kKeptPerCell);

  // body(j0, valid, idx, cell, pc) per lane and chunk: candidate j0 + lane of
  // the sequence, its index in a.pts, its cell and the cell's first j
  auto chunks = [&](auto&& body) {
    for (J j0 = 0; j0 < total; j0 += 32) {
      const J j = j0 + lane;
      int c = 0;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1)
        if (__shfl_sync(kAll, cpre, c + s) <= j) c += s;
      const J pc = __shfl_sync(kAll, cpre, c);
      const int idx = __shfl_sync(kAll, cbase, c) + (int)(j - pc);
      body(j0, j < total, idx, c, pc);
    }
  };
  // The same for the capped passes (A, B and the walk sums; carry = the
  // pass's per-cell kept counts): when the cell the chunk ended in already
  // has its 48 kept candidates, the rest of it is skipped -- none of them can
  // be kept.
  auto capped_chunks = [&](const int& carry, auto&& body) {
    for (J j0 = 0; j0 < total;) {
      const J j = j0 + lane;
      int c = 0;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1)
        if (__shfl_sync(kAll, cpre, c + s) <= j) c += s;
      const J pc = __shfl_sync(kAll, cpre, c);
      const int idx = __shfl_sync(kAll, cbase, c) + (int)(j - pc);
      body(j0, j < total, idx, c, pc);
      j0 += 32;
      if (capped) {
        const int last = __shfl_sync(kAll, c, 31);
        if (__shfl_sync(kAll, carry, last) >= kKeptPerCell) j0 = max(j0, __shfl_sync(kAll, J(cpre + ccnt), last));
      }
    }
  };
  // the candidate's t and offset from the ray; true when within the radius
  auto eval = [&](bool valid, int idx, float& t, float& e0, float& e1, float& e2) -> bool {
    if (!valid) return false;
    const float4 p = __ldg(a.pts + idx);
    if (__float_as_int(p.w) < 0) return false;
    t = ray_t(r, inv_dd, p);
    e0 = __fsub_rn(p.x, __fmaf_rn(t, r.d[0], r.o[0]));
    e1 = __fsub_rn(p.y, __fmaf_rn(t, r.d[1], r.o[1]));
    e2 = __fsub_rn(p.z, __fmaf_rn(t, r.d[2], r.o[2]));
    const float q = squared(e0, e1, e2);
    return q < rt.lo2 || (!(q > rt.hi2) && norm3df(e0, e1, e2) < rt.r);
  };
  // kept candidates that are among the first 48 kept of their cell; `carry`
  // (lane c's copy is cell c's) counts a cell's kept candidates of earlier chunks
  auto accept = [&](bool kept, J j0, int cell, J pc, int& carry) -> bool {
    if (!capped) return kept;
    const unsigned m = __ballot_sync(kAll, kept);
    const int before = __shfl_sync(kAll, carry, cell) + __popc(m & below & ~lane_span(0, span(pc - j0)));
    carry += __popc(m & lane_span(span(cpre - j0), span(cpre + ccnt - j0)));
    return kept && before < kKeptPerCell;
  };
  const BinDiv& bdiv = a.bins;
  auto bin_of = [&](float t, float tmin) {
    return bin_index(bdiv, __fsub_rn(t, tmin));
  };

  // pass A: tmin / tmax
  float tmin = 1e3f, tmax = -1e3f;
  {
    int carry = 0;
    capped_chunks(carry, [&](J j0, bool valid, int idx, int cell, J pc) {
      float t = 0.f, e0, e1, e2;
      if (accept(eval(valid, idx, t, e0, e1, e2), j0, cell, pc, carry)) {
        if (tmin > t) tmin = t;
        if (tmax < t) tmax = t;
      }
    });
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float a0 = __shfl_xor_sync(kAll, tmin, o), a1 = __shfl_xor_sync(kAll, tmax, o);
    if (tmin > a0) tmin = a0;
    if (tmax < a1) tmax = a1;
  }

  float* o_xyz = a.sp_xyz + (size_t)ray * S * 3;
  float* o_t = a.sp_t + (size_t)ray * S;
  uint8_t* o_m = a.mask + (size_t)ray * S;
  int* o_idx = a.pc_idx + (size_t)ray * S * P;
  int emitted = 0;
  float te[kTeReg];
#pragma unroll
  for (int q = 0; q < kTeReg; q++) te[q] = 0.0f;

  if (!(tmin > tmax)) {
    // pass B: which bins hold >= 2 kept points (the only ones the walk uses)
    unsigned s1[kBins / 32], s2[kBins / 32];
#pragma unroll
    for (int q = 0; q < kBins / 32; q++) s1[q] = 0u, s2[q] = 0u;
    {
      int carry = 0;
      capped_chunks(carry, [&](J j0, bool valid, int idx, int cell, J pc) {
        float t = 0.f, e0, e1, e2;
        if (accept(eval(valid, idx, t, e0, e1, e2), j0, cell, pc, carry)) {
          const int b = bin_of(t, tmin);
          if (b < kBins) {
            const unsigned bit = 1u << (b & 31);
#pragma unroll
            for (int q = 0; q < kBins / 32; q++)
              if (q == (b >> 5)) {
                s2[q] |= s1[q] & bit;
                s1[q] |= bit;
              }
          }
        }
      });
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int q = 0; q < kBins / 32; q++) {
        const unsigned o1 = __shfl_xor_sync(kAll, s1[q], o), o2 = __shfl_xor_sync(kAll, s2[q], o);
        s2[q] = s2[q] | o2 | (s1[q] & o1);
        s1[q] |= o1;
      }
    }
    // first bin >= from holding >= 2 points (kBins if none)
    auto next_bin = [&](int from) {
      int b = kBins;
#pragma unroll
      for (int q = kBins / 32 - 1; q >= 0; q--) {
        unsigned m = s2[q];
        if (q * 32 + 32 <= from)
          m = 0u;
        else if (q * 32 < from)
          m &= ~0u << (from - q * 32);
        if (m) b = q * 32 + __ffs(m) - 1;
      }
      return b;
    };
    // walk: the bins' sums are gathered kWalkBatch bins per pass, in ascending order
    float transmit = 1.0f;
    int from = 0;
    bool done = false;
    while (!done) {
      int bb[kWalkBatch];
      int nb = 0;
#pragma unroll
      for (int q = 0; q < kWalkBatch; q++) {
        bb[q] = next_bin(q == 0 ? from : bb[q - 1] + 1);
        nb += bb[q] < kBins ? 1 : 0;
      }
      if (nb == 0) break;
      float bsum[kWalkBatch];
      int bcnt[kWalkBatch];
#pragma unroll
      for (int q = 0; q < kWalkBatch; q++) bsum[q] = 0.0f, bcnt[q] = 0;
      int carry = 0;
      capped_chunks(carry, [&](J j0, bool valid, int idx, int cell, J pc) {
        float t = 0.f, e0 = 0.f, e1 = 0.f, e2 = 0.f;
        int mine = -1;
        float dist = 0.0f;
        if (accept(eval(valid, idx, t, e0, e1, e2), j0, cell, pc, carry)) {
          const int b = bin_of(t, tmin);
#pragma unroll
          for (int q = 0; q < kWalkBatch; q++)
            if (bb[q] == b) mine = q;
          if (mine >= 0) dist = norm3df(e0, e1, e2);
        }
#pragma unroll
        for (int q = 0; q < kWalkBatch; q++) {
          unsigned mm = __ballot_sync(kAll, mine == q);
          while (mm) {
            const int l = __ffs(mm) - 1;
            mm &= mm - 1;
            bsum[q] = __fadd_rn(bsum[q], __shfl_sync(kAll, dist, l));
            bcnt[q]++;
          }
        }
      });
#pragma unroll
      for (int q = 0; q < kWalkBatch; q++) {
        if (q >= nb) break;
        if (transmit < 1e-3f || emitted >= S) {
          done = true;
          break;
        }
        const float sdf = __fdiv_rn(bsum[q], __fadd_rn((float)bcnt[q], 1e-6f));
        const float alpha = __fmul_rn(a.opt.gamma, __expf(__fdiv_rn(-sdf, a.opt.alpha_g)));
        const float weight = __fmul_rn(alpha, transmit);
        if (weight > 1e-3f) {
          const float t = __fmaf_rn((float)bb[q], a.opt.t_intvl, tmin);
          if (lane == 0) {
            o_xyz[emitted * 3 + 0] = __fmaf_rn(t, r.d[0], r.o[0]);
            o_xyz[emitted * 3 + 1] = __fmaf_rn(t, r.d[1], r.o[1]);
            o_xyz[emitted * 3 + 2] = __fmaf_rn(t, r.d[2], r.o[2]);
            o_t[emitted] = t;
            o_m[emitted] = 1;
          }
#pragma unroll
          for (int e = 0; e < kTeReg; e++)
            if (e == emitted) te[e] = t;
          emitted++;
        }
        transmit = __fsub_rn(transmit, alpha);
      }
      if (nb < kWalkBatch) break;
      from = bb[kWalkBatch - 1] + 1;
    }
  }
  __syncwarp();

  // per-sample point selection, two samples per pass, buffers fed hits in
  // order.  The buffers (distance and id of kBallBuf hits per sample) live in
  // the serving warp's 32 words of shared memory (wbuf), written by lane 0;
  // their size, minimum-then-maximum tracking and state are warp-uniform
  // registers.
  static_assert(2 * kBallPass * kBallBuf <= 32, "ball buffers exceed the warp's words");
  float* sbd = reinterpret_cast<float*>(wbuf);              // [kBallPass][kBallBuf] distances
  int* sbi = reinterpret_cast<int*>(wbuf) + kBallPass * kBallBuf;  // [kBallPass][kBallBuf] ids
  const float omax = fmaxf(fabsf(r.o[0]), fmaxf(fabsf(r.o[1]), fabsf(r.o[2])));
  for (int s0 = 0; s0 < emitted; s0 += kBallPass) {
    const int ns = min(kBallPass, emitted - s0);
    float ts[kBallPass], reach[kBallPass], spx[kBallPass], spy[kBallPass], spz[kBallPass], maxd[kBallPass];
    int bsize[kBallPass], maxi[kBallPass];
    bool settled[kBallPass];
#pragma unroll
    for (int q = 0; q < kBallPass; q++) {
      float t = 0.0f;
      if (q < ns) {
        t = o_t[s0 + q];
#pragma unroll
        for (int e = 0; e < kTeReg; e++)
          if (e == s0 + q) t = te[e];
      }
      ts[q] = t;
      reach[q] = q < ns ? radius * 1.001f + 1e-5f * (1.0f + fabsf(t) + omax) : -1.0f;
      spx[q] = __fmaf_rn(t, r.d[0], r.o[0]);
      spy[q] = __fmaf_rn(t, r.d[1], r.o[1]);
      spz[q] = __fmaf_rn(t, r.d[2], r.o[2]);
      bsize[q] = 0;
      maxi[q] = 0;
      maxd[q] = 1e3f;
      settled[q] = false;
    }
    chunks([&](J, bool valid, int idx, int, J) {
      float dq[kBallPass];
      bool hq[kBallPass];
      int id = -1;
#pragma unroll
      for (int q = 0; q < kBallPass; q++) dq[q] = 0.0f, hq[q] = false;
      if (valid) {
        const float4 p = __ldg(a.pts + idx);
        id = __float_as_int(p.w);
        if (id >= 0) {
          const float along = dot3(p.x - r.o[0], p.y - r.o[1], p.z - r.o[2], r.d[0], r.d[1], r.d[2]);
#pragma unroll
          for (int q = 0; q < kBallPass; q++)
            if (fabsf(along - ts[q]) <= reach[q]) {
              dq[q] = norm3df(__fsub_rn(spx[q], p.x), __fsub_rn(spy[q], p.y), __fsub_rn(spz[q], p.z));
              hq[q] = dq[q] < radius;
            }
        }
      }
#pragma unroll
      for (int q = 0; q < kBallPass; q++) {
        // Which of the chunk's hits can change the buffer (bsize, settled and
        // maxd are the same in every lane).  While filling: all of them.  Once
        // full and replaced at least once, maxd is the buffer's true maximum and
        // only decreases, so only hits below it.  Full but never replaced, maxd
        // is the minimum of the first eight (the reference's quirk) and the
        // buffer stays as it is until a hit falls below it; from that hit on,
        // maxd becomes the true maximum, so every later hit is looked at.
        unsigned mm;
        if (bsize[q] < kBallBuf || settled[q]) {
          mm = __ballot_sync(kAll, hq[q] && (bsize[q] < kBallBuf || dq[q] < maxd[q]));
        } else {
          const unsigned first = __ballot_sync(kAll, hq[q] && dq[q] < maxd[q]);
          const unsigned all = __ballot_sync(kAll, hq[q]);
          mm = first ? all & ~((1u << (__ffs(first) - 1)) - 1u) : 0u;
        }
        while (mm) {
          const int l = __ffs(mm) - 1;
          mm &= mm - 1;
          const float dist = __shfl_sync(kAll, dq[q], l);
          const int cid = __shfl_sync(kAll, id, l);
          if (bsize[q] < kBallBuf) {
            if (lane == 0) {
              sbd[q * kBallBuf + bsize[q]] = dist;
              sbi[q * kBallBuf + bsize[q]] = cid;
            }
            if (maxd[q] > dist) {
              maxd[q] = dist;
              maxi[q] = bsize[q];
            }
            bsize[q]++;
          } else if (dist < maxd[q]) {
            if (lane == 0) {
              sbd[q * kBallBuf + maxi[q]] = dist;
              sbi[q * kBallBuf + maxi[q]] = cid;
            }
            __syncwarp();
            // the new maximum; a scan from the replaced slot's value keeps the
            // replaced slot when it holds the maximum, else the first slot that does
            const float ve = lane < kBallBuf ? sbd[q * kBallBuf + lane] : -1.0f;
            float md = ve;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) md = fmaxf(md, __shfl_xor_sync(kAll, md, o));
            const unsigned at = __ballot_sync(kAll, lane < kBallBuf && ve == md);
            maxi[q] = md == dist ? maxi[q] : __ffs(at) - 1;
            maxd[q] = md;
            settled[q] = true;
          }
        }
      }
    });
#pragma unroll
    for (int q = 0; q < kBallPass; q++) {
      if (q >= ns) break;
      int* row = o_idx + (size_t)(s0 + q) * P;
      __syncwarp();
      const int val = lane < bsize[q] ? sbi[q * kBallBuf + lane] : -1;
      if (lane < min(P, kBallBuf)) row[lane] = val;
      if (P > kBallBuf)
        for (int e = kBallBuf + lane; e < P; e += 32) row[e] = -1;
    }
  }
  if (emitted < S) {
    const int n3 = (S - emitted) * 3, n1 = S - emitted, np = (S - emitted) * P;
    for (int e = lane; e < n3; e += 32) o_xyz[emitted * 3 + e] = 0.0f;
    for (int e = lane; e < n1; e += 32) o_t[emitted + e] = 0.0f, o_m[emitted + e] = 0;
    for (int e = lane; e < np; e += 32) o_idx[(size_t)emitted * P + e] = -1;
  }
  __syncwarp();
}

// A listed candidate's squared distance to the ray may exceed the radius by
// this much: what the ball query can take lies within the radius of a sample
// on the ray, so within the radius of the ray but for the rounding of t, of the
// sample point and of the differences -- a few 1e-7 of |t| and |o|, against a
// margin of 1e-5 of them plus a thousandth of the radius.
__device__ __forceinline__ float near_limit(float c0, float t) {
  const float lim = __fmaf_rn(1e-5f, fabsf(t), c0);
  return __fmul_rn(lim, lim);
}

// The slots [from, S) of a ray's outputs: nothing emitted.  `lane` of `n` lanes.
__device__ __forceinline__ void default_slots(const SampleArgs& a, size_t ray, int from, int lane, int n) {
  const int S = a.opt.S, P = a.opt.P;
  const int left = S - from;
  if (left <= 0) return;
  float* o_xyz = a.sp_xyz + (ray * S + from) * 3;
  float* o_t = a.sp_t + ray * S + from;
  uint8_t* o_m = a.mask + ray * S + from;
  int* o_idx = a.pc_idx + (ray * S + from) * P;
  for (int e = lane; e < left * 3; e += n) o_xyz[e] = 0.0f;
  for (int e = lane; e < left; e += n) o_t[e] = 0.0f, o_m[e] = 0;
  if ((P & 3) == 0 && ((uintptr_t)a.pc_idx & 15) == 0) {
    for (int e = lane; e < left * P / 4; e += n) reinterpret_cast<int4*>(o_idx)[e] = make_int4(-1, -1, -1, -1);
  } else {
    for (int e = lane; e < left * P; e += n) o_idx[e] = -1;
  }
}

// sqrt with an error of a few ulp
__device__ __forceinline__ float sqrt_fast(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// What serve_rays leaves to serve_exact, by its lanes' groups.
struct Unsettled {
  int n;        // listed candidates; -1: none are listed yet
  int emitted;  // samples emitted; -1: the walk is to be done again
  bool balls;   // their points are to be selected again
};

// Serve 32 / L rays, L lanes each: `entry` is the group's list entry (ray < 0:
// none); pool: the warp's kHistWords words and `entries` listed candidates.
// Returns the lanes of groups left unserved, for sample_ray_warp (their list
// overflows), and in `left` what else is left, for serve_exact.
//
// The walk uses mean distances from the histogram's quantised sums, and the ball
// buffers order their hits by squared distance.  Both know their error; where a
// comparison is closer than that (about one ray in a thousand of a cloud
// without equal distances), the ray's walk or point selection is left to
// serve_exact, and so are rays whose window's rows are no runs (at the image's
// edge, where they repeat cells); it has the reference's own arithmetic (sums of
// norm3df in window order, buffers ordered by norm3df), so every decision is the
// reference's.
__device__ __forceinline__ unsigned serve_rays(const SampleArgs& a, const int L, int4 entry, unsigned char* pool,
                                               int entries, Unsettled& left) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr unsigned kCloseKeys = 512;  // of a float's bits: at least 2^-15 of its value
  constexpr int kSumBits = 21, kQuant = 10;  // histogram word: sum of distances in radius / 2^kQuant, count above;
                                             // 2^kQuant entries fit
  const int lane = threadIdx.x & 31;
  const int gb = lane & ~(L - 1), sl = lane & (L - 1);  // the group's first lane, this lane's place
  const unsigned gmask = (kAll >> (32 - L)) << gb;
  const unsigned below = gmask & ((1u << lane) - 1u);
  const int most_hits = kHistWords / 64 * L;  // ball hits held, in the group's share of the histogram words
  unsigned* hist = reinterpret_cast<unsigned*>(pool) + gb * (kHistWords / 32);
  uint2* hits = reinterpret_cast<uint2*>(hist);
  const int cap = entries * L / 32;
  int* list = reinterpret_cast<int*>(pool + kHistWords * 4) + gb * (entries / 32);
  const int W = a.cam.width, H = a.cam.height, k = a.opt.k;
  const int lo = ((k + 1) >> 1) - 1;
  const int S = a.opt.S, P = a.opt.P;
  const int ray = entry.x;
  bool live = ray >= 0;
  const int v = live ? ray / W : 0, u = live ? ray - v * W : 0;
  Ray r;
#pragma unroll
  for (int i = 0; i < 3; i++) r.o[i] = __ldg(a.cam.c2w + 4 * i + 3);
  r.d[0] = __int_as_float(entry.y), r.d[1] = __int_as_float(entry.z), r.d[2] = __int_as_float(entry.w);
  r.dd = dot3(r.d[0], r.d[1], r.d[2], r.d[0], r.d[1], r.d[2]);
  const float inv_dd = __frcp_rn(r.dd);
  const RadiusTest& rt = a.rt;

  // The window's rows: row q is the run [base, base + count) of the packed
  // candidates, when its cells' buckets follow one another (they do in every
  // table the build makes; clamped columns repeat cells and need not).
  // Candidate j of the window is packed candidate j + base + the steps of the
  // rows it is beyond.
  int p1, p2, p3, p4, T;  // first candidate of rows 1..4, all candidates
  int base, step1, step2, step3, step4;
  bool good = true, deep = false;  // deep: a cell holds more than 48
  {
    int cnt = 0, first = 0;
    if (live && sl < k) {
      const int2* row = a.hash + (size_t)min(max(v - lo + sl, 0), H - 1) * W;
#pragma unroll
      for (int c = 0; c < kMaxKernel; c++) {
        if (c < k) {
          const int2 rg = bucket_range(__ldg(row + min(max(u - lo + c, 0), W - 1)), a.n_sorted);
          const int m = rg.y - rg.x;
          if (m > 0) {
            if (cnt == 0) first = rg.x;
            good = good && rg.x == first + cnt;
            deep = deep || m > kKeptPerCell;
            cnt += m;
          }
        }
      }
    }
    const int c0 = __shfl_sync(kAll, cnt, gb), c1 = __shfl_sync(kAll, cnt, gb + 1), c2 = __shfl_sync(kAll, cnt, gb + 2),
              c3 = __shfl_sync(kAll, cnt, gb + 3), c4 = __shfl_sync(kAll, cnt, gb + 4);
    p1 = c0, p2 = (int)((unsigned)p1 + c1), p3 = (int)((unsigned)p2 + c2), p4 = (int)((unsigned)p3 + c3);
    T = (int)((unsigned)p4 + c4);
    // clamped rows repeat: their sum may pass 2^31 (less what the passes number beyond it)
    good = good && (p2 | p3 | p4 | T | (int)((unsigned)T + 64u)) >= 0;
    base = __shfl_sync(kAll, first, gb);
    const int f1 = __shfl_sync(kAll, first, gb + 1), f2 = __shfl_sync(kAll, first, gb + 2),
              f3 = __shfl_sync(kAll, first, gb + 3), f4 = __shfl_sync(kAll, first, gb + 4);
    step1 = f1 - (base + c0), step2 = f2 - (f1 + c1), step3 = f3 - (f2 + c2), step4 = f4 - (f3 + c3);
    good = (__ballot_sync(kAll, !good) & gmask) == 0u;
  }
  // lane c: window cell c's first candidate and count, for rays with a deep cell (served by a whole warp)
  int cpre = 0, ccnt = 0, carry = 0;
  const bool capped = __any_sync(kAll, deep);
  if (capped) {
    if (live && lane < k * k) {
      const int q = lane / k;
      const int2 rg = cell_range(a, min(max(v + q - lo, 0), H - 1), min(max(u + (lane - q * k) - lo, 0), W - 1));
      ccnt = rg.y - rg.x;
    }
    cpre = ccnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(kAll, cpre, o);
      if (lane >= o) cpre += t;
    }
    cpre -= ccnt;
    good = good && L == 32;
  }
  int n = live && !good ? -1 : 0;  // no runs: nothing is listed here
  left = {n, 0, false};
  live = live && good;
  if (!__any_sync(kAll, live)) return 0u;
  if (!live) T = 0;

  // pass A: tmin over the kept candidates (epcq_render_topk.cu:132-161) and the list
  const float omax = fmaxf(fabsf(r.o[0]), fmaxf(fabsf(r.o[1]), fabsf(r.o[2])));
  const float c0 = __fmaf_rn(1e-5f, 1.0f + omax, a.near0);
  float tmin = 1e3f;
  {
    const int Tmax = __reduce_max_sync(kAll, T);
    auto index = [&](int j) {
      int i = j + base;
      if (j >= p1) i += step1;
      if (j >= p2) i += step2;
      if (j >= p3) i += step3;
      if (j >= p4) i += step4;
      return i;
    };
    int idx = index(sl);
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
    if (sl < T) p = __ldg(a.pts + idx);
    for (int j0 = 0; j0 < Tmax; j0 += L) {
      const int jn = j0 + L + sl;
      const int idx_n = index(jn);
      float4 pn = p;
      if (jn < T) pn = __ldg(a.pts + idx_n);
      const bool in = jn - L < T && __float_as_int(p.w) >= 0;
      const float t = ray_t(r, inv_dd, p);
      const float e0 = __fsub_rn(p.x, __fmaf_rn(t, r.d[0], r.o[0]));
      const float e1 = __fsub_rn(p.y, __fmaf_rn(t, r.d[1], r.o[1]));
      const float e2 = __fsub_rn(p.z, __fmaf_rn(t, r.d[2], r.o[2]));
      const float q = squared(e0, e1, e2);
      bool kept = within_radius(rt, in, q, e0, e1, e2);
      const bool near = kept || (in && q <= near_limit(c0, t));
      if (capped) {  // kept only among its cell's first 48 (carry: lane c's copy counts cell c's kept so far)
        const int j = j0 + lane;
        int c = 0;
#pragma unroll
        for (int s = 16; s > 0; s >>= 1)
          if (__shfl_sync(kAll, cpre, c + s) <= j) c += s;
        const int pc = __shfl_sync(kAll, cpre, c);
        const unsigned m = __ballot_sync(kAll, kept);
        const int before = __shfl_sync(kAll, carry, c) + __popc(m & below & ~lane_span(0, max(pc - j0, 0)));
        carry += __popc(m & lane_span(min(max(cpre - j0, 0), 32), min(max(cpre + ccnt - j0, 0), 32)));
        kept = kept && before < kKeptPerCell;
      }
      if (kept) tmin = fminf(tmin, t);
      const unsigned nm = __ballot_sync(kAll, near);
      const int pos = n + __popc(nm & below);
      if (near && pos < cap) list[pos] = kept ? idx : idx | (int)0x80000000u;
      n += __popc(nm & gmask);
      if (L == 32 && n > cap) break;  // the general walk's (8 lanes hold every window they get)
      idx = idx_n;
      p = pn;
    }
  }
  const unsigned over = __ballot_sync(kAll, n > cap);  // more listed candidates than the group holds
  if (n > cap) live = false, n = 0;
  for (int o = L >> 1; o > 0; o >>= 1) tmin = fminf(tmin, __shfl_xor_sync(kAll, tmin, o));
  __syncwarp();

  const BinDiv& bdiv = a.bins;
  const size_t slot0 = (size_t)(live ? ray : 0) * S;
  // the kept entries' bins: counts and quantised distance sums, in rows of L words; `rows`: the group's rows
  // that hold one
  const int nmax = __reduce_max_sync(kAll, n);
  unsigned rows = 0u;
  if (nmax > 0) {
    for (int c = 4 * sl; c < kBins; c += 4 * L) *reinterpret_cast<uint4*>(hist + c) = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    const float quant = (float)(1 << kQuant) * a.quanta;
    for (int i0 = 0; i0 < nmax; i0 += L) {
      const int i = i0 + sl;
      const int idx = list[min(i, cap - 1)];
      const bool in = i < n && idx >= 0;
      float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
      if (in) p = __ldg(a.pts + idx);
      const float t = ray_t(r, inv_dd, p);
      const int b = bin_index(bdiv, in, __fsub_rn(t, tmin));
      const float q = squared(__fsub_rn(p.x, __fmaf_rn(t, r.d[0], r.o[0])), __fsub_rn(p.y, __fmaf_rn(t, r.d[1], r.o[1])),
                              __fsub_rn(p.z, __fmaf_rn(t, r.d[2], r.o[2])));
      const unsigned dq = min((unsigned)(sqrt_fast(q) * quant), 1u << kQuant);
      if (in && b < kBins) {
        atomicAdd(hist + b, dq | (1u << kSumBits));
        rows |= 1u << (b / L);
      }
    }
    __syncwarp();
    for (int o = L >> 1; o > 0; o >>= 1) rows |= __shfl_xor_sync(kAll, rows, o);
  }

  int emitted = 0;
  // how far the walk's alpha can be off by the quantised sums (relative); the mean lies within half a quantum
  const float eps = __fmaf_rn(a.eps, 1.0f / (1 << kQuant) + 1e-5f, 1e-5f);
  bool close = rows != 0u && (!(eps < 0.05f) || !rt.fast);  // a comparison was closer than its error
  {
    // primary-surface walk (epcq_render_topk.cu:181-204): L bins at a time, their alphas side by side
    float transmit = 1.0f, off = 0.0f, t0 = 0.0f, t1 = 0.0f;
    while (__any_sync(kAll, rows != 0u)) {
      const int row = rows ? __ffs(rows) - 1 : 0;
      const int bin = row * L + sl;
      const unsigned x = rows != 0u ? hist[bin] : 0u;
      rows &= rows - 1;
      const int cnt = x >> kSumBits;
      unsigned todo = __ballot_sync(kAll, cnt > 1) & gmask;
      if (!__any_sync(kAll, todo != 0u)) continue;
      const float sum = ((float)(x & ((1u << kSumBits) - 1u)) + 0.5f * (float)cnt) * (a.opt.radius * (1.0f / (1 << kQuant)));
      const float sdf = __fdividef(sum, (float)cnt + 1e-6f);
      const float alpha = a.opt.gamma * __expf(__fdividef(-sdf, a.opt.alpha_g));
      const float t = __fmaf_rn((float)bin, a.opt.t_intvl, tmin);
      int slot = -1;  // this lane's bin emits into this slot
      while (__any_sync(kAll, todo != 0u)) {
        const int src = todo ? __ffs(todo) - 1 : lane;
        const float al = __shfl_sync(kAll, alpha, src), tl = __shfl_sync(kAll, t, src);
        if (todo) {
          todo &= todo - 1;
          if (fabsf(transmit - 1e-3f) <= off) close = true;
          if (transmit < 1e-3f || emitted >= S) {
            todo = 0u, rows = 0u;
          } else {
            const float weight = __fmul_rn(al, transmit);
            if (fabsf(weight - 1e-3f) <= fabsf(al) * off + fabsf(weight) * eps) close = true;
            if (weight > 1e-3f) {
              if (lane == src) slot = emitted;
              if (emitted == 0) t0 = tl;
              if (emitted == 1) t1 = tl;
              emitted++;
            }
            transmit = __fsub_rn(transmit, al);
            off += fabsf(al) * eps + 1e-6f * (fabsf(transmit) + fabsf(al));
          }
        }
      }
      if (slot >= 0) {
        const size_t at = slot0 + slot;
#pragma unroll
        for (int i = 0; i < 3; i++) a.sp_xyz[at * 3 + i] = __fmaf_rn(t, r.d[i], r.o[i]);
        a.sp_t[at] = t;
        a.mask[at] = 1;
      }
    }
    if ((__ballot_sync(kAll, close) & gmask) != 0u) emitted = -1;
    close = false;

    // per-sample point selection (epcq_render_topk.cu:10-81), a sample at a time
    const int most = __reduce_max_sync(kAll, emitted);
    const int nball = __reduce_max_sync(kAll, emitted > 0 ? n : 0);
#pragma unroll 1
    for (int s = 0; s < most; s++) {
      const bool on = s < emitted;
      __syncwarp();
      if (s > 1 && on) t0 = *(volatile const float*)(a.sp_t + slot0 + s);
      const float sx = __fmaf_rn(t0, r.d[0], r.o[0]), sy = __fmaf_rn(t0, r.d[1], r.o[1]),
                  sz = __fmaf_rn(t0, r.d[2], r.o[2]);
      t0 = t1;
      const int m = on ? n : 0;
      // The buffer: lanes 0..7 of the group hold the slots' keys -- the squared distance's bits with the slot's
      // number in the low three, ascending, so lane 7 is the slot the reference's scan would replace -- and lane
      // s the list entry in slot s.  Keys less than kCloseKeys apart are too close for the order of norm3df.
      unsigned key = 0u, limit = 0u;  // a later hit with a key below `limit` replaces an entry
      int held_entry = 0;
      bool settled = false;   // one was replaced: limit is the true maximum (before: the minimum)
      int cnt = 0, held = 0;  // hits looked at; hits in shared memory, not yet looked at
#pragma unroll 1
      for (int i0 = 0;; i0 += L) {
        const int i = i0 + sl;
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < m) p = __ldg(a.pts + (list[i] & 0x7fffffff));
        const float e0 = __fsub_rn(sx, p.x), e1 = __fsub_rn(sy, p.y), e2 = __fsub_rn(sz, p.z);
        const float d = squared(e0, e1, e2);
        const bool hit = within_radius(rt, i < m, d, e0, e1, e2);
        const unsigned hm = __ballot_sync(kAll, hit);
        if (hit) hits[held + __popc(hm & below)] = make_uint2(__float_as_uint(d) & ~7u, (unsigned)i);
        held += __popc(hm & gmask);
        const bool last = i0 + L >= nball;
        if (!last && !__any_sync(kAll, held + L > most_hits)) continue;
        // look at the held hits, in order
        __syncwarp();
        const int todo = last || held + L > most_hits ? held : 0;
        if (todo > 0) held = 0;
        const bool first = cnt == 0 && todo > 0;
        cnt += todo;
        for (int h = 0; __any_sync(kAll, h < todo); h += L) {
          bool later = h + sl < todo;  // may replace an entry
          const uint2 x = hits[min(h + sl, most_hits - 1)];
          if (h == 0 && __any_sync(kAll, first)) {  // the first eight fill the slots
            if (first && sl < kBallBuf) {
              key = (later ? x.x : 0x7f800000u) | (unsigned)sl;
              held_entry = (int)x.y;
              later = false;
            }
            if (__any_sync(kAll, first && todo > kBallBuf)) {
              unsigned sk = key;
#pragma unroll
              for (int w = 2; w <= 8; w <<= 1) {
#pragma unroll
                for (int o = w >> 1; o > 0; o >>= 1) {
                  const unsigned ok = __shfl_xor_sync(kAll, sk, o);
                  const bool up = (lane & w) == 0 || w == 8;  // this run ascends
                  sk = ((lane & o) != 0) != up ? min(sk, ok) : max(sk, ok);
                }
              }
              const unsigned prev = __shfl_up_sync(kAll, sk, 1), least = __shfl_sync(kAll, sk, gb);
              if (first && todo > kBallBuf) {
                if (sl < kBallBuf) key = sk;
                if (sl > 0 && sl < kBallBuf && sk - prev < kCloseKeys + kBallBuf) close = true;
                limit = least;
              }
            }
          }
          unsigned pm;
          while (pm = __ballot_sync(kAll, later && limit > 0u && x.x < limit + kCloseKeys), pm != 0u) {
            pm &= gmask;
            const bool has = pm != 0u;
            const int l = has ? __ffs(pm) - 1 : lane;
            if (lane <= l) later = false;
            const unsigned nk = __shfl_sync(kAll, x.x, l);
            const int ni = __shfl_sync(kAll, (int)x.y, l);
            // the slot replaced: the maximum's, before the first replacement the minimum's
            const int out = settled ? kBallBuf - 1 : 0;
            const unsigned freed = __shfl_sync(kAll, key, gb + out) & 7u;
            const unsigned mk = nk | freed;
            const unsigned smaller = __ballot_sync(kAll, settled && sl < kBallBuf && key < mk) & gmask;
            const int at = min(__popc(smaller), kBallBuf - 1);
            const unsigned uk = __shfl_up_sync(kAll, key, 1);
            if (has && sl < kBallBuf) {
              if ((key > mk ? key - mk : mk - key) < kCloseKeys + kBallBuf) close = true;  // the slots' numbers too
              if (sl == at)
                key = mk;
              else if (sl > at && sl <= out)
                key = uk;
              if (sl == (int)freed) held_entry = ni;
            }
            const unsigned top = __shfl_sync(kAll, key, gb + kBallBuf - 1);
            if (has) settled = true, limit = top;
          }
        }
        __syncwarp();
        if (last) break;
      }
      if (on) {
        int* row = a.pc_idx + (slot0 + s) * P;
        if (sl < kBallBuf && sl < P)
          row[sl] = sl < cnt ? __float_as_int(__ldg(a.pts + (list[held_entry] & 0x7fffffff)).w) : -1;
        for (int e = kBallBuf + sl; e < P; e += L) row[e] = -1;
      }
    }
  }
  if (live && emitted >= 0) default_slots(a, (size_t)ray, emitted, sl, L);
  left = {n, emitted, (__ballot_sync(kAll, close) & gmask) != 0u};
  return over;
}

// The rays that serve_rays left, as it serves them: their list (made here from
// the cells where there is none), the walk over sums of norm3df added in window
// order, a ray at a time by the whole warp, and the point selection with buffers
// of norm3df in slot order, the warp's rays side by side.  Returns the lanes of
// groups whose list overflows.
//
// A ray by sample_ray_warp walks its window three times and more; where many
// rays come here (repeated or lattice points, whose distances tie) the whole
// view waited for that.  1M points at 800 x 800, sampling alone: each place
// three times 2910 us with it, 640 so (980 with one thread a ray); rounded to a
// lattice 2360 and 580 (880); buckets out of pixel order 1980 and 834 (865; 950
// with a cell at a time).
__device__ __forceinline__ unsigned serve_exact(const SampleArgs& a, int L, int4 entry, unsigned char* pool, int entries,
                                             Unsettled left) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int gb = lane & ~(L - 1), sl = lane & (L - 1);
  const unsigned group = kAll >> (32 - L), gmask = group << gb;
  const unsigned before = (1u << lane) - 1u, below = gmask & before;
  const int cap = entries * L / 32;
  int* lists = reinterpret_cast<int*>(pool + kHistWords * 4);
  int* list = lists + gb * (entries / 32);
  const int S = a.opt.S, P = a.opt.P;
  const RadiusTest& rt = a.rt;
  const int ray = entry.x;
  Ray r;
#pragma unroll
  for (int i = 0; i < 3; i++) r.o[i] = __ldg(a.cam.c2w + 4 * i + 3);
  r.d[0] = __int_as_float(entry.y), r.d[1] = __int_as_float(entry.z), r.d[2] = __int_as_float(entry.w);
  r.dd = dot3(r.d[0], r.d[1], r.d[2], r.d[0], r.d[1], r.d[2]);
  int n = left.n, emitted = left.emitted;
  bool balls = left.balls;

  // the list of a window whose rows are no runs: L cells at a time, their candidates numbered through
  if (__any_sync(kAll, n < 0)) {
    const bool make = n < 0;
    n = make ? 0 : n;
    const int W = a.cam.width, H = a.cam.height, k = a.opt.k, lo = ((k + 1) >> 1) - 1;
    const float inv_dd = __frcp_rn(r.dd);
    const float omax = fmaxf(fabsf(r.o[0]), fmaxf(fabsf(r.o[1]), fabsf(r.o[2])));
    const float c0 = __fmaf_rn(1e-5f, 1.0f + omax, a.near0);
    const int v = make ? ray / W : 0, u = make ? ray - v * W : 0;
    for (int cell0 = 0; cell0 < k * k; cell0 += L) {
      const int l = cell0 + sl;
      int2 rg = make_int2(0, 0);
      if (make && l < k * k) rg = cell_range(a, min(max(v + l / k - lo, 0), H - 1), min(max(u + l % k - lo, 0), W - 1));
      const unsigned cnt = (unsigned)(rg.y - rg.x);
      unsigned pre = cnt;
      for (int o = 1; o < L; o <<= 1) {
        const unsigned t = __shfl_up_sync(kAll, pre, o);
        if (sl >= o) pre = min(pre + t, 0x7fffffffu);  // both below 2^31
      }
      unsigned total = __shfl_sync(kAll, pre, gb + L - 1);
      if (total == 0x7fffffffu) n = cap + 1;  // too many to number: the general walk's
      pre -= cnt;
      int carry = 0;  // this lane's cell: kept so far
      for (unsigned j0 = 0; __any_sync(kAll, j0 < total && n <= cap); j0 += (unsigned)L) {
        const unsigned j = j0 + sl;
        int c = gb;
        for (int s = L >> 1; s > 0; s >>= 1)
          if (__shfl_sync(kAll, pre, c + s) <= j) c += s;
        const unsigned first = __shfl_sync(kAll, pre, c);
        const int idx = __shfl_sync(kAll, rg.x, c) + (int)(j - first);
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
        bool in = j < total && n <= cap;
        if (in) p = __ldg(a.pts + idx);
        in = in && __float_as_int(p.w) >= 0;
        const float t = ray_t(r, inv_dd, p);
        const float e0 = __fsub_rn(p.x, __fmaf_rn(t, r.d[0], r.o[0]));
        const float e1 = __fsub_rn(p.y, __fmaf_rn(t, r.d[1], r.o[1]));
        const float e2 = __fsub_rn(p.z, __fmaf_rn(t, r.d[2], r.o[2]));
        const float q = squared(e0, e1, e2);
        bool kept = within_radius(rt, in, q, e0, e1, e2);
        const bool near = kept || (in && q <= near_limit(c0, t));
        const unsigned km = __ballot_sync(kAll, kept), nm = __ballot_sync(kAll, near);
        auto lane_of = [&](unsigned x) { return gb + min(max((int)(x - j0), 0), L); };  // of candidate x
        const int had = __shfl_sync(kAll, carry, c) + __popc(km & below & ~lane_span(0, lane_of(first)));
        kept = kept && had < kKeptPerCell;
        carry = min(carry + __popc(km & lane_span(lane_of(pre), lane_of(pre + cnt))), kKeptPerCell);
        const int pos = n + __popc(nm & below);
        if (near && pos < cap) list[pos] = kept ? idx : idx | (int)0x80000000u;
        n = min(n + __popc(nm & gmask), cap + 1);
      }
    }
    if (make) emitted = n > cap ? 0 : -1;
    __syncwarp();
  }
  const unsigned over = __ballot_sync(kAll, n > cap);

  // the walk (epcq_render_topk.cu:181-204)
  float* sums = reinterpret_cast<float*>(pool);
  int* counts = reinterpret_cast<int*>(pool) + kBins;
  static_assert(2 * kBins <= kHistWords, "sums and counts");
  const unsigned walks = __ballot_sync(kAll, emitted < 0);
  for (unsigned todo = walks; todo;) {
    const int g = __ffs(todo) - 1;
    todo &= ~(group << g);
    const int* from = lists + g * (entries / 32);
    const int m = __shfl_sync(kAll, n, g);
    Ray w;
#pragma unroll
    for (int i = 0; i < 3; i++) w.o[i] = r.o[i], w.d[i] = __shfl_sync(kAll, r.d[i], g);
    w.dd = __shfl_sync(kAll, r.dd, g);
    const float inv_dd = __frcp_rn(w.dd);
    for (int b = lane; b < 2 * kBins; b += 32) reinterpret_cast<int*>(pool)[b] = 0;
    auto entry_at = [&](int i, float4& p) {
      const int idx = i < m ? from[i] : -1;  // listed but not kept: below 0, too
      p = make_float4(0.f, 0.f, 0.f, 0.f);
      if (idx >= 0) p = __ldg(a.pts + idx);
      return idx >= 0;
    };
    float tmin = 1e3f;
    for (int i0 = 0; i0 < m; i0 += 32) {
      float4 p;
      if (entry_at(i0 + lane, p)) tmin = fminf(tmin, ray_t(w, inv_dd, p));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tmin = fminf(tmin, __shfl_xor_sync(kAll, tmin, o));
    __syncwarp();
    for (int i0 = 0; i0 < m; i0 += 32) {
      float4 p;
      bool in = entry_at(i0 + lane, p);
      const float t = ray_t(w, inv_dd, p);
      const int b = bin_index(a.bins, in, __fsub_rn(t, tmin));
      const float dist = norm3df(__fsub_rn(p.x, __fmaf_rn(t, w.d[0], w.o[0])), __fsub_rn(p.y, __fmaf_rn(t, w.d[1], w.o[1])),
                                 __fsub_rn(p.z, __fmaf_rn(t, w.d[2], w.o[2])));
      in = in && b < kBins;
      // a bin's first lane adds those of the bin in order
      const unsigned peers = __match_any_sync(kAll, in ? b : kBins + lane);
      const bool first = in && (peers & before) == 0u;
      unsigned rest = first ? peers : 0u;
      float sum = first ? sums[b] : 0.0f;
      while (__any_sync(kAll, rest != 0u)) {
        const float x = __shfl_sync(kAll, dist, rest ? __ffs(rest) - 1 : lane);
        if (rest) sum = __fadd_rn(sum, x);
        rest &= rest - 1;
      }
      if (first) sums[b] = sum, counts[b] += __popc(peers);
      __syncwarp();
    }
    const size_t slot0 = (size_t)__shfl_sync(kAll, ray, g) * S;
    float transmit = 1.0f;
    int out = 0;
    bool more = true;
    for (int b0 = 0; b0 < kBins && more; b0 += 32) {
      const int cnt = counts[b0 + lane];
      unsigned used = __ballot_sync(kAll, cnt > 1);
      if (!used) continue;
      const float sdf = __fdiv_rn(sums[b0 + lane], __fadd_rn((float)cnt, 1e-6f));
      const float alpha = __fmul_rn(a.opt.gamma, __expf(__fdiv_rn(-sdf, a.opt.alpha_g)));
      const float t = __fmaf_rn((float)(b0 + lane), a.opt.t_intvl, tmin);
      int slot = -1;
      while (used && more) {
        const int src = __ffs(used) - 1;
        used &= used - 1;
        const float al = __shfl_sync(kAll, alpha, src);
        more = !(transmit < 1e-3f || out >= S);
        if (more) {
          if (__fmul_rn(al, transmit) > 1e-3f) {
            if (lane == src) slot = out;
            out++;
          }
          transmit = __fsub_rn(transmit, al);
        }
      }
      if (slot >= 0) {
        const size_t at = slot0 + slot;
#pragma unroll
        for (int i = 0; i < 3; i++) a.sp_xyz[at * 3 + i] = __fmaf_rn(t, w.d[i], w.o[i]);
        a.sp_t[at] = t;
        a.mask[at] = 1;
      }
    }
    if (gb == g) emitted = out, balls = out > 0;
    __syncwarp();
  }

  // point selection (epcq_render_topk.cu:10-81): lanes 0..7 of a group hold its buffer's slots
  const size_t slot0 = (size_t)(ray < 0 ? 0 : ray) * S;
  const int most = __reduce_max_sync(kAll, balls ? emitted : 0), nball = __reduce_max_sync(kAll, balls ? n : 0);
  for (int s = 0; s < most; s++) {
    const bool on = balls && s < emitted;
    const float ts = on ? *(volatile const float*)(a.sp_t + slot0 + s) : 0.0f;
    const float sx = __fmaf_rn(ts, r.d[0], r.o[0]), sy = __fmaf_rn(ts, r.d[1], r.o[1]), sz = __fmaf_rn(ts, r.d[2], r.o[2]);
    float held = 0.0f, farthest = 1e3f;  // this lane's slot; the group's "farthest" entry and its slot
    int held_id = -1, size = 0, at = 0;
    bool settled = false;  // one was replaced: `farthest` is the maximum (before: the minimum of what came)
    for (int i0 = 0; i0 < nball; i0 += L) {
      float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
      const bool in = on && i0 + sl < n;
      if (in) p = __ldg(a.pts + (list[i0 + sl] & 0x7fffffff));
      const float e0 = __fsub_rn(sx, p.x), e1 = __fsub_rn(sy, p.y), e2 = __fsub_rn(sz, p.z);
      const bool look = in && !(squared(e0, e1, e2) > rt.hi2);
      if (!__any_sync(kAll, look)) continue;
      const float dist = norm3df(e0, e1, e2);
      const bool hit = look && dist < rt.r;
      // those that can change the buffer: all while it fills; then those below `farthest`, and, before the first of
      // these has replaced an entry, any after it
      const unsigned hits = __ballot_sync(kAll, hit) & gmask, nearer = __ballot_sync(kAll, hit && dist < farthest) & gmask;
      unsigned todo = size < kBallBuf ? hits : settled ? nearer : nearer ? hits & ~((nearer & -nearer) - 1u) : 0u;
      while (__any_sync(kAll, todo != 0u)) {
        const int src = todo ? __ffs(todo) - 1 : lane;
        const float x = __shfl_sync(kAll, dist, src);
        const int id = __shfl_sync(kAll, __float_as_int(p.w), src);
        const bool fill = todo && size < kBallBuf, swap = todo && !fill && x < farthest;
        if (fill || swap) {
          const int slot = fill ? size : at;
          if (sl == slot) held = x, held_id = id;
        }
        if (fill) {
          if (farthest > x) farthest = x, at = size;
          size++;
        }
        if (__any_sync(kAll, swap)) {  // the new maximum: the slot just filled if it holds it, else the first that does
          float top = sl < kBallBuf ? held : -1.0f;
#pragma unroll
          for (int o = kBallBuf / 2; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(kAll, top, o));
          top = __shfl_sync(kAll, top, gb);
          const unsigned tops = __ballot_sync(kAll, sl < kBallBuf && held == top) & gmask;
          if (swap) {
            if (top != x) at = __ffs(tops) - 1 - gb;
            farthest = top;
            settled = true;
          }
        }
        todo &= todo - 1;
      }
    }
    if (on) {
      int* row = a.pc_idx + (slot0 + s) * P;
      if (sl < kBallBuf && sl < P) row[sl] = sl < size ? held_id : -1;
      for (int e = kBallBuf + sl; e < P; e += L) row[e] = -1;
    }
  }
  if ((walks >> lane) & 1u) default_slots(a, (size_t)ray, emitted, sl, L);
  return over;
}

// All that serve_rays leaves; one call, out of line: called one by one, the two
// took registers from the rays that never come here (shapes view 446 us, so 425).
template <class J>
__device__ __noinline__ void serve_left(const SampleArgs& a, int L, int4 entry, unsigned char* pool, int entries,
                                        Unsettled left, unsigned over) {
#ifdef HP_TESTING  // by the general walk, to hold serve_exact against it
  over |= __ballot_sync(0xffffffffu, left.n < 0 || left.emitted < 0 || left.balls);
#else
  over |= serve_exact(a, L, entry, pool, entries, left);
#endif
  while (over) {  // the general walk, ray by ray
    const int l = __ffs(over) - 1;
    over &= ~((0xffffffffu >> (32 - L)) << l);
    const int ray = __shfl_sync(0xffffffffu, entry.x, l);
    __syncwarp();
    sample_ray_warp<J>(a, ray / a.cam.width, ray % a.cam.width, reinterpret_cast<unsigned*>(pool));
  }
}

// ---------------------------------------------------------------------------
// the ray list
// ---------------------------------------------------------------------------
// Rays of one kTileH x kTileW tile, one thread per pixel: the window counts by
// rows then columns from the tile's halo in shared memory; default outputs for
// rays without a candidate; the others into the list, ordered by count so that
// the four rays of a unit run loops of the same length.
template <int kTileH, int kTileW>
__device__ __forceinline__ void list_tile(const SampleArgs& a, int v0, int u0, int view, const RayList& rl) {
  constexpr int kHaloH = kTileH + kMaxKernel - 1, kHaloW = kTileW + kMaxKernel - 1;
  constexpr int kFlag = 1 << 26;  // a cell above 48 entries; 25 cells' counts stay below it
  __shared__ int halo[kHaloH * kHaloW];
  __shared__ int row_sum[kHaloH][kTileW];
  __shared__ int cls[kClasses], cls_base[kClasses];
  __shared__ unsigned empty[kTileH];
  __shared__ unsigned s_front, s_back;
  const int tid = threadIdx.x, lane = tid & 31;
  const int W = a.cam.width, H = a.cam.height, k = a.opt.k;
  const int koff = (k + 1) >> 1, lo = koff - 1, hi = k - koff;
  const int rv0 = max(0, v0 - lo), rv1 = min(H - 1, v0 + kTileH - 1 + hi);
  const int ru0 = max(0, u0 - lo), ru1 = min(W - 1, u0 + kTileW - 1 + hi);
  const int nv = rv1 - rv0 + 1, nu = ru1 - ru0 + 1;
  if (tid < kClasses) cls[tid] = 0;
  for (int c = tid; c < nv * nu; c += kThreads) {
    const int vv = c / nu;
    const int2 rg = cell_range(a, rv0 + vv, ru0 + (c - vv * nu));
    const int n = min(rg.y - rg.x, 1 << 20);
    halo[c] = n > kKeptPerCell ? n | kFlag : n;
  }
  __syncthreads();
  for (int c = tid; c < nv * kTileW; c += kThreads) {
    const int vv = c / kTileW, uu = c % kTileW;
    int s = 0;
    for (int q = -lo; q <= hi; q++) s += halo[vv * nu + min(max(u0 + uu + q, ru0), ru1) - ru0];
    row_sum[vv][uu] = s;
  }
  __syncthreads();
  const int pv = v0 + tid / kTileW, pu = u0 + tid % kTileW;
  const bool in = pv < H && pu < W;
  int s = 0;
  if (in)
    for (int q = -lo; q <= hi; q++) s += row_sum[min(max(pv + q, 0), H - 1) - rv0][tid % kTileW];
  const int T = s & (kFlag - 1);
  // whole-warp rays: many candidates, a cell above the cap, or repeated (clamped) columns
  const bool back = T > 0 && (T > rl.light || s >= kFlag || pu - lo < 0 || pu + hi > W - 1);
  const unsigned none = __ballot_sync(0xffffffffu, in && T == 0);
  if constexpr (kTileW == 32) {
    if (lane == 0) empty[tid >> 5] = none;
  } else {
    if (lane == 0) empty[(tid >> 5) * 2] = none & 0xffffu, empty[(tid >> 5) * 2 + 1] = none >> 16;
  }
  // class 0: whole-warp rays; then by descending count in steps of 8 candidates; last: no candidate
  const int c = T == 0 ? kClasses - 1 : back ? 0 : 1 + max(0, kClasses - 3 - (T >> 3));
  const int local = atomicAdd(&cls[c], 1);
  __syncthreads();
  if (tid < 32) {
    const int n0 = cls[2 * tid], n1 = cls[2 * tid + 1];
    int incl = n0 + n1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (tid >= o) incl += t;
    }
    cls_base[2 * tid] = incl - n0 - n1;
    cls_base[2 * tid + 1] = incl - n1;
  }
  __syncthreads();
  const int nback = cls[0], nfront = kThreads - nback - cls[kClasses - 1];
  if (tid == 0) {
    s_front = nfront ? atomicAdd(rl.counts, (unsigned)((nfront + 3) & ~3)) : 0u;
    s_back = nback ? atomicAdd(rl.counts + 1, (unsigned)nback) : 0u;
  }
  __syncthreads();
  if (T > 0) {
    Ray r;
    make_ray(a.cam.c2w, a.cam.fx, a.cam.fy, a.cam.cx, a.cam.cy, pu, pv, r);
    const int4 e = make_int4(pv * W + pu, __float_as_int(r.d[0]), __float_as_int(r.d[1]), __float_as_int(r.d[2]));
    if (back) {
      const long long i = (long long)s_back + local;
      rl.rays[rl.cap - 1 - i] = e;
      if (rl.back_view) rl.back_view[i] = view;
    } else {
      const long long i = (long long)s_front + cls_base[c] - nback + local;
      rl.rays[i] = e;
      if (rl.front_view && (i & 3) == 0) rl.front_view[i >> 2] = view;
    }
  }
  if (tid < ((nfront + 3) & ~3) - nfront) rl.rays[(long long)s_front + nfront + tid] = make_int4(-1, 0, 0, 0);

  // default outputs of the rays without a candidate: a tile row's outputs are runs, written in order
  const int S = a.opt.S, P = a.opt.P;
  const int cols = min(kTileW, W - u0);
  for (int q = tid >> 5; q < kTileH && v0 + q < H; q += kWarps) {
    const unsigned m = empty[q];
    if (!m) continue;
    const size_t ray0 = (size_t)(v0 + q) * W + u0;
    auto fill4 = [&](void* base, int words, unsigned inverse, int value) {  // `words` 32-bit words a ray
      int* out = reinterpret_cast<int*>(base) + ray0 * words;
      const bool vec = (words & 3) == 0 && ((uintptr_t)base & 15) == 0;
      const int n = cols * words, step = vec ? 4 : 1;
      const int4 x = make_int4(value, value, value, value);
      for (int e = lane * step; e < n; e += 32 * step) {
        const unsigned ray = inverse ? __umulhi((unsigned)e, inverse) : (unsigned)e / (unsigned)words;
        if ((m >> ray) & 1u) {
          if (vec)
            *reinterpret_cast<int4*>(out + e) = x;
          else
            out[e] = value;
        }
      }
    };
    fill4(a.pc_idx, S * P, a.inv_idx, -1);
    fill4(a.sp_xyz, S * 3, a.inv_xyz, 0);
    fill4(a.sp_t, S, a.inv_t, 0);
    if ((S & 3) == 0 && ((uintptr_t)a.mask & 3) == 0) {
      int* out = reinterpret_cast<int*>(a.mask + ray0 * S);
      for (int e = lane; e < cols * (S >> 2); e += 32) {
        const unsigned ray = a.inv_t ? __umulhi((unsigned)e * 4u, a.inv_t) : (unsigned)e * 4u / (unsigned)S;
        if ((m >> ray) & 1u) out[e] = 0;
      }
    } else {
      for (int e = lane; e < cols * S; e += 32)
        if ((m >> (unsigned)(e / S)) & 1u) a.mask[ray0 * S + e] = 0;
    }
  }
}

// One block per tile, then the blocks that pack the candidates (which need no
// result of the tiles, so they fill in where a tile's blocks wait; interleaved
// with them they were no faster).  Bound by its writes and the packing's gather:
// 41 us cold for 1M points at 800 x 800 (48 us with 4 resident blocks and each
// tile's warps packing a share), 16 us of it the list alone.
template <int kTileH, int kTileW>
__global__ void __launch_bounds__(kThreads, 8) k_ray_list(const __grid_constant__ SampleArgs a, RayList rl,
                                                         int tiles_x, int ntiles) {
  const int t = blockIdx.x;
  if (t >= ntiles)
    pack_block(a, t - ntiles);
  else
    list_tile<kTileH, kTileW>(a, (t / tiles_x) * kTileH, (t % tiles_x) * kTileW, 0, rl);
}

// The persistent warps: the rays of a whole warp first (they run longest), then
// the units of four.  Each takes its next position before it serves the current one.
template <class Cfg, bool kBatch>
__device__ __forceinline__ void serve_list(const SampleArgs& a0, const SampleArgs* __restrict__ args, const RayList& rl,
                                           unsigned char* smem) {
  __shared__ SampleArgs s_args[kBatch ? kServeWarps : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned char* pool = smem + warp * Cfg::kWarpBytes;
  int have = -1;  // the view in s_args[warp]
  auto view_args = [&](int view) {
    if (view != have) {
      __syncwarp();
      if (lane == 0) s_args[warp] = args[view];
      __syncwarp();
      have = view;
    }
  };
  const SampleArgs& a = kBatch ? static_cast<const SampleArgs&>(s_args[warp]) : a0;
  const unsigned n_front = rl.counts[0], n_back = rl.counts[1];
  auto take = [&](unsigned* next, unsigned n) {
    unsigned x = 0;
    if (lane == 0) x = atomicAdd(next, n);
    return x;
  };
  const unsigned units = n_front >> 2;
  const unsigned step = max(1u, min(4u, units / (gridDim.x * kServeWarps * 8u)));
  // One loop over both parts of the list, so that serve_rays is in the kernel once: two copies of it
  // (or three, with one for 16 lanes) cost more in instruction-cache misses than their constants saved.
  bool back = true;
  unsigned x = take(rl.counts + 3, 1u), i = 0, end = 0;
  for (;;) {
    if (i == end) {
      i = __shfl_sync(0xffffffffu, x, 0);
      if (back && i >= n_back) {
        back = false;
        i = __shfl_sync(0xffffffffu, take(rl.counts + 2, step), 0);
      }
      if (!back && i >= units) break;
      end = back ? i + 1 : min(units, i + step);
      x = take(rl.counts + (back ? 3 : 2), back ? 1u : step);
    }
    const int L = back ? 32 : 8;
    const int4 e = __ldg(back ? rl.rays + (rl.cap - 1 - (long long)i) : rl.rays + (size_t)i * 4 + (lane >> 3));
    if constexpr (kBatch) view_args(back ? rl.back_view[i] : rl.front_view[i]);
    Unsettled left;
    const unsigned over = serve_rays(a, L, e, pool, Cfg::kEntries, left);
    if (__any_sync(0xffffffffu, left.n < 0 || left.emitted < 0 || left.balls) || over)
      serve_left<typename Cfg::Index>(a, L, e, pool, Cfg::kEntries, left, over);
    __syncwarp();
    i++;
  }
}

template <class Cfg>
__global__ void __launch_bounds__(kServeThreads, Cfg::kBlocks) k_quick_sampling(const __grid_constant__ SampleArgs a,
                                                                   RayList rl) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  serve_list<Cfg, false>(a, nullptr, rl, smem_raw);
}

// ---------------------------------------------------------------------------
// Batched launch: the rays of many views (different clouds, cameras, image
// sizes and options) in one list and one persistent kernel, so a view's tail
// overlaps the other views' work.  Every ray runs the same code as in a
// per-view launch, so the outputs are identical.

// Device view table -> per-view kernel arguments and the first global tile of
// each view (exclusive scan; tile_base[n_views] = all tiles).  One warp.
// Also the first packed-point slot of each view (pack_base; regions padded to
// 16 slots) and the views' packed-point arrays inside `pts`.
__global__ void k_batch_setup(const hp_view* __restrict__ views, int n_views, int tile_h, int tile_w,
                              SampleArgs* __restrict__ args, int* __restrict__ tile_base, int* __restrict__ pack_base,
                              float4* __restrict__ pts) {
  const int lane = threadIdx.x;
  int run = 0, prun = 0;
  for (int b = 0; b < n_views; b += 32) {
    const int v = b + lane;
    int tiles = 0, slots = 0;
    if (v < n_views) slots = ((int)views[v].n_sorted + 15) & ~15;
    int pincl = slots;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, pincl, o);
      if (lane >= o) pincl += t;
    }
    const int pfirst = prun + pincl - slots;
    if (v < n_views) pack_base[v] = pfirst;
    prun += __shfl_sync(0xffffffffu, pincl, 31);
    if (v < n_views) {
      const hp_view& hv = views[v];
      SampleArgs a;
      a.xyz = hv.xyz;
      a.sidx = hv.sorted_point_idx;
      a.pts = pts + pfirst;
      a.hash = (const int2*)hv.hash_table;
      a.n_points = (int)hv.n_points;
      a.n_sorted = (int)hv.n_sorted;
      a.cam.c2w = hv.cam.c2w;
      a.cam.fx = hv.cam.fx;
      a.cam.fy = hv.cam.fy;
      a.cam.cx = hv.cam.cx;
      a.cam.cy = hv.cam.cy;
      a.cam.width = hv.cam.width;
      a.cam.height = hv.cam.height;
      a.opt.k = hv.opt.kernel_size;
      a.opt.t_intvl = hv.opt.t_intvl;
      a.opt.radius = hv.opt.radius_threshold;
      a.opt.S = hv.opt.num_sample_points_per_ray;
      a.opt.P = hv.opt.num_point_cloud_per_sp;
      a.opt.num_point_per_ray = hv.opt.num_point_per_ray;
      a.opt.alpha_g = hv.opt.sdf2weight_gaussian_alpha;
      a.opt.gamma = hv.opt.sdf2weight_gaussian_gamma;
      a.sp_xyz = hv.sp_xyz;
      a.pc_idx = hv.pc_idx;
      a.sp_t = hv.sp_t;
      a.mask = hv.mask;
      derive_args(a);
      args[v] = a;
      tiles = ((hv.cam.width + tile_w - 1) / tile_w) * ((hv.cam.height + tile_h - 1) / tile_h);
    }
    int incl = tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (v < n_views) tile_base[v] = run + incl - tiles;
    run += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) {
    tile_base[n_views] = run;
    pack_base[n_views] = prun;
  }
}

// Pack every view's candidates (see packed_point); slot g of the batch.
__global__ void k_batch_pack(const SampleArgs* __restrict__ args, const int* __restrict__ pack_base, int n_views,
                             int total) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= total) return;
  int lo = 0, hi = n_views;  // pack_base[lo] <= g < pack_base[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (pack_base[mid] <= g)
      lo = mid;
    else
      hi = mid;
  }
  const SampleArgs& a = args[lo];
  const int j = g - pack_base[lo];
  if (j >= a.n_sorted) return;
  const_cast<float4*>(a.pts)[j] = packed_point(a.sidx, j, a.xyz, a.n_points);
}

// One block per global tile: find its view, then list the tile's rays.
template <int kTileH, int kTileW>
__global__ void __launch_bounds__(kThreads, 8) k_batch_ray_list(const SampleArgs* __restrict__ args,
                                                                const int* __restrict__ tile_base, int n_views,
                                                                RayList rl) {
  __shared__ SampleArgs s_args;
  const int g = blockIdx.x;
  int lo = 0, hi = n_views;  // tile_base[lo] <= g < tile_base[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (tile_base[mid] <= g)
      lo = mid;
    else
      hi = mid;
  }
  if (threadIdx.x == 0) s_args = args[lo];
  __syncthreads();
  const int tiles_x = (s_args.cam.width + kTileW - 1) / kTileW, t = g - tile_base[lo];
  list_tile<kTileH, kTileW>(s_args, (t / tiles_x) * kTileH, (t % tiles_x) * kTileW, lo, rl);
}

template <class Cfg>
__global__ void __launch_bounds__(kServeThreads, Cfg::kBlocks) k_quick_sampling_batch(const SampleArgs* __restrict__ args, RayList rl) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  serve_list<Cfg, true>(SampleArgs{}, args, rl, smem_raw);
}

__global__ void k_ray_directions(DevCamera cam, float* __restrict__ dirs) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= cam.width * cam.height) return;
  Ray r;
  make_ray(cam.c2w, cam.fx, cam.fy, cam.cx, cam.cy, p % cam.width, p / cam.width, r);
  dirs[3 * (size_t)p + 0] = r.d[0];
  dirs[3 * (size_t)p + 1] = r.d[1];
  dirs[3 * (size_t)p + 2] = r.d[2];
}

// The kernels and shapes of each stage configuration.
struct SamplingKernels {
  void (*view)(SampleArgs, RayList);
  void (*batch)(const SampleArgs*, RayList);
  void (*list)(SampleArgs, RayList, int, int);
  void (*batch_list)(const SampleArgs*, const int*, int, RayList);
  size_t smem;
  int stage, blocks, tile_h, tile_w, entries;
};
template <class Cfg>
static SamplingKernels sampling_kernels() {
  return {k_quick_sampling<Cfg>,
          k_quick_sampling_batch<Cfg>,
          k_ray_list<Cfg::kTileH, Cfg::kTileW>,
          k_batch_ray_list<Cfg::kTileH, Cfg::kTileW>,
          (size_t)Cfg::kSmem,
          Cfg::kStage,
          Cfg::kBlocks,
          Cfg::kTileH,
          Cfg::kTileW,
          Cfg::kEntries};
}
static const SamplingKernels& stage_kernels(int config) {  // config 1..kWideConfig
  static const SamplingKernels table[kWideConfig] = {sampling_kernels<Cfg1>(), sampling_kernels<Cfg2>(),
                                                     sampling_kernels<Cfg3>(), sampling_kernels<Cfg4>(),
                                                     sampling_kernels<Cfg5>(), sampling_kernels<CfgWide>()};
  return table[config - 1];
}

static int64_t tiles_of(int64_t H, int64_t W, int tile_h, int tile_w) {
  return ((W + tile_w - 1) / tile_w) * ((H + tile_h - 1) / tile_h);
}

// Ray-list entries an H x W view can need under any configuration: every ray,
// and up to three entries of padding per tile (workspaces are sized for the
// largest, so one workspace serves every tuning).
static int64_t max_view_entries(int64_t H, int64_t W) {
  const int64_t a = tiles_of(H, W, 8, 32), b = tiles_of(H, W, 16, 16);
  return H * W + 3 * (a > b ? a : b);
}

// Opt the configuration's kernels in to their dynamic shared memory once per
// device and size the persistent grid from their occupancy.
int32_t sampling_grid(int config, int* blocks, int* sm_count = nullptr) {
  static std::mutex mu;
  static int grid[128][kWideConfig] = {{0}}, sm_counts[128] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return set_error(HP_ERR_CUDA, "hp_quick_sampling: cudaGetDevice failed");
  if (dev < 0 || dev >= 128)
    return set_error(HP_ERR_UNSUPPORTED, "hp_quick_sampling: device ordinal %d is beyond the 128 devices it tracks",
                     dev);
  std::lock_guard<std::mutex> lock(mu);
  int& g = grid[dev][config - 1];
  if (!g) {
    const SamplingKernels& K = stage_kernels(config);
    cudaError_t e = cudaFuncSetAttribute(K.view, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)K.smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(K.batch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)K.smem);
    int sms = 0, per_sm = 0;
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, K.view, kServeThreads, K.smem);
    if (e != cudaSuccess) return set_error(HP_ERR_CUDA, "hp_quick_sampling: kernel set-up: %s", cudaGetErrorString(e));
    g = sms * (per_sm > 0 ? per_sm : 1);
    sm_counts[dev] = sms;
  }
  *blocks = g;
  if (sm_count) *sm_count = sm_counts[dev];
  return HP_OK;
}

// Launch tuning shared by both entry points; outputs never depend on it.
struct Tune {
  int heavy = kHeavyWindow, per_sm = 0, config = kDefaultStageConfig;
};

static int32_t read_tuning(const char* who, const hp_tuning* tuning, Tune& t) {
  if (!tuning) return HP_OK;
  if (tuning->heavy_window < 0 || tuning->heavy_window > kMaxHeavyWindow || tuning->blocks_per_sm < 0 ||
      tuning->stage_config < 0 || tuning->stage_config > kStageConfigs)
    return set_error(HP_ERR_INVALID_ARGUMENT,
                     "%s: tuning out of range (heavy_window 0..%d, blocks_per_sm >= 0, stage_config 0..%d)", who,
                     kMaxHeavyWindow, kStageConfigs);
  if (tuning->heavy_window > 0) t.heavy = tuning->heavy_window;
  t.per_sm = tuning->blocks_per_sm;
  if (tuning->stage_config > 0) t.config = tuning->stage_config;
  return HP_OK;
}

static constexpr size_t align256s(size_t x) { return (x + 255) & ~(size_t)255; }

struct ListLayout {
  size_t counts, rays, pts, total;
};

static ListLayout list_layout(int64_t H, int64_t W, int64_t n_sorted) {
  ListLayout L;
  L.counts = 0;
  L.rays = 256;
  L.pts = L.rays + align256s(sizeof(int4) * (size_t)max_view_entries(H, W));
  L.total = L.pts + align256s(sizeof(float4) * (size_t)n_sorted);
  return L;
}

// Batched launch: the list over all views' rays with each unit's view, then the
// per-view arguments, the views' first tiles and room for a copy of the view table.
struct BatchLayout {
  size_t counts, rays, front_view, back_view, args, tile_base, pack_base, views, pts, total;
};

static BatchLayout batch_layout(int64_t entries, int n_views, int64_t total_slots) {
  BatchLayout B;
  B.counts = 0;
  B.rays = 256;
  B.front_view = B.rays + align256s(sizeof(int4) * (size_t)entries);
  B.back_view = B.front_view + align256s(sizeof(int) * (size_t)(entries / 4 + 1));
  B.args = B.back_view + align256s(sizeof(int) * (size_t)entries);
  B.tile_base = B.args + align256s(sizeof(SampleArgs) * (size_t)n_views);
  B.pack_base = B.tile_base + align256s(sizeof(int) * (size_t)(n_views + 1));
  B.views = B.pack_base + align256s(sizeof(int) * (size_t)(n_views + 1));
  B.pts = B.views + align256s(sizeof(hp_view) * (size_t)n_views);
  B.total = B.pts + sizeof(float4) * (size_t)total_slots;
  return B;
}

int32_t check_camera(const hp_camera* cam, const char* who) {
  if (!cam) return set_error(HP_ERR_INVALID_ARGUMENT, "%s: cam is NULL", who);
  if (cam->height <= 0 || cam->width <= 0 || (int64_t)cam->height * cam->width >= (1ll << 31))
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: bad image size %dx%d", who, cam->height, cam->width);
  if (!cam->c2w) return set_error(HP_ERR_INVALID_ARGUMENT, "%s: c2w is NULL", who);
  return HP_OK;
}

DevCamera dev_camera(const hp_camera* cam) {
  DevCamera d;
  d.c2w = cam->c2w;
  d.fx = cam->fx;
  d.fy = cam->fy;
  d.cx = cam->cx;
  d.cy = cam->cy;
  d.width = cam->width;
  d.height = cam->height;
  return d;
}

DevOptions dev_options(const hp_options* o) {
  DevOptions d;
  d.k = o->kernel_size;
  d.t_intvl = o->t_intvl;
  d.radius = o->radius_threshold;
  d.S = o->num_sample_points_per_ray;
  d.P = o->num_point_cloud_per_sp;
  d.num_point_per_ray = o->num_point_per_ray;
  d.alpha_g = o->sdf2weight_gaussian_alpha;
  d.gamma = o->sdf2weight_gaussian_gamma;
  return d;
}

}  // namespace hp

using namespace hp;

extern "C" size_t hp_quick_sampling_workspace_size(int64_t n_sorted, int32_t height, int32_t width) {
  if (height <= 0 || width <= 0 || n_sorted < 0) return 0;
  return list_layout(height, width, n_sorted).total;
}

// Argument checks shared by the per-view and batched entry points.
static int32_t check_sampling(const char* who, const float* xyz, int64_t n_points, const hp_camera* cam,
                              const hp_options* opt, const int32_t* sorted_point_idx, int64_t n_sorted,
                              const int32_t* hash_table, const float* sp_xyz, const int32_t* pc_idx, const float* sp_t,
                              const uint8_t* mask) {
  if (int32_t rc = check_camera(cam, who)) return rc;
  if (!opt) return set_error(HP_ERR_INVALID_ARGUMENT, "%s: opt is NULL", who);
  if (opt->kernel_size < 1 || opt->kernel_size > kMaxKernel)
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: kernel_size %d outside 1..%d (the reference's windows hold 32 cells)",
                     who, opt->kernel_size, kMaxKernel);
  if (!(opt->t_intvl > 0.0f)) return set_error(HP_ERR_INVALID_ARGUMENT, "%s: t_intvl must be > 0", who);
  if (opt->num_sample_points_per_ray < 1 || opt->num_point_cloud_per_sp < 1)
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: num_sample_points_per_ray and num_point_cloud_per_sp must be >= 1",
                     who);
  const int64_t hw = (int64_t)cam->height * cam->width;
  if (tiles_of(cam->height, cam->width, 16, 16) >= kMaxTilesPerView ||
      tiles_of(cam->height, cam->width, 8, 32) >= kMaxTilesPerView)
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: image too large (%lld pixels)", who, (long long)hw);
  if (hw * opt->num_sample_points_per_ray * (int64_t)(opt->num_point_cloud_per_sp > 3 ? opt->num_point_cloud_per_sp : 3) >=
      (1ll << 40))
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: output too large", who);
  if (n_points < 0 || n_points >= (1ll << 31) || n_sorted < 0 || n_sorted >= (1ll << 31))
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: n_points / n_sorted out of range", who);
  if (!hash_table || !sp_xyz || !pc_idx || !sp_t || !mask || (n_points > 0 && !xyz) ||
      (n_sorted > 0 && !sorted_point_idx))
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: null pointer", who);
  if (((uintptr_t)hash_table & 7) != 0)
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: hash_table must be 8-byte aligned", who);
  return HP_OK;
}

extern "C" int32_t hp_stage_config_info(int32_t config, int32_t* tile_h, int32_t* tile_w, int32_t* stage_points,
                                        int32_t* blocks_per_sm) {
  if (config == 0) config = kDefaultStageConfig;
  if (config < 1 || config > kStageConfigs)
    return set_error(HP_ERR_INVALID_ARGUMENT, "hp_stage_config_info: stage_config %d outside 0..%d", config,
                     kStageConfigs);
  const SamplingKernels& K = stage_kernels(config);
  if (tile_h) *tile_h = K.tile_h;
  if (tile_w) *tile_w = K.tile_w;
  if (stage_points) *stage_points = K.stage;
  if (blocks_per_sm) *blocks_per_sm = K.blocks;
  return HP_OK;
}

extern "C" int32_t hp_quick_sampling_tuned(const float* xyz, int64_t n_points, const hp_camera* cam,
                                           const hp_options* opt, const int32_t* sorted_point_idx, int64_t n_sorted,
                                           const int32_t* hash_table, float* sp_xyz, int32_t* pc_idx, float* sp_t,
                                           uint8_t* mask, const hp_tuning* tuning, void* workspace,
                                           size_t workspace_bytes, hp_stream_t stream) {
  if (int32_t rc = check_sampling("hp_quick_sampling", xyz, n_points, cam, opt, sorted_point_idx, n_sorted, hash_table,
                                  sp_xyz, pc_idx, sp_t, mask))
    return rc;
  Tune tn;
  if (int32_t rc = read_tuning("hp_quick_sampling", tuning, tn)) return rc;
  if (n_sorted > kIntIds) tn.config = kWideConfig;
  const ListLayout L = list_layout(cam->height, cam->width, n_sorted);
  if (!workspace || workspace_bytes < L.total || ((uintptr_t)workspace & 255) != 0)
    return set_error(HP_ERR_WORKSPACE, "hp_quick_sampling: workspace needs %zu bytes, 256-byte aligned (got %zu)",
                     L.total, workspace_bytes);
  SampleArgs a;
  a.xyz = xyz;
  a.sidx = sorted_point_idx;
  a.pts = (const float4*)((char*)workspace + L.pts);
  a.hash = (const int2*)hash_table;
  a.n_points = (int)n_points;
  a.n_sorted = (int)n_sorted;
  a.cam = dev_camera(cam);
  a.opt = dev_options(opt);
  a.sp_xyz = sp_xyz;
  a.pc_idx = pc_idx;
  a.sp_t = sp_t;
  a.mask = mask;
  derive_args(a);
  int blocks = 0, sms = 0;
  if (int32_t rc = sampling_grid(tn.config, &blocks, &sms)) return rc;
  if (tn.per_sm > 0 && tn.per_sm * sms < blocks) blocks = tn.per_sm * sms;
  const SamplingKernels& K = stage_kernels(tn.config);
  const int tiles_x = (cam->width + K.tile_w - 1) / K.tile_w;
  const int ntiles = (int)tiles_of(cam->height, cam->width, K.tile_h, K.tile_w);
  char* ws = (char*)workspace;
  RayList rl;
  rl.rays = (int4*)(ws + L.rays);
  rl.cap = max_view_entries(cam->height, cam->width);
  rl.counts = (unsigned*)(ws + L.counts);
  rl.front_view = rl.back_view = nullptr;
  rl.light = tn.heavy < K.entries / 4 ? tn.heavy : K.entries / 4;
  cudaStream_t st = (cudaStream_t)stream;
  if (cudaMemsetAsync(rl.counts, 0, 4 * sizeof(unsigned), st) != cudaSuccess)
    return set_error(HP_ERR_CUDA, "hp_quick_sampling: cudaMemsetAsync failed");
  const int packs = (int)((n_sorted + kPackPerBlock - 1) / kPackPerBlock);
  K.list<<<ntiles + packs, kThreads, 0, st>>>(a, rl, tiles_x, ntiles);
  if (int32_t rc = check_launch("k_ray_list")) return rc;
  // at least a unit of four rays a warp
  const int64_t most = (int64_t)ntiles * (kThreads / 4 / kServeWarps);
  K.view<<<blocks < most ? blocks : (int)most, kServeThreads, K.smem, st>>>(a, rl);
  return check_launch("k_quick_sampling");
}

extern "C" int32_t hp_quick_sampling(const float* xyz, int64_t n_points, const hp_camera* cam, const hp_options* opt,
                                     const int32_t* sorted_point_idx, int64_t n_sorted, const int32_t* hash_table,
                                     float* sp_xyz, int32_t* pc_idx, float* sp_t, uint8_t* mask, void* workspace,
                                     size_t workspace_bytes, hp_stream_t stream) {
  return hp_quick_sampling_tuned(xyz, n_points, cam, opt, sorted_point_idx, n_sorted, hash_table, sp_xyz, pc_idx, sp_t,
                                 mask, nullptr, workspace, workspace_bytes, stream);
}

// packed-point slots of a batch: each view's n_sorted rounded up to 16
static int64_t batch_slots(const hp_view* views, int32_t n_views) {
  int64_t total = 0;
  for (int32_t v = 0; v < n_views; v++) total += (views[v].n_sorted + 15) & ~(int64_t)15;
  return total;
}

static int64_t batch_tiles(const hp_view* views, int32_t n_views, int tile_h, int tile_w) {
  int64_t total = 0;
  for (int32_t v = 0; v < n_views; v++) total += tiles_of(views[v].cam.height, views[v].cam.width, tile_h, tile_w);
  return total;
}

// Ray-list entries a batch can need under any configuration.
static int64_t batch_entries(const hp_view* views, int32_t n_views) {
  int64_t total = 0;
  for (int32_t v = 0; v < n_views; v++) total += max_view_entries(views[v].cam.height, views[v].cam.width);
  return total;
}

extern "C" size_t hp_quick_sampling_batch_workspace_size(const hp_view* views, int32_t n_views) {
  if (!views || n_views <= 0) return 0;
  for (int32_t v = 0; v < n_views; v++)
    if (views[v].cam.width <= 0 || views[v].cam.height <= 0 || views[v].n_sorted < 0) return 0;
  return batch_layout(batch_entries(views, n_views), n_views, batch_slots(views, n_views)).total;
}

extern "C" int32_t hp_quick_sampling_batch(const hp_view* views, const hp_view* views_device, int32_t n_views,
                                           const hp_tuning* tuning, void* workspace, size_t workspace_bytes,
                                           hp_stream_t stream) {
  static const char* who = "hp_quick_sampling_batch";
  if (!views || n_views <= 0) return set_error(HP_ERR_INVALID_ARGUMENT, "%s: no views", who);
  Tune tn;
  if (int32_t rc = read_tuning(who, tuning, tn)) return rc;
  for (int32_t v = 0; v < n_views; v++) {
    const hp_view& hv = views[v];
    if (int32_t rc = check_sampling(who, hv.xyz, hv.n_points, &hv.cam, &hv.opt, hv.sorted_point_idx, hv.n_sorted,
                                    hv.hash_table, hv.sp_xyz, hv.pc_idx, hv.sp_t, hv.mask)) {
      char msg[256];
      snprintf(msg, sizeof(msg), "%s", hp_last_error());
      return set_error(rc, "%s (view %d)", msg, v);
    }
    if (hv.n_sorted > kIntIds) tn.config = kWideConfig;
  }
  const int64_t entries = batch_entries(views, n_views);
  const int64_t total_slots = batch_slots(views, n_views);
  if (entries >= (1ll << 32) || total_slots >= (1ll << 31))
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: too many tiles or points in one batch", who);
  const BatchLayout B = batch_layout(entries, n_views, total_slots);
  if (!workspace || workspace_bytes < B.total || ((uintptr_t)workspace & 255) != 0)
    return set_error(HP_ERR_WORKSPACE, "%s: workspace needs %zu bytes, 256-byte aligned (got %zu)", who, B.total,
                     workspace_bytes);
  int blocks = 0, sms = 0;
  if (int32_t rc = sampling_grid(tn.config, &blocks, &sms)) return rc;
  if (tn.per_sm > 0 && tn.per_sm * sms < blocks) blocks = tn.per_sm * sms;
  const SamplingKernels& K = stage_kernels(tn.config);
  const int64_t total_tiles = batch_tiles(views, n_views, K.tile_h, K.tile_w);
  char* ws = (char*)workspace;
  cudaStream_t st = (cudaStream_t)stream;
  if (!views_device) {  // copy the table into the workspace
    if (cudaMemcpyAsync(ws + B.views, views, sizeof(hp_view) * (size_t)n_views, cudaMemcpyHostToDevice, st) !=
        cudaSuccess)
      return set_error(HP_ERR_CUDA, "%s: copying the view table failed", who);
    views_device = (const hp_view*)(ws + B.views);
  }
  RayList rl;
  rl.rays = (int4*)(ws + B.rays);
  rl.cap = entries;
  rl.counts = (unsigned*)(ws + B.counts);
  rl.front_view = (int*)(ws + B.front_view);
  rl.back_view = (int*)(ws + B.back_view);
  rl.light = tn.heavy < K.entries / 4 ? tn.heavy : K.entries / 4;
  SampleArgs* args = (SampleArgs*)(ws + B.args);
  int* tile_base = (int*)(ws + B.tile_base);
  int* pack_base = (int*)(ws + B.pack_base);
  if (cudaMemsetAsync(rl.counts, 0, 4 * sizeof(unsigned), st) != cudaSuccess)
    return set_error(HP_ERR_CUDA, "%s: memset failed", who);
  k_batch_setup<<<1, 32, 0, st>>>(views_device, n_views, K.tile_h, K.tile_w, args, tile_base, pack_base,
                                  (float4*)(ws + B.pts));
  if (int32_t rc = check_launch("k_batch_setup")) return rc;
  if (total_slots > 0) {
    k_batch_pack<<<(unsigned)((total_slots + 255) / 256), 256, 0, st>>>(args, pack_base, n_views, (int)total_slots);
    if (int32_t rc = check_launch("k_batch_pack")) return rc;
  }
  K.batch_list<<<(unsigned)total_tiles, kThreads, 0, st>>>(args, tile_base, n_views, rl);
  if (int32_t rc = check_launch("k_batch_ray_list")) return rc;
  const int64_t most = total_tiles * (kThreads / 4 / kServeWarps);
  K.batch<<<blocks < most ? blocks : (int)most, kServeThreads, K.smem, st>>>(args, rl);
  return check_launch("k_quick_sampling_batch");
}

extern "C" int32_t hp_ray_directions(const hp_camera* cam, float* dirs, hp_stream_t stream) {
  if (int32_t rc = check_camera(cam, "hp_ray_directions")) return rc;
  if (!dirs) return set_error(HP_ERR_INVALID_ARGUMENT, "hp_ray_directions: dirs is NULL");
  const int hw = cam->width * cam->height;
  k_ray_directions<<<(hw + 255) / 256, 256, 0, (cudaStream_t)stream>>>(dev_camera(cam), dirs);
  return check_launch("k_ray_directions");
}
