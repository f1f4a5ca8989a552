// Aggregator forward (epcq/epcq.py:406-507) on the tcgen05 tensor cores.
//
// The reference runs, per valid (sample, point) pair, the 284-wide input
// [feat, PE(feat, 3), PE(dist_feat, 5)] through block1 (284->256->256,
// LeakyReLU) and, with [rgb, dir - ray_d, dir . ray_d] appended, block3
// (263->256->256); the alpha branch (256->1, softplus(x - 1)) and the
// inverse-distance weights then reduce each sample's P points to one alpha and
// one 256-wide feature, which with PE(ray_d, 4) goes through the colour branch
// (280->128->128->128->3, sigmoid).  Everything is fp32 torch, chunked by
// 20000 samples, with boolean-mask gathers and scatters between the layers.
//
// Here two persistent kernels do the whole forward, GEMMs in bf16 with fp32
// accumulation in TMEM:
//
//   k_agg_pairs   one tile = 128 pair rows (128 / P samples), one CTA per SM,
//                 two tiles in flight, warp-specialised:
//                   warps 0-7 and 8-15 (a team per tile) build the tile's
//                              284-wide inputs (positional encodings: one
//                              __sincosf per channel, higher bands by the
//                              double-angle formulas) into the team's operand
//                              A, and run the epilogues: read the team's
//                              accumulator with tcgen05.ld, add the bias,
//                              LeakyReLU, write the next layer's bf16 operand
//                              over the last one's (block3's seven extra
//                              inputs beside it, columns 256..271)
//                              (warp w: TMEM lane quarter w % 4, columns
//                              32 (w / 4 % 2) .. + 31 of each 64);
//                   warp 16    issues tcgen05.mma (M 128, N 256, K 16) from A
//                              and the streamed weights, a layer of one team's
//                              tile, then the same layer of the other's;
//                   warp 17    streams the pre-packed weights (256 outputs x 32
//                              K, 16 KB, 64-byte swizzled) from L2 into a
//                              4-stage ring with cp.async.bulk.
//                 While one team's layer runs on the tensor cores the other
//                 team is in its epilogue or builds its next tile's inputs: a
//                 tile's own steps are one chain, so with one tile at a time
//                 the tensor cores waited for every epilogue and the warps for
//                 every layer.  60,000 samples x 8: 500 -> 382 us, tensor pipe
//                 26 -> 34% active (143,000 x 8: 1141 -> ~800 us).  Of that the
//                 second tile gave 6%, the MMA loop run by a whole warp 15%
//                 (one lane took 590 cycles a chunk of two 128-cycle MMAs), the
//                 biases and alpha weights from shared memory 9%.  Then
//                 warps 16 and 17 issuing by elect.sync with uniform operands:
//                 a layer's wait 5.8 -> 4.5 k cycles, the whole forward of
//                 143,000 x 8, colour branch included, 898 -> 761 us (671 with the steps below).  What is
//                 left is each team's chain: inputs 4 k cycles, four layers of
//                 about 4 k with the other team's in between, three epilogues
//                 2 k each, the last one 8 k, the alphas 2 k.
//   k_agg_color   one CTA = 128 samples at a time: three layers on the tensor
//                 cores, the final 128->3 layer and the sigmoid on the CUDA
//                 cores.  Its weights (144 KB) are loaded once and stay in
//                 shared memory; the next tile's input columns 128.. are
//                 loaded while this tile's hidden layers, whose operand is
//                 columns 0..127, run, and the rest at its end.  A tile's
//                 steps are one chain (load, layer, epilogue, ...), which
//                 bounds the kernel.  143,000 samples, the whole forward: 761
//                 us with the weights streamed for every tile, the load of its
//                 inputs waited for and 8 warps, 710 so.
//   k_agg_scatter alpha and colour of sample m to the m-th set position of
//                 mask_out, zeros elsewhere.
//
// Rows of invalid points are computed like the others (their inputs are the
// zero rows FeatureQuery wrote) and enter the reductions with weight 0, as in
// the reference, where their canvas rows are zeros times weight 0.  Every
// wait is bounded; a wait that gives up sets the CTA's abort flag (the other
// roles' waits then give up at once) and the status word.
#include <cuda_bf16.h>

#include <mutex>

#include "hp_common.cuh"
#include "hp_tc.cuh"
#ifdef HP_TESTING
#include "../../include/hashpoint_b200_testing.h"
#endif

namespace hp {

constexpr int kAggRows = 128;                      // pair rows (or samples) per tile = MMA M
constexpr int kTeams = 2;                          // tiles in flight per CTA
constexpr int kTeamThreads = 256;                  // math warps of a team
constexpr int kMathThreads = kTeams * kTeamThreads;  // warps 0..15
constexpr int kPairThreads = kMathThreads + 64;    // + MMA warp + load warp
constexpr int kColorThreads = 512;
constexpr int kMmaWarp = 16, kLoadWarp = 17;
constexpr int kPairChunkK = 32;                    // pair weight chunk: 256 outputs x 32 K, 64-byte swizzled
constexpr int kChunkK = 64;                        // colour weight chunk: 128 outputs x 64 K, 128-byte swizzled
constexpr int kChunkN = 128;
constexpr unsigned kChunkBytes = 16384;            // either chunk
constexpr int kStages = 4;                         // weight chunks in flight
constexpr int kFeatDim = 32;                       // pc_feat width the layer sizes imply (284 = 32 + 192 + 60)

// pair layers L = 0..3: padded K of the streamed operand (block3.0's seven
// extra inputs, columns 256..262, go through their own K = 16 MMA), real input width
__host__ __device__ constexpr int pair_k(int L) { return L == 0 ? 320 : 256; }
__host__ __device__ constexpr int pair_real_k(int L) { return L == 0 ? 284 : L == 2 ? 263 : 256; }
constexpr int kPairN = 256;
constexpr int kPairChunks = (320 + 256 + 256 + 256) / kPairChunkK;  // 34
// colour layers L = 0..2
__host__ __device__ constexpr int color_k(int L) { return L == 0 ? 320 : 128; }
__host__ __device__ constexpr int color_real_k(int L) { return L == 0 ? 280 : 128; }
constexpr int kColorN = 128;
constexpr int kColorChunks = (320 + 128 + 128) / kChunkK;  // 9
constexpr int kWideK = 320;
constexpr unsigned kATileBytes = kAggRows * kWideK * 2;     // 80 KB: one colour-input tile
constexpr unsigned kW3bBytes = kPairN * 16 * 2;             // block3.0 columns 256..262 (+ zeros), no swizzle

// packed weight buffer: pair chunks, W3b, colour chunks, fp32 parameters
constexpr size_t kPairBytes = (size_t)kPairChunks * kChunkBytes;
constexpr size_t kW3bOff = kPairBytes;
constexpr size_t kColorOff = kW3bOff + kW3bBytes;
constexpr size_t kColorBytes = (size_t)kColorChunks * kChunkBytes;
constexpr size_t kParamOff = kColorOff + kColorBytes;
// (the slots kPB1 and kPB3 are written and not read: these biases come in through the weight blocks)
enum : int {
  kPB1 = 0, kPB2 = 256, kPB3 = 512, kPB4 = 768, kPWA = 1024, kPBA = 1280,
  kPCB1 = 1284, kPCB2 = 1412, kPCB3 = 1540, kPWC4 = 1668, kPCB4 = 2052, kParams = 2056
};
constexpr size_t kPackedBytes = kParamOff + (size_t)kParams * 4;

// A pair operand: columns 0..255 in four 128-byte-swizzled blocks, then columns
// 256..287 in a 64-byte-swizzled one (layer 1's last inputs, block3.0's extra
// ones).  The packed weights' columns 288..319 of layer 1 are zeros and are
// neither streamed nor multiplied.
constexpr int kPairInputK = 288;
static_assert(kPairInputK == 256 + kPairChunkK, "one chunk beyond the 128-byte-swizzled blocks");
constexpr unsigned kTail = kAggRows * 256 * 2;                 // byte offset of the 64-byte-swizzled block
constexpr unsigned kABytes = kTail + kAggRows * 32 * 2;        // 72 KB
__host__ __device__ constexpr int pair_chunks(int L) { return (L == 0 ? kPairInputK : 256) / kPairChunkK; }
__host__ __device__ constexpr int pair_chunk0(int L) { return L == 0 ? 0 : (320 + 256 * (L - 1)) / kPairChunkK; }

// pair kernel shared memory (from a 1024-byte aligned base)
constexpr unsigned kPA = 0;
constexpr unsigned kPStages = kPA + kTeams * kABytes;
constexpr unsigned kPW3b = kPStages + kStages * kChunkBytes;
constexpr unsigned kPBar = kPW3b + kW3bBytes;
constexpr unsigned kPScratch = kPBar + 256;
constexpr unsigned kPParams = kPScratch + 2 * 4 * kAggRows * 4;  // block1.2 bias, block3.2 bias, alpha weights
// colour kernel shared memory
constexpr unsigned kCWeights = kATileBytes;                    // all of the branch's chunks, loaded once
constexpr unsigned kCBar = kCWeights + (unsigned)kColorBytes;
constexpr unsigned kCParams = kCBar + 256;                     // the 128->3 layer's weights
constexpr unsigned kAHead = kAggRows * 256;                    // columns 0..127 of the operand: two blocks

struct PairBars {
  uint64_t full[kStages];
  uint64_t empty[kStages];
  uint64_t acc_full[kTeams];  // MMA warp -> team: a layer completed into its accumulator
  uint64_t a_ready[kTeams];   // team -> MMA warp: the next layer's operand is written
  uint64_t w3b;               // W3b landed
  uint64_t idle;              // MMA warp: everything it issued has completed
  uint32_t tmem;
  int abort;
};

// The order in which the CTA's layers run on the tensor cores, walked alike by
// the load warp and the MMA warp: layer L of team 0's tile, of team 1's, then
// layer L + 1 (f returns false to stop).  A whole tile of one team at a time,
// or team 1 two layers behind, were within 2%.
template <class F>
__device__ __forceinline__ void each_layer(long long my_tiles, F&& f) {
  for (long long i = 0; i < my_tiles; i += kTeams) {
#pragma unroll 1
    for (int s = 0; s < 4 * kTeams; s++)
      if (i + s % kTeams < my_tiles && !f(s % kTeams, s / kTeams)) return;
  }
}

struct PairScratch {           // of one team
  float apart[4][kAggRows];    // alpha-branch partial dot products (column quarters)
};

struct ColorBars {
  uint64_t w[kColorChunks];  // weight chunk c landed
  uint64_t a;                // both parts of the input tile landed
  uint64_t done;             // all MMAs of a layer completed
  uint32_t tmem;
};

// Wait for a phase; gives up (and raises the CTA's abort flag) after limit_ns,
// or at once when another role raised it.
__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, unsigned parity, volatile int* abort,
                                              unsigned long long limit_ns) {
  if (tc::mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = tc::global_ns();
  for (;;) {
    if (tc::mbar_try_wait(bar, parity)) return true;
    if (*abort) return false;
    if (tc::global_ns() - t0 > limit_ns) {
      *abort = 1;
      return false;
    }
  }
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ uint4 pack8(const float* v) {
  return make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
}

// columns 8u .. 8u + 7 of row r of a pair operand
__device__ __forceinline__ void store_pair_unit(uint8_t* A, int r, int u, const float* v) {
  const uint32_t at = u < 32 ? tc::operand_offset(r, u * 8, kAggRows) : kTail + tc::sw64_offset(r, u * 8 - 256);
  *reinterpret_cast<uint4*>(A + at) = pack8(v);
}

// columns 8u .. 8u + 7 of row r of a 128-row swizzled operand
__device__ __forceinline__ void store_unit(uint8_t* A, int r, int u, const float* v) {
  *reinterpret_cast<uint4*>(A + tc::operand_offset(r, u * 8, kAggRows)) = pack8(v);
}

__device__ __forceinline__ void zero_unit(uint8_t* A, int r, int u) {
  *reinterpret_cast<uint4*>(A + tc::operand_offset(r, u * 8, kAggRows)) = make_uint4(0, 0, 0, 0);
}

__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
  const uint32_t a = tc::smem_addr(p);
  return p + (((a + 1023u) & ~1023u) - a);
}

// LeakyReLU(0.01): max(x, 0.01 x) is x for x >= 0 and 0.01 x below.
__device__ __forceinline__ float leaky(float x) { return fmaxf(x, __fmul_rn(x, 0.01f)); }

__device__ __forceinline__ float2 leaky2(float2 x) {
  const float2 y = tc::mul2(x, make_float2(0.01f, 0.01f));
  return make_float2(fmaxf(x.x, y.x), fmaxf(x.y, y.y));
}

__device__ __forceinline__ float softplus(float x) { return x > 20.0f ? x : log1pf(expf(x)); }

// sin / cos of x * 2^f, f < F: one __sincosf, then sin 2a = 2 sin a cos a, cos 2a = 1 - 2 sin^2 a.
template <int F>
__device__ __forceinline__ void bands(float x, float* s, float* c) {
  __sincosf(x, &s[0], &c[0]);
#pragma unroll
  for (int f = 1; f < F; f++) {
    s[f] = __fmul_rn(2.0f, __fmul_rn(s[f - 1], c[f - 1]));
    c[f] = __fmaf_rn(-2.0f * s[f - 1], s[f - 1], 1.0f);
  }
}

struct AggArgs {
  const uint8_t* packed;
  const float* pc_xyz;   // [M, P, 3]
  const float* pc_rgb;   // [M, P, 3]
  const float* pc_dir;   // [M, P, 3]
  const float* pc_feat;  // [M, P, 32]
  const float* sp_xyz;   // [M, 3]
  const uint8_t* valid;  // [M, P]
  const float* rays_d;   // [M, 3]
  long long M;
  int P;
  uint8_t* color_in;  // colour-branch input tiles (operand layout, K = 320)
  float* alpha;       // [M]
  float* color;       // [M, 3]
  int* status;
  unsigned long long wait_ns;  // limit of each wait of the pair kernel's roles (tc::kWaitNs)
  int withhold_w3b;            // a test of those waits: W3b is never loaded, so its wait gives up
};

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Layer-1 operand units U0 .. U1-1 of row r: columns 0..31 feat, 32..223 PE(feat, 3)
// (argument a = channel * 3 + band at columns 32 + 2a (sin), 33 + 2a (cos)), 224..283
// PE(dist_feat, 5), 284 the constant 1 (its weight column holds block1.0's bias),
// 285..287 zeros.  (Rows beyond the last sample are encoded like zeros: their weight is 0
// and no sample of theirs is written.)
template <int U0, int U1>
__device__ __forceinline__ void input_units(uint8_t* A, int r, const float* feat, const float* df) {
  float sf[3], cf[3], sd[5], cd[5];
  int chf = -1, chd = -1;
#pragma unroll
  for (int u = U0; u < U1; u++) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int col = 8 * u + i;
      float x = 0.0f;
      if (col < 32) {
        x = feat[col];
      } else if (col < 224) {
        const int a = (col - 32) >> 1, c = a / 3, f = a % 3;
        if (c != chf) {
          bands<3>(feat[c], sf, cf);
          chf = c;
        }
        x = ((col - 32) & 1) ? cf[f] : sf[f];
      } else if (col < 284) {
        const int a = (col - 224) >> 1, c = a / 5, f = a % 5;
        if (c != chd) {
          bands<5>(df[c], sd, cd);
          chd = c;
        }
        x = ((col - 224) & 1) ? cd[f] : sd[f];
      } else if (col == 284) {
        x = 1.0f;
      }
      v[i] = x;
    }
    store_pair_unit(A, r, u, v);
  }
}

// A team's view of one tile's inputs: builds A; returns the aggregation weight of the
// thread's row, and whether its point is valid.
__device__ __forceinline__ float build_inputs(const AggArgs& g, long long t, int spt, uint8_t* A, int tid,
                                              bool& valid) {
  const int P = g.P;
  const int r = tid & (kAggRows - 1), h = tid >> 7;  // h: which 18 of the row's 36 units
  const long long m = t * spt + r / P;
  const int p = r % P;
  const bool in = r < spt * P && m < g.M;
  const long long e = m * P + p;
  float feat[kFeatDim], df[6];
  float inv = 0.0f;
  valid = false;
#pragma unroll
  for (int i = 0; i < kFeatDim; i++) feat[i] = 0.0f;
#pragma unroll
  for (int i = 0; i < 6; i++) df[i] = 0.0f;
  if (in) {
    const float4* fp = reinterpret_cast<const float4*>(g.pc_feat + e * kFeatDim);
#pragma unroll
    for (int i = 0; i < kFeatDim / 4; i++) {
      const float4 q = __ldg(fp + i);
      feat[4 * i] = q.x, feat[4 * i + 1] = q.y, feat[4 * i + 2] = q.z, feat[4 * i + 3] = q.w;
    }
    float d2 = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const float x = __ldg(g.pc_xyz + e * 3 + i), s = __ldg(g.sp_xyz + m * 3 + i);
      df[i] = __fsub_rn(x, s);
      df[3 + i] = __fsub_rn(__fmul_rn(x, x), __fmul_rn(s, s));
      d2 = __fmaf_rn(df[i], df[i], d2);
    }
    valid = __ldg(g.valid + e) != 0;
    if (valid) inv = __fdiv_rn(1.0f, __fadd_rn(sqrtf(d2), 1e-6f));
  }
  // aggregation weight: inv / (sum over the sample's P rows + 1e-6); the rows are adjacent lanes
  float sum = inv;
  for (int o = 1; o < P; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (h == 0)
    input_units<0, 18>(A, r, feat, df);
  else
    input_units<18, 36>(A, r, feat, df);
  return __fdiv_rn(inv, __fadd_rn(sum, 1e-6f));
}

// Epilogue of a hidden layer: LeakyReLU(x + bias) -> bf16 into the next operand,
// over the one the layer has read.  A thread takes columns 64 kb + 32 g .. + 31 of
// its row er, kb = 0..3.  bias is null for the layers whose bias came in through
// the MMA.
__device__ __forceinline__ void epilogue_hidden(uint32_t acc_addr, const float* bias, uint8_t* A, int er, int g) {
#pragma unroll 1
  for (int kb = 0; kb < 4; kb++) {
    const int col0 = 64 * kb + 32 * g;
    float v[32];
    tc::tmem_ld32(acc_addr + (uint32_t)col0, v);
    if (bias) {
      const float4* b4 = reinterpret_cast<const float4*>(bias + col0);
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const float4 b = b4[q];
        const float2 lo = tc::add2(make_float2(v[4 * q], v[4 * q + 1]), make_float2(b.x, b.y));
        const float2 hi = tc::add2(make_float2(v[4 * q + 2], v[4 * q + 3]), make_float2(b.z, b.w));
        v[4 * q] = lo.x, v[4 * q + 1] = lo.y, v[4 * q + 2] = hi.x, v[4 * q + 3] = hi.y;
      }
    }
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      const float2 y = leaky2(make_float2(v[i], v[i + 1]));
      v[i] = y.x, v[i + 1] = y.y;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) store_unit(A, er, col0 / 8 + q, v + 8 * q);
  }
}

// The last epilogue's transpose buffer of a warp: 32 rows x 64 columns fp32, 16-byte
// piece c of row r at piece c ^ (r % 16).
constexpr int kRedBytes = 32 * 64 * 4;
__device__ __forceinline__ uint32_t red_offset(int r, int c) { return (uint32_t)(r * 256 + ((c ^ (r & 15)) << 4)); }

// Sums over each sample's P rows of a warp's transpose buffer, rows in order; lane l
// takes columns 2 l and 2 l + 1 and stores their bf16 pair, so a sample's 64 columns
// (col0 ..) are one 128-byte row of the colour-input tile.
template <int P>
__device__ __forceinline__ void sample_sums(const uint8_t* red, int lane, long long m0, long long M, uint8_t* color_in,
                                            int col0) {
  constexpr int G = 32 / P;
  constexpr int kAhead = P < 8 ? P : 8;  // rows loaded before they are added
// samples unrolled: their loads overlap (143,000 x 8, a forward: 685 us one by one, 671 so)
#pragma unroll 4
  for (int gs = 0; gs < G; gs++) {
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int p0 = 0; p0 < P; p0 += kAhead) {
      float2 v[kAhead];
#pragma unroll
      for (int p = 0; p < kAhead; p++)
        v[p] = *reinterpret_cast<const float2*>(red + red_offset(gs * P + p0 + p, lane >> 1) + (lane & 1) * 8);
#pragma unroll
      for (int p = 0; p < kAhead; p++) acc = p0 + p == 0 ? v[0] : tc::add2(acc, v[p]);
    }
    const long long m = m0 + gs;
    if (m < M)
      *reinterpret_cast<uint32_t*>(color_in + (size_t)(m / kAggRows) * kATileBytes +
                                   tc::operand_offset((int)(m % kAggRows), col0 + 2 * lane, kAggRows)) =
          pack2(acc.x, acc.y);
  }
}

// ---------------------------------------------------------------------------
// pair MLP: block1, block3, alpha branch, weighted reduction
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kPairThreads, 1) k_agg_pairs(AggArgs g, long long n_tiles) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* stages = smem + kPStages;
  uint8_t* W3b = smem + kPW3b;
  PairBars& bar = *reinterpret_cast<PairBars*>(smem + kPBar);
  volatile int* abort = &bar.abort;
  const float* prm = reinterpret_cast<const float*>(g.packed + kParamOff);
  float* s_b2 = reinterpret_cast<float*>(smem + kPParams);  // read from shared memory: from L2 each epilogue waited
  float* s_b4 = s_b2 + kPairN;                              // for them (the operands leave next to no L1)
  float* s_wa = s_b4 + kPairN;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int P = g.P, spt = kAggRows / P;
  if (tid < kPairN) {
    s_b2[tid] = prm[kPB2 + tid];
    s_b4[tid] = prm[kPB4 + tid];
    s_wa[tid] = prm[kPWA + tid];
  }

  if (tid == 0) {
    for (int i = 0; i < kStages; i++) {
      tc::mbar_init(&bar.full[i], 1);
      tc::mbar_init(&bar.empty[i], 1);
    }
    for (int i = 0; i < kTeams; i++) {
      tc::mbar_init(&bar.acc_full[i], 1);
      tc::mbar_init(&bar.a_ready[i], kTeamThreads);
    }
    tc::mbar_init(&bar.w3b, 1);
    tc::mbar_init(&bar.idle, 1);
    bar.abort = 0;
    tc::mbar_init_fence();
  }
  if (warp == 0) tc::tmem_alloc(&bar.tmem, 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = bar.tmem;
  // the CTA's tiles blockIdx.x + i * gridDim.x; team i % 2 serves tile i
  const long long my_tiles = blockIdx.x < n_tiles ? (n_tiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  bool fail = false;
  // a converged warp's wait: the same answer in every lane, also when one of them gives up
  auto wait_warp = [&](uint64_t* b, unsigned parity) -> bool {
    if (__all_sync(0xffffffffu, tc::mbar_try_wait(b, parity))) return true;
    return __all_sync(0xffffffffu, wait_or_abort(b, parity, abort, g.wait_ns));
  };

  if (warp == kLoadWarp) {
    // ---- weight loads: W3b once, then each layer's chunks for one team's tile and again for the other's.
    // A whole warp like the MMA issue: a stage is free for one chunk's MMAs only, so the time from its
    // commit to the copy counts.
    if (!g.withhold_w3b) tc::warp_bulk_load(W3b, g.packed + kW3bOff, kW3bBytes, &bar.w3b);
    uint32_t q = 0;
    each_layer(my_tiles, [&](int, int L) -> bool {
      const uint8_t* src = g.packed + (size_t)pair_chunk0(L) * kChunkBytes;
#pragma unroll
      for (int kc = 0; kc < pair_chunks(L); kc++, q++) {
        const uint32_t st = q % kStages;
        if (q >= kStages && !wait_warp(&bar.empty[st], ((q / kStages) - 1) & 1)) return false;
        tc::warp_bulk_load(stages + (size_t)st * kChunkBytes, src + (size_t)kc * kChunkBytes, kChunkBytes,
                           &bar.full[st]);
      }
      return true;
    });
    // the last copy into each stage has landed before the CTA ends
    for (uint32_t d = q > kStages ? q - kStages : 0; d < q; d++)
      if (!tc::mbar_wait(&bar.full[d % kStages], (d / kStages) & 1)) fail = true;
    if (!g.withhold_w3b && !tc::mbar_wait(&bar.w3b, 0)) fail = true;
    __syncwarp();
  } else if (warp == kMmaWarp) {
    // ---- MMA issue: layer L of team 0's tile, of team 1's, then layer L + 1.  The whole warp runs the
    // loop, so that descriptors and barrier phases are warp-uniform, and issues by elect.sync.  (A chunk of
    // two 128-cycle MMAs took 590 cycles with one lane running the loop, 410 with the warp running it and
    // lane 0 issuing in a branch.)
    const uint32_t idesc = tc::idesc_bf16(kAggRows, kPairN);
    const uint64_t w3b_desc = tc::smem_desc_plain(tc::smem_addr(W3b), 128u, 256u);
    const uint64_t b_base = tc::smem_desc_sw64(tc::smem_addr(stages));
    unsigned a_ph = 0;  // bit team: phase of its operand
    uint32_t q = 0;     // weight chunks consumed
    bool ok = wait_warp(&bar.w3b, 0);
    // a chunk of K: two K = 16 steps of the operand at `a`
    auto chunk = [&](uint32_t acc, uint64_t a, bool first) -> bool {
      const uint32_t st = q % kStages;
      if (!wait_warp(&bar.full[st], (q / kStages) & 1)) return false;
      tc::warp_mma2_commit(acc, a, b_base + st * (kChunkBytes >> 4), idesc, first ? 0u : 1u, &bar.empty[st]);
      q++;
      return true;
    };
    if (ok) {
      each_layer(my_tiles, [&](int team, int L) -> bool {
        if (!(ok = wait_warp(&bar.a_ready[team], (a_ph >> team) & 1))) return false;
        a_ph ^= 1u << team;
        tc::tc_fence_after();
        const uint32_t acc = tmem + (uint32_t)team * 256u;
        const uint32_t a_addr = tc::smem_addr(smem + kPA + team * kABytes);
        const uint64_t a_base = tc::smem_desc_sw128(a_addr), a_tail = tc::smem_desc_sw64(a_addr + kTail);
#pragma unroll
        for (int kc = 0; kc < 256 / kPairChunkK && ok; kc++)
          ok = chunk(acc, a_base + (uint32_t)((kc >> 1) * (kAggRows * 128 / 16) + (kc & 1) * 4), kc == 0);
        if (ok && L == 0) ok = chunk(acc, a_tail, false);
        if (ok && L == 2)  // block3.0's extra inputs (columns 256..271) times W3b
          tc::warp_mma_bf16(acc, a_tail, w3b_desc, idesc, 1u);
        tc::warp_commit(&bar.acc_full[team]);
        return ok;
      });
    }
    if (!ok) fail = true;
    tc::warp_commit(&bar.idle);
    if (!tc::mbar_wait(&bar.idle, 0)) fail = true;
    __syncwarp();
  } else {
    // ---- a team: inputs, epilogues, reductions of its tiles
    const int team = warp >> 3, ttid = tid & (kTeamThreads - 1);
    const int er = 32 * (warp & 3) + lane, cq = (warp >> 2) & 1;  // row, column group
    uint8_t* A = smem + kPA + team * kABytes;
    PairScratch& sc = reinterpret_cast<PairScratch*>(smem + kPScratch)[team];
    const uint32_t acc = tmem + (uint32_t)team * 256u + ((uint32_t)(32 * (warp & 3)) << 16);
    unsigned acc_ph = 0;
    const float ba = __ldg(prm + kPBA);
    int stop = 0;
    auto ready = [&] {  // the operand is written and the accumulator read
      tc::tc_fence_before();
      tc::fence_async_smem();
      tc::mbar_arrive(&bar.a_ready[team]);
    };
    auto layer = [&] {  // the layer is in the accumulator
      if (!wait_or_abort(&bar.acc_full[team], (acc_ph++) & 1, abort, g.wait_ns)) fail = true;
      tc::tc_fence_after();
    };
    for (long long i = team; i < my_tiles && !stop; i += kTeams) {
      const long long t = blockIdx.x + i * gridDim.x;
      bool valid;
      const float w = build_inputs(g, t, spt, A, ttid, valid);  // of row er, which is the row the thread built
      ready();
      // layer 1 (its bias: column 284 of the inputs)
      layer();
      epilogue_hidden(acc, nullptr, A, er, cq);
      ready();
      // layer 2, and block3's extra inputs
      float ex[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (cq == 1) {
        const long long m = t * spt + er / P;
        const long long e = m * P + er % P;
        if (er < spt * P && m < g.M) {
          float dot = 0.0f, ray[3];
#pragma unroll
          for (int c = 0; c < 3; c++) {
            const float dv = __ldg(g.pc_dir + e * 3 + c), rd = __ldg(g.rays_d + m * 3 + c);
            ray[c] = rd;
            ex[c] = __ldg(g.pc_rgb + e * 3 + c);
            ex[3 + c] = __fsub_rn(dv, rd);
            dot = c == 0 ? __fmul_rn(dv, rd) : __fmaf_rn(dv, rd, dot);
          }
          ex[6] = dot;
          ex[7] = 1.0f;  // its W3b column holds block3.0's bias
          // The colour row's ray columns, PE(ray_d, 4) -> 256..279 and zeros to 319: here, while layer 2 runs.
          // At the tile's end they waited for the ray again, and the alphas below for the valid flags: 710 us
          // a forward of 143,000 x 8, 685 so.
          if (er % P == 0) {
            uint8_t* crow = g.color_in + (size_t)(m / kAggRows) * kATileBytes;
            const int cr = (int)(m % kAggRows);
            float s4[3][4], c4[3][4];
#pragma unroll
            for (int c = 0; c < 3; c++) bands<4>(ray[c], s4[c], c4[c]);
#pragma unroll
            for (int u = 0; u < 3; u++) {
              float v[8];
#pragma unroll
              for (int c = 0; c < 4; c++) {
                const int a = 4 * u + c;
                v[2 * c] = s4[a / 4][a % 4];
                v[2 * c + 1] = c4[a / 4][a % 4];
              }
              store_unit(crow, cr, 32 + u, v);
            }
#pragma unroll
            for (int u = 35; u < 40; u++) zero_unit(crow, cr, u);
          }
        }
      }
      layer();
      if (cq == 1) {
        store_pair_unit(A, er, 32, ex);
        *reinterpret_cast<uint4*>(A + kTail + tc::sw64_offset(er, 8)) = make_uint4(0, 0, 0, 0);
      }
      epilogue_hidden(acc, s_b2, A, er, cq);
      ready();
      // layer 3 (its bias: column 7 of the extra inputs)
      layer();
      epilogue_hidden(acc, nullptr, A, er, cq);
      ready();
      if (i + kTeams < my_tiles) {  // the next tile's inputs on their way to L2
        const long long e = ((t + (long long)kTeams * gridDim.x) * spt) * P + (ttid & (kAggRows - 1));
        if (e < g.M * P) {
          if (ttid < kAggRows)
            prefetch_l2(g.pc_feat + e * kFeatDim);
          else if ((ttid & 7) == 0)
            prefetch_l2(g.pc_xyz + e * 3);
        }
      }
      // layer 4: alpha-branch dot product per row, and the weighted sum over each sample's
      // rows: the warp's 32 rows x 64 columns go through a transpose buffer (in A, whose
      // last reader, layer 4, has completed), and lane l sums columns 2 l and 2 l + 1 of
      // each sample and writes them to its colour-input row (sample_sums).
      layer();
      {
        const float2 w2 = make_float2(w, w);
        uint8_t* red = A + (warp & 7) * kRedBytes;
        const long long m0 = (t * kAggRows + 32 * (warp & 3)) / P;  // the warp's first sample
#pragma unroll 1
        for (int cc = 0; cc < 2; cc++) {
          const int col0 = 128 * cq + 64 * cc;
          float adot = 0.0f;
#pragma unroll
          for (int half = 0; half < 2; half++) {
            float v[32];
            tc::tmem_ld32(acc + (uint32_t)(col0 + 32 * half), v);
#pragma unroll
            for (int q = 0; q < 8; q++) {
              const float4 b = reinterpret_cast<const float4*>(s_b4 + col0 + 32 * half)[q];
              const float4 a = reinterpret_cast<const float4*>(s_wa + col0 + 32 * half)[q];
              const float2 f0 = leaky2(tc::add2(make_float2(v[4 * q], v[4 * q + 1]), make_float2(b.x, b.y)));
              const float2 f1 = leaky2(tc::add2(make_float2(v[4 * q + 2], v[4 * q + 3]), make_float2(b.z, b.w)));
              adot = __fmaf_rn(f0.x, a.x, adot);
              adot = __fmaf_rn(f0.y, a.y, adot);
              adot = __fmaf_rn(f1.x, a.z, adot);
              adot = __fmaf_rn(f1.y, a.w, adot);
              const float2 x0 = tc::mul2(f0, w2), x1 = tc::mul2(f1, w2);
              *reinterpret_cast<float4*>(red + red_offset(lane, 8 * half + q)) = make_float4(x0.x, x0.y, x1.x, x1.y);
            }
          }
          sc.apart[2 * cq + cc][er] = adot;
          __syncwarp();
          switch (P) {
            case 1: sample_sums<1>(red, lane, m0, g.M, g.color_in, col0); break;
            case 2: sample_sums<2>(red, lane, m0, g.M, g.color_in, col0); break;
            case 4: sample_sums<4>(red, lane, m0, g.M, g.color_in, col0); break;
            case 8: sample_sums<8>(red, lane, m0, g.M, g.color_in, col0); break;
            case 16: sample_sums<16>(red, lane, m0, g.M, g.color_in, col0); break;
            default: sample_sums<32>(red, lane, m0, g.M, g.color_in, col0); break;
          }
          __syncwarp();
        }
      }
      tc::tc_fence_before();
      stop = tc::named_sync_or(fail || *abort, 1 + team, kTeamThreads);
      if (stop) break;
      // alpha: softplus(branch - 1) of each valid row, weighted sum over the sample
      if (ttid < kAggRows) {
        const int r = ttid;
        const long long m = t * spt + r / P;
        const int p = r % P;
        const bool in = r < spt * P && m < g.M;
        float a = 0.0f;
        if (valid) {
          const float z = __fadd_rn(__fadd_rn(__fadd_rn(sc.apart[0][r], sc.apart[1][r]),
                                              __fadd_rn(sc.apart[2][r], sc.apart[3][r])), ba);
          a = softplus(__fsub_rn(z, 1.0f));
        }
        float x = __fmul_rn(a, w);
        for (int o = 1; o < P; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (in && p == 0) g.alpha[m] = x;
      }
      // apart is rewritten next tile
      if (i + kTeams < my_tiles) stop = tc::named_sync_or(fail || *abort, 1 + team, kTeamThreads);
    }
  }

  if (fail) atomicExch(g.status, 1);
  if (tid == 0 && bar.abort) atomicExch(g.status, 1);
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, 512);
  }
}

// ---------------------------------------------------------------------------
// colour branch
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kColorThreads, 1) k_agg_color(AggArgs g, long long n_tiles) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* A = smem;
  ColorBars& bar = *reinterpret_cast<ColorBars*>(smem + kCBar);
  float* s_wc = reinterpret_cast<float*>(smem + kCParams);
  const float* prm = reinterpret_cast<const float*>(g.packed + kParamOff);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < 3 * kColorN) s_wc[tid] = prm[kPWC4 + tid];

  if (tid == 0) {
    for (int c = 0; c < kColorChunks; c++) tc::mbar_init(&bar.w[c], 1);
    tc::mbar_init(&bar.a, 2);  // the tile's two parts
    tc::mbar_init(&bar.done, 1);
    tc::mbar_init_fence();
  }
  if (warp == 0) tc::tmem_alloc(&bar.tmem, 128);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = bar.tmem;
  // warp 0 loads and issues: a tile's columns 0..127 (the hidden layers' operand too) and the rest apart
  long long a_parts = 0, a_done = 0;  // loads issued (two a tile), tiles waited for
  auto load_head = [&](long long t) {
    tc::warp_bulk_load(A, g.color_in + (size_t)t * kATileBytes, kAHead, &bar.a);
    a_parts++;
  };
  auto load_rest = [&](long long t) {
    tc::warp_bulk_load(A + kAHead, g.color_in + (size_t)t * kATileBytes + kAHead, kATileBytes - kAHead, &bar.a);
    a_parts++;
  };
  if (warp == 0 && blockIdx.x < n_tiles) {
    load_head(blockIdx.x);
    load_rest(blockIdx.x);
    for (int c = 0; c < kColorChunks; c++)
      tc::warp_bulk_load(smem + kCWeights + c * kChunkBytes, g.packed + kColorOff + (size_t)c * kChunkBytes,
                         kChunkBytes, &bar.w[c]);
  }
  auto wait_warp = [&](uint64_t* b, unsigned parity) -> bool {
    return __all_sync(0xffffffffu, tc::mbar_wait(b, parity));
  };
  const uint32_t idesc = tc::idesc_bf16(kAggRows, kColorN);
  const uint64_t a_base = tc::smem_desc_sw128(tc::smem_addr(A));
  const uint64_t w_base = tc::smem_desc_sw128(tc::smem_addr(smem + kCWeights));
  const int er = 32 * (warp & 3) + lane, cq = warp >> 2;  // row, column quarter
  const uint32_t lane_addr = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
  // the last layer's partial sums, in the operand (its last reader, that layer, has completed)
  float(*opart)[kAggRows][4] = reinterpret_cast<float(*)[kAggRows][4]>(A);
  unsigned done_phase = 0;
  bool fail = false;
  int stop = 0;

  for (long long t = blockIdx.x; t < n_tiles && !stop; t += gridDim.x) {
    const bool more = t + gridDim.x < n_tiles;
    int chunk0 = 0;
#pragma unroll
    for (int L = 0; L < 3; L++) {
      const int chunks = color_k(L) / kChunkK;
      if (warp == 0) {
        bool ok = true;
        if (L == 0) {
          ok = wait_warp(&bar.a, (unsigned)a_done & 1);
          a_done += ok;
        }
        tc::tc_fence_after();
        for (int c = 0; c < chunks && ok; c++) {
          if (t == blockIdx.x) ok = wait_warp(&bar.w[chunk0 + c], 0);
          if (!ok) break;
          // of the last input chunk (columns 256..319) the upper half is zeros on both sides
          const int steps = L == 0 && c == chunks - 1 ? kChunkK / 32 : kChunkK / 16;
          for (int j = 0; j < steps; j++)
            tc::warp_mma_bf16(tmem, a_base + (uint32_t)(c * (kAggRows * 128 / 16) + 2 * j),
                              w_base + (uint32_t)((chunk0 + c) * (kChunkBytes / 16) + 2 * j), idesc,
                              (c > 0 || j > 0) ? 1u : 0u);
        }
        if (!ok) fail = true;
        tc::warp_commit(&bar.done);  // also on failure, so the other warps' wait ends
      }
      chunk0 += chunks;
      // the biases on their way while the layer runs: of 32 columns, 64 in the last layer's warps
      const float4* bias = reinterpret_cast<const float4*>(prm + (L == 0 ? kPCB1 : L == 1 ? kPCB2 : kPCB3));
      constexpr int kLast = kColorN / 2 / 4;
      float4 b[kLast];
      if (L < 2) {
#pragma unroll
        for (int q = 0; q < 8; q++) b[q] = __ldg(bias + 8 * cq + q);
      } else if (cq < 2) {
#pragma unroll
        for (int q = 0; q < kLast; q++) b[q] = __ldg(bias + kLast * cq + q);
      }
      if (!tc::mbar_wait(&bar.done, done_phase & 1)) fail = true;
      done_phase++;
      tc::tc_fence_after();
      if (L == 0 && more && warp == 0 && !__any_sync(0xffffffffu, fail)) load_rest(t + gridDim.x);
      if (L < 2) {
        const int col0 = 32 * cq;
        float v[32];
        tc::tmem_ld32(lane_addr + (uint32_t)col0, v);
#pragma unroll
        for (int q = 0; q < 8; q++) {
          v[4 * q] = leaky(__fadd_rn(v[4 * q], b[q].x));
          v[4 * q + 1] = leaky(__fadd_rn(v[4 * q + 1], b[q].y));
          v[4 * q + 2] = leaky(__fadd_rn(v[4 * q + 2], b[q].z));
          v[4 * q + 3] = leaky(__fadd_rn(v[4 * q + 3], b[q].w));
        }
#pragma unroll
        for (int q = 0; q < 4; q++) store_unit(A, er, col0 / 8 + q, v + 8 * q);
      } else if (cq < 2) {
        float o[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int cc = 0; cc < 2; cc++) {
          const int col0 = 64 * cq + 32 * cc;
          float v[32];
          tc::tmem_ld32(lane_addr + (uint32_t)col0, v);
#pragma unroll
          for (int q = 0; q < 8; q++) {
            const float4 bq = b[8 * cc + q];
            const float f0 = leaky(__fadd_rn(v[4 * q], bq.x)), f1 = leaky(__fadd_rn(v[4 * q + 1], bq.y));
            const float f2 = leaky(__fadd_rn(v[4 * q + 2], bq.z)), f3 = leaky(__fadd_rn(v[4 * q + 3], bq.w));
#pragma unroll
            for (int j = 0; j < 3; j++) {
              const float4 w = *reinterpret_cast<const float4*>(s_wc + j * kColorN + col0 + 4 * q);
              o[j] = __fmaf_rn(f3, w.w, __fmaf_rn(f2, w.z, __fmaf_rn(f1, w.y, __fmaf_rn(f0, w.x, o[j]))));
            }
          }
        }
        *reinterpret_cast<float4*>(opart[cq][er]) = make_float4(o[0], o[1], o[2], 0.0f);
      }
      tc::tc_fence_before();
      tc::fence_async_smem();
      stop = __syncthreads_or(fail);
      if (stop) break;
    }
    if (stop) break;
    if (tid < kAggRows) {
      const long long m = t * kAggRows + tid;
      if (m < g.M) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
          const float z = __fadd_rn(__fadd_rn(opart[0][tid][j], opart[1][tid][j]), prm[kPCB4 + j]);
          const float s = 1.0f / (1.0f + expf(-z));
          g.color[m * 3 + j] = __fsub_rn(__fmul_rn(s, 1.002f), 0.001f);
        }
      }
    }
    __syncthreads();  // opart is read
    if (warp == 0 && more) load_head(t + gridDim.x);
  }

  if (warp == 0) {  // what was issued has completed before the CTA ends
    if (a_parts % 2 && lane == 0) tc::mbar_arrive(&bar.a);  // gave up between a tile's two loads
    __syncwarp();
    if (a_parts > 2 * a_done && !tc::mbar_wait(&bar.a, (unsigned)a_done & 1)) fail = true;
    if (blockIdx.x < n_tiles)
      for (int c = 0; c < kColorChunks; c++)
        if (!tc::mbar_wait(&bar.w[c], 0)) fail = true;
    tc::warp_commit(&bar.done);
    if (!tc::mbar_wait(&bar.done, done_phase & 1)) fail = true;
  }
  if (fail) atomicExch(g.status, 1);
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, 128);
  }
}

// alpha / colour of sample offsets[i] at every set position i of mask_out, zeros elsewhere
__global__ void k_agg_scatter(const uint8_t* __restrict__ mask, const int* __restrict__ offsets, long long n,
                              long long M, const float* __restrict__ alpha, const float* __restrict__ color,
                              float* __restrict__ alpha_out, float* __restrict__ color_out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long m = offsets[i];
  const bool set = mask[i] != 0 && m < M;
  alpha_out[i] = set ? alpha[m] : 0.0f;
#pragma unroll
  for (int j = 0; j < 3; j++) color_out[i * 3 + j] = set ? color[m * 3 + j] : 0.0f;
}

// ---------------------------------------------------------------------------
// weight packing: fp32 nn.Linear weights -> bf16 chunks in operand layout
// ---------------------------------------------------------------------------
struct PackArgs {
  const float* w[9];
  const float* b[9];
};

// element e of the colour chunk stream -> (chunk, n, k within the chunk); a chunk is
// 128 rows x 64 K, 128-byte swizzled (tc::operand_offset with one K block)
__device__ __forceinline__ void chunk_coords(long long e, int& chunk, int& n, int& k) {
  const int per = kChunkN * kChunkK;
  chunk = (int)(e / per);
  const int o = (int)(e % per) * 2;  // byte offset in the chunk
  n = o >> 7;
  const int c = ((o >> 4) & 7) ^ (n & 7);
  k = c * 8 + ((o & 15) >> 1);
}

__global__ void k_agg_pack(PackArgs a, uint8_t* __restrict__ packed) {
  const long long n_pair = (long long)kPairBytes / 2, n_w3b = kW3bBytes / 2, n_color = (long long)kColorBytes / 2;
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(packed);
  if (e < n_pair) {  // pair chunk: 256 rows x 32 K, 64-byte swizzled (tc::sw64_offset)
    const int chunk = (int)(e / (kPairN * kPairChunkK));
    const int o = (int)(e % (kPairN * kPairChunkK)) * 2;
    const int row = o >> 6, k = ((((o >> 4) & 3) ^ ((row >> 1) & 3)) << 3) + ((o & 15) >> 1);
    int L = 0, c0 = 0;
    while (chunk >= c0 + pair_k(L) / kPairChunkK) c0 += pair_k(L++) / kPairChunkK;
    const int col = (chunk - c0) * kPairChunkK + k;
    const int streamed = L == 2 ? 256 : pair_real_k(L);  // block3.0's columns 256.. go to W3b
    float w = col < streamed ? a.w[L][(size_t)row * pair_real_k(L) + col] : 0.0f;
    if (L == 0 && col == 284) w = a.b[0][row];  // block1.0's bias, against the constant input column
    out[e] = __float2bfloat16_rn(w);
  } else if (e < n_pair + n_w3b) {
    const int o = (int)(e - n_pair) * 2;  // W3b: 256 rows x 16 K, no swizzle (tc::plain16_offset)
    const int row = (o / 256) * 8 + (o % 128) / 16, col = ((o % 256) / 128) * 8 + (o % 16) / 2;
    out[e] = __float2bfloat16_rn(col < 7 ? a.w[2][(size_t)row * 263 + 256 + col] : col == 7 ? a.b[2][row] : 0.0f);
  } else if (e < n_pair + n_w3b + n_color) {
    int chunk, n, k;
    chunk_coords(e - n_pair - n_w3b, chunk, n, k);
    int L = 0, c0 = 0;
    while (chunk >= c0 + color_k(L) / kChunkK) c0 += color_k(L++) / kChunkK;
    const int col = (chunk - c0) * kChunkK + k;
    out[e] = __float2bfloat16_rn(col < color_real_k(L) ? a.w[5 + L][(size_t)n * color_real_k(L) + col] : 0.0f);
  } else if (e < n_pair + n_w3b + n_color + kParams) {
    const int q = (int)(e - n_pair - n_w3b - n_color);
    float* prm = reinterpret_cast<float*>(packed + kParamOff);
    float v = 0.0f;
    if (q < kPWA) v = a.b[q / 256][q % 256];
    else if (q < kPBA) v = a.w[4][q - kPWA];
    else if (q < kPCB1) v = q == kPBA ? a.b[4][0] : 0.0f;
    else if (q < kPWC4) v = a.b[5 + (q - kPCB1) / 128][(q - kPCB1) % 128];
    else if (q < kPCB4) v = a.w[8][q - kPWC4];
    else v = q < kPCB4 + 3 ? a.b[8][q - kPCB4] : 0.0f;
    prm[q] = v;
  }
}

// The two tensor-core kernels exceed the 48 KB default of dynamic shared
// memory: opt them in once per device, and note the device's SM count.
static int32_t agg_setup(unsigned pair_smem, unsigned color_smem, int* sms) {
  static std::mutex mu;
  static int sm_counts[128] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 128)
    return set_error(HP_ERR_CUDA, "hp_aggregator_forward: cudaGetDevice failed");
  std::lock_guard<std::mutex> lock(mu);
  if (!sm_counts[dev]) {
    int n = 0;
    cudaError_t e = cudaFuncSetAttribute(k_agg_pairs, cudaFuncAttributeMaxDynamicSharedMemorySize, pair_smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_agg_color, cudaFuncAttributeMaxDynamicSharedMemorySize, color_smem);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess || n <= 0)
      return set_error(HP_ERR_CUDA, "hp_aggregator_forward: kernel set-up: %s", cudaGetErrorString(e));
    sm_counts[dev] = n;
  }
  *sms = sm_counts[dev];
  return HP_OK;
}

}  // namespace hp

using namespace hp;

namespace {
constexpr size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

struct AggLayout {
  size_t color_in, alpha, color, status, total;
};

AggLayout agg_layout(long long M) {
  AggLayout L;
  const long long tiles = (M + kAggRows - 1) / kAggRows;
  size_t o = 0;
  L.color_in = o;
  o += align256((size_t)(tiles > 0 ? tiles : 1) * kATileBytes);
  L.alpha = o;
  o += align256(sizeof(float) * (size_t)(M > 0 ? M : 1));
  L.color = o;
  o += align256(sizeof(float) * 3 * (size_t)(M > 0 ? M : 1));
  L.status = o;
  o += 256;
  L.total = o;
  return L;
}

constexpr unsigned kPairSmem = kPParams + 3 * kPairN * 4 + 1024;
static_assert(kTeams * sizeof(PairScratch) == kPParams - kPScratch, "scratch");
constexpr unsigned kColorSmem = kCParams + 3 * kColorN * 4 + 1024;
static_assert(sizeof(PairBars) <= 256 && sizeof(ColorBars) <= 256, "barrier block");
static_assert(kPairSmem <= 227 * 1024 && kColorSmem <= 227 * 1024, "shared memory");
static_assert(kTeamThreads / 32 * kRedBytes <= kABytes && kABytes % 1024 == 0, "transpose buffers fit in A");
}  // namespace

extern "C" size_t hp_aggregator_packed_size(void) { return kPackedBytes; }

extern "C" int32_t hp_aggregator_pack(const hp_aggregator_weights* w, void* packed, size_t packed_bytes,
                                      hp_stream_t stream) {
  if (!w || !packed) return set_error(HP_ERR_INVALID_ARGUMENT, "hp_aggregator_pack: null pointer");
  if (packed_bytes < kPackedBytes || ((uintptr_t)packed & 255) != 0)
    return set_error(HP_ERR_WORKSPACE, "hp_aggregator_pack: needs %zu bytes, 256-byte aligned", kPackedBytes);
  PackArgs a;
  for (int i = 0; i < 9; i++) {
    if (!w->weight[i] || !w->bias[i]) return set_error(HP_ERR_INVALID_ARGUMENT, "hp_aggregator_pack: layer %d", i);
    a.w[i] = w->weight[i];
    a.b[i] = w->bias[i];
  }
  const long long n = (long long)(kPairBytes + kW3bBytes + kColorBytes) / 2 + kParams;
  k_agg_pack<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(a, (uint8_t*)packed);
  return check_launch("k_agg_pack");
}

extern "C" size_t hp_aggregator_workspace_size(int64_t n_samples) {
  if (n_samples < 0) return 0;
  return agg_layout(n_samples).total;
}

static int32_t agg_forward(const void* packed, const float* pc_xyz, const float* pc_rgb, const float* pc_dir,
                           const float* pc_feat, int32_t feat_dim, const float* sp_xyz, const uint8_t* valid,
                           const float* rays_d, int64_t n_samples, int32_t P, const uint8_t* mask_out,
                           const int32_t* mask_offsets, int64_t n_positions, float* alpha_out, float* color_out,
                           void* workspace, size_t workspace_bytes, hp_stream_t stream, unsigned long long wait_ns,
                           int withhold_w3b) {
  static const char* who = "hp_aggregator_forward";
  if (feat_dim != kFeatDim)
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: feature width %d (the layers take %d)", who, feat_dim, kFeatDim);
  if (P < 1 || P > 32 || (P & (P - 1)) != 0)
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: points per sample %d (1, 2, 4, ..., 32 supported)", who, P);
  if (n_samples < 0 || n_samples * P >= (1ll << 40) || n_positions < 0 || n_positions >= (1ll << 31))
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: sizes out of range", who);
  if (!packed || !workspace || (n_positions > 0 && (!mask_out || !mask_offsets || !alpha_out || !color_out)) ||
      (n_samples > 0 && (!pc_xyz || !pc_rgb || !pc_dir || !pc_feat || !sp_xyz || !valid || !rays_d)))
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: null pointer", who);
  if (((uintptr_t)pc_feat & 15) != 0 || ((uintptr_t)packed & 255) != 0)
    return set_error(HP_ERR_INVALID_ARGUMENT, "%s: pc_feat must be 16-byte and packed 256-byte aligned", who);
  const AggLayout L = agg_layout(n_samples);
  if (workspace_bytes < L.total || ((uintptr_t)workspace & 255) != 0)
    return set_error(HP_ERR_WORKSPACE, "%s: workspace needs %zu bytes, 256-byte aligned", who, L.total);
  cudaStream_t st = (cudaStream_t)stream;
  char* ws = (char*)workspace;
  AggArgs g;
  g.packed = (const uint8_t*)packed;
  g.pc_xyz = pc_xyz;
  g.pc_rgb = pc_rgb;
  g.pc_dir = pc_dir;
  g.pc_feat = pc_feat;
  g.sp_xyz = sp_xyz;
  g.valid = valid;
  g.rays_d = rays_d;
  g.M = n_samples;
  g.P = P;
  g.color_in = (uint8_t*)(ws + L.color_in);
  g.alpha = (float*)(ws + L.alpha);
  g.color = (float*)(ws + L.color);
  g.status = (int*)(ws + L.status);
  g.wait_ns = wait_ns;
  g.withhold_w3b = withhold_w3b;
  if (cudaMemsetAsync(g.status, 0, sizeof(int), st) != cudaSuccess)
    return set_error(HP_ERR_CUDA, "%s: memset failed", who);
  if (n_samples > 0) {
    int sms = 0;
    if (int32_t rc = agg_setup(kPairSmem, kColorSmem, &sms)) return rc;
    const int spt = kAggRows / P;
    const long long pair_tiles = (n_samples + spt - 1) / spt;
    const long long color_tiles = (n_samples + kAggRows - 1) / kAggRows;
    const unsigned pg = (unsigned)(pair_tiles < sms ? pair_tiles : sms);
    const unsigned cg = (unsigned)(color_tiles < sms ? color_tiles : sms);
    k_agg_pairs<<<pg, kPairThreads, kPairSmem, st>>>(g, pair_tiles);
    if (int32_t rc = check_launch("k_agg_pairs")) return rc;
    k_agg_color<<<cg, kColorThreads, kColorSmem, st>>>(g, color_tiles);
    if (int32_t rc = check_launch("k_agg_color")) return rc;
  }
  if (n_positions > 0) {
    k_agg_scatter<<<(unsigned)((n_positions + 255) / 256), 256, 0, st>>>(mask_out, mask_offsets, n_positions,
                                                                         n_samples, g.alpha, g.color, alpha_out,
                                                                         color_out);
    if (int32_t rc = check_launch("k_agg_scatter")) return rc;
  }
  return HP_OK;
}

extern "C" int32_t hp_aggregator_forward(const void* packed, const float* pc_xyz, const float* pc_rgb,
                                         const float* pc_dir, const float* pc_feat, int32_t feat_dim,
                                         const float* sp_xyz, const uint8_t* valid, const float* rays_d,
                                         int64_t n_samples, int32_t P, const uint8_t* mask_out,
                                         const int32_t* mask_offsets, int64_t n_positions, float* alpha_out,
                                         float* color_out, void* workspace, size_t workspace_bytes,
                                         hp_stream_t stream) {
  return agg_forward(packed, pc_xyz, pc_rgb, pc_dir, pc_feat, feat_dim, sp_xyz, valid, rays_d, n_samples, P, mask_out,
                     mask_offsets, n_positions, alpha_out, color_out, workspace, workspace_bytes, stream, tc::kWaitNs,
                     0);
}

#ifdef HP_TESTING
// Test library only (include/hashpoint_b200_testing.h): the forward with the
// pair kernel's W3b block never loaded, so the tensor-core warp's bounded wait
// for it gives up after wait_limit_us, every other role's wait ends at once,
// the kernels return and hp_aggregator_status reports the failure.
extern "C" int32_t hp_aggregator_forward_withheld(const void* packed, const float* pc_xyz, const float* pc_rgb,
                                                  const float* pc_dir, const float* pc_feat, int32_t feat_dim,
                                                  const float* sp_xyz, const uint8_t* valid, const float* rays_d,
                                                  int64_t n_samples, int32_t P, const uint8_t* mask_out,
                                                  const int32_t* mask_offsets, int64_t n_positions, float* alpha_out,
                                                  float* color_out, void* workspace, size_t workspace_bytes,
                                                  int32_t wait_limit_us, hp_stream_t stream) {
  if (wait_limit_us <= 0)
    return set_error(HP_ERR_INVALID_ARGUMENT, "hp_aggregator_forward_withheld: wait_limit_us must be > 0");
  return agg_forward(packed, pc_xyz, pc_rgb, pc_dir, pc_feat, feat_dim, sp_xyz, valid, rays_d, n_samples, P, mask_out,
                     mask_offsets, n_positions, alpha_out, color_out, workspace, workspace_bytes, stream,
                     1000ull * (unsigned long long)wait_limit_us, 1);
}
#endif

extern "C" int32_t hp_aggregator_status(const void* workspace, int64_t n_samples, hp_stream_t stream) {
  if (!workspace || n_samples < 0) return set_error(HP_ERR_INVALID_ARGUMENT, "hp_aggregator_status: bad arguments");
  const AggLayout L = agg_layout(n_samples);
  int flag = 0;
  if (cudaMemcpyAsync(&flag, (const char*)workspace + L.status, sizeof(int), cudaMemcpyDeviceToHost,
                      (cudaStream_t)stream) != cudaSuccess ||
      cudaStreamSynchronize((cudaStream_t)stream) != cudaSuccess)
    return set_error(HP_ERR_CUDA, "hp_aggregator_status: %s", cudaGetErrorString(cudaGetLastError()));
  if (flag) return set_error(HP_ERR_CUDA, "hp_aggregator_forward: a tensor-core wait timed out");
  return HP_OK;
}
