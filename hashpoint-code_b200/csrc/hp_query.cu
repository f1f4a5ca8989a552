// Ray query for listed pixel rays, and the multi-bin z-buffer.
//
// hp_quick_query_for_nearby_point replaces _C.quick_query_for_nearby_point
// (epcq/csrc/epcq_render_topk.cu:287-339, kernel :222-283).  The reference
// gives each window cell a lane that gathers up to 32 ids within the ray
// radius and then reserves output slots with atomicAdd, so the order of a
// row -- and which ids survive when the row overflows -- depends on atomic
// timing.  Here a warp serves one ray at a time with its lanes over the
// candidates: 32 window cells at a time, their buckets concatenated, a
// candidate's place in the row from a ballot.  Rows are deterministic
// (window-cell order, bucket order) and an overflowing row keeps its first
// num_point_per_ray ids.
//
// hp_scatter replaces _C.scatter (epcq/csrc/rasterization.cu:88-128, kernel
// :36-86): per pixel the `bins` nearest points by depth, sorted ascending.
#include "hp_common.cuh"

namespace hp {

int32_t check_camera(const hp_camera* cam, const char* who);
DevCamera dev_camera(const hp_camera* cam);
DevOptions dev_options(const hp_options* o);

constexpr int kQueryWarps = 4;
#ifdef HP_TESTING
constexpr unsigned kWindowMax = 64;  // so that small tables take several rounds a window
#else
constexpr unsigned kWindowMax = 0x7fffffffu;
#endif
constexpr int kQueryRays = 8;  // rays a warp serves in turn in a long list, their directions computed side by side
constexpr int64_t kLongList = 1 << 17;  // rays from which it does

// Bound by the latency of the dependent loads (bucket, id, point) and the
// instructions of each ray's set-up; the rows themselves are 67 MB for 65,536
// rays of 256 (10 us).  A lane per cell left a warp waiting for its longest
// bucket, twice, with a division and a norm a candidate: 132 us for 65,536 rays
// of a 1M-point view at 800 x 800, 5 x 5 window (launch and flushed caches
// included), 60 us so.  A warp a ray fills the SMs from the shortest lists on
// (kRays = 1: 500 rays 29 us, with eight a warp 55; 5,000 rays 30 and 59; 65,536
// rays 60 and 65); from some 100,000 rays the shared set-up is worth more
// (300,000 rays: 203 us with one, 188 with eight).
template <int kRays>
__global__ void __launch_bounds__(kQueryWarps * 32) k_quick_query(const float* __restrict__ xyz, int n_points,
                                                                  const int* __restrict__ sidx, int n_sorted,
                                                                  const int2* __restrict__ hash, DevCamera cam,
                                                                  DevOptions opt, RadiusTest rt,
                                                                  const int* __restrict__ ray_ids, int n_rays,
                                                                  int* __restrict__ out) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int64_t r0 = ((int64_t)blockIdx.x * kQueryWarps + (threadIdx.x >> 5)) * kRays;
  if (r0 >= n_rays) return;
  const int cap = opt.num_point_per_ray, k = opt.k, k2 = k * k, W = cam.width, H = cam.height;
  int my_ray = -1;
  Ray mine{};
  if (lane < kRays && r0 + lane < n_rays) {
    my_ray = __ldg(ray_ids + r0 + lane);
    if (my_ray < 0 || my_ray >= W * H) my_ray = -1;
    if (my_ray >= 0) make_ray(cam.c2w, cam.fx, cam.fy, cam.cx, cam.cy, my_ray % W, my_ray / W, mine);
  }
  // clipped bucket of cell c0 + lane of a ray's window
  auto bucket = [&](int ray, int c0) -> int2 {
    const int l = c0 + lane;
    if (ray < 0 || l >= k2) return make_int2(0, 0);
    int vv, uu;
    window_cell(ray / W, ray % W, k, H, W, l, vv, uu);
    return bucket_range(__ldg(hash + (size_t)vv * W + uu), n_sorted);
  };
  const int rays = (int)(n_rays - r0 < kRays ? n_rays - r0 : kRays);
  int2 ahead = bucket(__shfl_sync(kAll, my_ray, 0), 0);
  for (int q = 0; q < rays; q++) {
    const int ray = __shfl_sync(kAll, my_ray, q);
    Ray r;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      r.o[i] = __shfl_sync(kAll, mine.o[i], q);
      r.d[i] = __shfl_sync(kAll, mine.d[i], q);
    }
    r.dd = __shfl_sync(kAll, mine.dd, q);
    const float inv_dd = __frcp_rn(r.dd);
    int2 rg = ahead;
    if (q + 1 < rays) ahead = bucket(__shfl_sync(kAll, my_ray, q + 1), 0);
    int* row = out + (r0 + q) * cap;
    int base = 0;
    for (int c0 = 0, cells = 32; c0 < k2 && base < cap && ray >= 0; c0 += cells) {
      if (c0 > 0) rg = bucket(ray, c0);
      // Candidates are numbered in 32 bits.  Clamped windows repeat buckets and tables may overlap, so 32 cells can
      // hold more than 2^31: then the round takes the cells before the one that reaches kWindowMax (at least one).
      unsigned cnt = (unsigned)(rg.y - rg.x), pre = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(kAll, pre, o);
        if (lane >= o) pre = min(pre + t, kWindowMax);  // both below 2^31
      }
      const unsigned beyond = __ballot_sync(kAll, pre >= kWindowMax);
      cells = beyond ? max(__ffs(beyond) - 1, 1) : 32;
      const unsigned total = __shfl_sync(kAll, pre, cells - 1);
      if (lane >= cells) cnt = 0, pre = total;
      pre -= cnt;
      const bool deep = __any_sync(kAll, cnt > kQueryPerCell);
      int carry = 0;  // lane c's copy: cell c's ids of earlier chunks
      for (unsigned j0 = 0; j0 < total && base < cap;) {
        const unsigned j = j0 + lane;
        int c = 0;
#pragma unroll
        for (int s = 16; s > 0; s >>= 1)
          if (__shfl_sync(kAll, pre, c + s) <= j) c += s;
        const unsigned first = __shfl_sync(kAll, pre, c);
        const int at = __shfl_sync(kAll, rg.x, c) + (int)(j - first);
        int id = -1;
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j < total) {
          id = __ldg(sidx + at);
          if ((unsigned)id < (unsigned)n_points) p = load_point(xyz, id);
          else id = -1;
        }
        const float t = ray_t(r, inv_dd, p);
        const float e0 = __fsub_rn(p.x, __fmaf_rn(t, r.d[0], r.o[0]));
        const float e1 = __fsub_rn(p.y, __fmaf_rn(t, r.d[1], r.o[1]));
        const float e2 = __fsub_rn(p.z, __fmaf_rn(t, r.d[2], r.o[2]));
        bool in = within_radius(rt, id >= 0, squared(e0, e1, e2), e0, e1, e2);
        unsigned m = __ballot_sync(kAll, in);
        if (deep) {  // only a cell's first kQueryPerCell
          const int before = __shfl_sync(kAll, carry, c) + __popc(m & below & ~lane_span(0, max((int)(first - j0), 0)));
          carry += __popc(m & lane_span(min(max((int)(pre - j0), 0), 32), min(max((int)(pre + cnt - j0), 0), 32)));
          in = in && before < kQueryPerCell;
          m = __ballot_sync(kAll, in);
        }
        const int pos = base + __popc(m & below);
        if (in && pos < cap) row[pos] = id;
        base += __popc(m);
        j0 += 32;
        if (deep) {  // the cell the chunk ended in has given its ids: on to the next one
          const int last = __shfl_sync(kAll, c, 31);
          if (__shfl_sync(kAll, carry, last) >= kQueryPerCell) j0 = max(j0, __shfl_sync(kAll, pre + cnt, last));
        }
      }
    }
    const int written = min(base, cap);
    if ((cap & 3) == 0 && ((uintptr_t)out & 15) == 0) {
      const int whole = (written + 3) & ~3;
      if (written + lane < whole) row[written + lane] = -1;
      for (int e = whole + 4 * lane; e < cap; e += 128) *reinterpret_cast<int4*>(row + e) = make_int4(-1, -1, -1, -1);
    } else {
      for (int e = written + lane; e < cap; e += 32) row[e] = -1;
    }
  }
}

// Per pixel: first index of its run by binary search over the sorted pixel
// ids (cuda_util.cuh:558-579), then the reference's buffer of the `bins`
// nearest depths, then a stable ascending sort (its bubble sort's result).
constexpr int kMaxBins = 64;

__global__ void __launch_bounds__(128) k_scatter_multibin(const int* __restrict__ point_idx,
                                                          const int* __restrict__ point2img,
                                                          const float* __restrict__ depth, int n, int hw, int bins,
                                                          float* __restrict__ out_depth, int* __restrict__ out_idx) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= hw) return;
  int lo = 0, hi = n;  // lower_bound of p
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (point2img[mid] < p)
      lo = mid + 1;
    else
      hi = mid;
  }
  float bd[kMaxBins];
  int bi[kMaxBins];
  int size = 0, maxi = -1;
  float maxz = -1000.0f;
  for (int j = lo; j < n && point2img[j] == p; j++) {
    const float d = depth[j];
    if (d < 0) continue;  // the reference spins forever here; the point is skipped instead
    if (size < bins) {
      bd[size] = d;
      bi[size] = point_idx[j];
      if (d > maxz) maxz = d, maxi = size;
      size++;
    } else if (d < maxz) {
      bd[maxi] = d;
      bi[maxi] = point_idx[j];
      maxz = d;
      for (int q = 0; q < bins; q++)
        if (bd[q] > maxz) maxz = bd[q], maxi = q;
    }
  }
  // stable insertion sort ascending by depth (same result as a stable bubble sort)
  for (int a = 1; a < size; a++) {
    const float kd = bd[a];
    const int ki = bi[a];
    int b = a - 1;
    while (b >= 0 && bd[b] > kd) {
      bd[b + 1] = bd[b];
      bi[b + 1] = bi[b];
      b--;
    }
    bd[b + 1] = kd;
    bi[b + 1] = ki;
  }
  float* od = out_depth + (size_t)p * bins;
  int* oi = out_idx + (size_t)p * bins;
  for (int q = 0; q < bins; q++) {
    od[q] = q < size ? bd[q] : -1.0f;
    oi[q] = q < size ? bi[q] : -1;
  }
}

}  // namespace hp

using namespace hp;

extern "C" int32_t hp_quick_query_for_nearby_point(const float* xyz, int64_t n_points, const hp_camera* cam,
                                                   const hp_options* opt, const int32_t* sorted_point_idx,
                                                   int64_t n_sorted, const int32_t* hash_table, const int32_t* ray_ids,
                                                   int64_t n_rays, int32_t* out, hp_stream_t stream) {
  if (int32_t rc = check_camera(cam, "hp_quick_query_for_nearby_point")) return rc;
  if (!opt) return set_error(HP_ERR_INVALID_ARGUMENT, "hp_quick_query_for_nearby_point: opt is NULL");
  // the reference rejects windows that need 1024 threads per block (epcq_render_topk.cu:321-323)
  if (opt->kernel_size < 1 || opt->kernel_size > 31)
    return set_error(HP_ERR_INVALID_ARGUMENT, "hp_quick_query_for_nearby_point: kernel_size %d outside 1..31",
                     opt->kernel_size);
  if (opt->num_point_per_ray < 0)
    return set_error(HP_ERR_INVALID_ARGUMENT, "hp_quick_query_for_nearby_point: num_point_per_ray < 0");
  if (n_rays < 0 || n_rays >= (1ll << 31) || n_points < 0 || n_points >= (1ll << 31) || n_sorted < 0 ||
      n_sorted >= (1ll << 31))
    return set_error(HP_ERR_INVALID_ARGUMENT, "hp_quick_query_for_nearby_point: bad sizes");
  if (n_rays == 0 || opt->num_point_per_ray == 0) return HP_OK;
  if (!hash_table || !ray_ids || !out || (n_points > 0 && !xyz) || (n_sorted > 0 && !sorted_point_idx))
    return set_error(HP_ERR_INVALID_ARGUMENT, "hp_quick_query_for_nearby_point: null pointer");
  if (((uintptr_t)hash_table & 7) != 0)
    return set_error(HP_ERR_INVALID_ARGUMENT, "hp_quick_query_for_nearby_point: hash_table must be 8-byte aligned");
  const bool one = n_rays < kLongList;
  const int64_t block = kQueryWarps * (one ? 1 : kQueryRays);
  (one ? k_quick_query<1> : k_quick_query<kQueryRays>)<<<(unsigned)((n_rays + block - 1) / block), kQueryWarps * 32, 0,
                                                        (cudaStream_t)stream>>>(
      xyz, (int)n_points, sorted_point_idx, (int)n_sorted, (const int2*)hash_table, dev_camera(cam), dev_options(opt),
      make_radius_test(opt->radius_threshold), ray_ids, (int)n_rays, out);
  return check_launch("k_quick_query");
}

extern "C" int32_t hp_scatter(const int32_t* point_idx, const int32_t* point2img, const float* depth, int64_t n,
                              int32_t height, int32_t width, int32_t bins, float* buffer_depth,
                              int32_t* buffer_point_index, hp_stream_t stream) {
  if (height <= 0 || width <= 0 || (int64_t)height * width >= (1ll << 31))
    return set_error(HP_ERR_INVALID_ARGUMENT, "hp_scatter: bad image size %dx%d", height, width);
  if (bins < 1 || bins > kMaxBins)
    return set_error(HP_ERR_INVALID_ARGUMENT, "hp_scatter: bins %d outside 1..%d", bins, kMaxBins);
  if (n < 0 || n >= (1ll << 31)) return set_error(HP_ERR_INVALID_ARGUMENT, "hp_scatter: n out of range");
  if (!buffer_depth || !buffer_point_index || (n > 0 && (!point_idx || !point2img || !depth)))
    return set_error(HP_ERR_INVALID_ARGUMENT, "hp_scatter: null pointer");
  const int hw = height * width;
  k_scatter_multibin<<<(hw + 127) / 128, 128, 0, (cudaStream_t)stream>>>(point_idx, point2img, depth, (int)n, hw,
                                                                          bins, buffer_depth, buffer_point_index);
  return check_launch("k_scatter_multibin");
}
