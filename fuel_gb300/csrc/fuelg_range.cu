// fuelg_range.cu -- range search of rows of up to 128 dimensions in register tiles
// (linear_scan_range, src/api/search.rs:154-166).
//
// One pass over all pairs (tile_dists: 64 queries x 128 index rows) counts each
// query's hits and writes their keys into the query's slots in whatever order
// they come; the keys are unique, so the sort by (distance, index) that the result
// needs anyway makes the order definite.  The counts' prefix sums are the result's
// offsets, and one warp (above 256 hits: one block) sorts a query's slots into its
// place.  Only when a query has more hits than slots, or there is no room for slots,
// does a second pass fill the lists at their offsets, for a segmented sort.
#include <algorithm>
#include <cub/device/device_scan.cuh>
#include <cub/device/device_segmented_sort.cuh>

#include "fuelg_common.cuh"
#include "fuelg_internal.h"
#include "fuelg_select.cuh"
#include "fuelg_tile.cuh"

namespace fuelg {
namespace {

constexpr int kRows = kTileQ * kTileMaxWarps;  // 64 queries of a block
constexpr int kRangeMaxD = 128;
constexpr int kMaxStrip = 8;                // most 128-row tiles that one CTA works through
constexpr int kTwoPerSm = 2 * 152;          // places on the chip with two CTAs per SM
constexpr int kTwoCtas = 112 * 1024;        // shared memory with which two CTAs fit an SM
// Most slots of a query: what range_long_kernel's block sorts in 34 KB of shared
// memory.  (With 1024 the 300-hit self-join had rows past them and took
// 4.29 ms for 1.74.)
constexpr int kSlots = 4096;
constexpr int kWarpSort = 256;              // most keys that a warp sorts
constexpr size_t kSlotBytes = 1u << 30;     // all queries' slots together

struct RangeTileArgs {
  const float* A;  // queries [m, d]
  int64_t m;
  const float* B;  // points [n, d]
  int64_t n;
  int d, nb, metric, strip, bufs;
  float radius;
  const float* radii;  // [m] or nullptr
  int exclude_self;
  // [m] hits so far; then [m]: a zero, [m + 1]: set when a query has more than cap, [m + 2]:
  // more than kWarpSort
  unsigned long long* counts;
  const int64_t* offs;         // [m] where a query's keys start, or nullptr: at query * cap
  int64_t cap;                 // most keys written for a query
  uint64_t* out;               // keys (squared distance, index)
  f32x2 nz;  // kNegZero2 (tile_dists)
};

// Bits of the largest squared distance that is a hit, -1 for none: the root is
// monotone, so the hits of a Euclidean radius are the squared distances up to the
// last one whose root does not exceed it (a few steps below the upper bound).
__device__ __forceinline__ int range_limit(float radius, int metric) {
  if (!(radius >= 0.0f)) return -1;
  float s = __uint_as_float(tile_limit_bits(radius + 0.0f, metric));  // (-0 counts as 0)
  if (metric == METRIC_EUCLIDEAN)
    while (__fsqrt_rn(s) > radius) s = __uint_as_float(__float_as_uint(s) - 1);
  return __float_as_int(s);
}

// Bound by FP32 issue like the kNN scan (20 000 queries and points, d = 16: 0.48 ms
// at 3 operations per pair and dimension unpacked).  A tile's distances are tested
// in registers; a warp without a hit leaves with one vote, and hits are written as
// squared distances: the sort takes the roots, of full warps of hits.  20 000-point
// self-join, d = 16, some 300 hits a row: 0.99 ms (the two passes of the
// thread-per-query scan: 2.73); with roots and a test per distance 1.28.
template <bool FMA8>
__global__ void __launch_bounds__(256, 2) range_tile_kernel(RangeTileArgs a) {
  extern __shared__ __align__(16) float rsm[];
  float* qT = rsm;                            // [d][kTileQS]
  float* xT = qT + (size_t)a.d * kTileQS;     // [bufs][d][kTilePS]
  const size_t xbuf = (size_t)a.d * kTilePS;
  __shared__ __align__(16) int s_lim[kRows];  // range_limit of each query
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t q0 = (int64_t)blockIdx.x * kRows;
  const int64_t qw = q0 + warp * kTileQ;
  int64_t t = (int64_t)blockIdx.y * a.strip;
  const int64_t t_end = min((a.n + kTileP - 1) / kTileP, t + a.strip);
  tile_stage(qT, kTileQS, a.A, q0, kRows, a.m, a.d, a.nb);
  tile_stage(xT, kTilePS, a.B, t * kTileP, kTileP, a.n, a.d, a.nb);
  if (threadIdx.x < kRows) {
    const int64_t q = q0 + threadIdx.x;
    s_lim[threadIdx.x] = q >= a.m ? -1 : range_limit(a.radii != nullptr ? a.radii[q] : a.radius, a.metric);
  }
  for (int buf = 0; t < t_end; t++) {
    cp_async_wait_all();
    __syncthreads();  // this tile has landed; with two buffers the other is no longer read
    if (a.bufs == 2 && t + 1 < t_end)
      tile_stage(xT + (buf ^ 1) * xbuf, kTilePS, a.B, (t + 1) * kTileP, kTileP, a.n, a.d, a.nb);
    float s[kTileQ][4];
    tile_dists<FMA8>(qT + warp * kTileQ, xT + buf * xbuf + lane, a.d, a.nb, a.nz, s);
    const int64_t p0 = t * kTileP;
    const float kNaN = __int_as_float(0x7fffffff);
    if (p0 + kTileP > a.n) {  // rows past the index are no hits
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (p0 + lane + 32 * i >= a.n)
#pragma unroll
          for (int j = 0; j < kTileQ; j++) s[j][i] = kNaN;
    }
    if (a.exclude_self && qw < p0 + kTileP && p0 < qw + kTileQ) {
#pragma unroll
      for (int j = 0; j < kTileQ; j++)
#pragma unroll
        for (int i = 0; i < 4; i++)
          if (p0 + lane + 32 * i == qw + j) s[j][i] = kNaN;
    }
    // squared distances are >= +0 or the canonical NaN: integer order, NaN above every limit
    const int4 l0 = *reinterpret_cast<const int4*>(s_lim + warp * kTileQ);
    const int4 l1 = *reinterpret_cast<const int4*>(s_lim + warp * kTileQ + 4);
    const int lim[kTileQ] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
    bool any = false;
#pragma unroll
    for (int j = 0; j < kTileQ; j++) any |= (int)tile_min_bits(s[j]) <= lim[j];
    if (__any_sync(0xffffffffu, any)) {
      int cnt = 0;  // lane j: hits of row j
#pragma unroll
      for (int j = 0; j < kTileQ; j++) {
        int c = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) c += __popc(__ballot_sync(0xffffffffu, __float_as_int(s[j][i]) <= lim[j]));
        if (lane == j) cnt = c;
      }
      // one lane per row takes the places of the row's hits
      uint64_t* place = nullptr;
      if (cnt > 0) {
        const int64_t q = qw + lane;
        const int64_t base = (int64_t)atomicAdd(a.counts + q, (unsigned long long)cnt);
        if (base + cnt > kWarpSort) a.counts[a.m + 2] = 1;
        if (base + cnt > a.cap) a.counts[a.m + 1] = 1;
        else place = a.out + (a.offs != nullptr ? a.offs[q] : q * a.cap) + base;
      }
#pragma unroll
      for (int j = 0; j < kTileQ; j++) {
        uint64_t* out = reinterpret_cast<uint64_t*>(shfl_u64(reinterpret_cast<uint64_t>(place), j));
        if (out == nullptr) continue;
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const bool hit = __float_as_int(s[j][i]) <= lim[j];
          const unsigned in = __ballot_sync(0xffffffffu, hit);
          if (hit) out[__popc(in & ((1u << lane) - 1u))] = make_key(s[j][i], (uint32_t)(p0 + lane + 32 * i));
          out += __popc(in);
        }
      }
    }
    if (a.bufs == 2) {
      buf ^= 1;
    } else if (t + 1 < t_end) {
      __syncthreads();
      tile_stage(xT, kTilePS, a.B, (t + 1) * kTileP, kTileP, a.n, a.d, a.nb);
    }
  }
}

// The key that a list is sorted by: the metric's distance for the squared one.
__device__ __forceinline__ uint64_t range_key(uint64_t key, int metric) {
  return metric == METRIC_EUCLIDEAN ? make_key(__fsqrt_rn(key_dist(key)), (uint32_t)key) : key;
}

// The c <= 32 R keys at `in`, sorted, to put(rank, key).
template <int R, typename Put>
__device__ __forceinline__ void sort_slots(const uint64_t* __restrict__ in, int c, int metric, int lane, Put put) {
  uint64_t v[R];
#pragma unroll
  for (int r = 0; r < R; r++) v[r] = lane + 32 * r < c ? range_key(in[lane + 32 * r], metric) : KEY_NONE;
  warp_sort_keys<R>(v, lane);
#pragma unroll
  for (int r = 0; r < R; r++)
    if (lane * R + r < c) put(lane * R + r, v[r]);
}
template <typename Put>
__device__ __forceinline__ void warp_sort_slots(const uint64_t* __restrict__ in, int c, int metric, int lane, Put put) {
  if (c <= 32) sort_slots<1>(in, c, metric, lane, put);
  else if (c <= 64) sort_slots<2>(in, c, metric, lane, put);
  else if (c <= 128) sort_slots<4>(in, c, metric, lane, put);
  else sort_slots<8>(in, c, metric, lane, put);
}

// A query's slots sorted into its place of the result, up to kWarpSort keys: a warp
// per query, in registers.
__global__ void __launch_bounds__(256) range_rows_kernel(const uint64_t* __restrict__ slots, int64_t cap, int64_t m,
                                                         int metric, const int64_t* __restrict__ offs,
                                                         int64_t* __restrict__ idx, float* __restrict__ dist) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t q = (int64_t)blockIdx.x * 8 + warp;
  if (q >= m) return;
  const int64_t o = offs[q], c = offs[q + 1] - o;
  if (c > 0 && c <= kWarpSort)
    warp_sort_slots(slots + q * cap, (int)c, metric, lane, [&](int e, uint64_t key) {
      idx[o + e] = key_idx(key);
      dist[o + e] = key_dist(key);
    });
}

// The longer lists, up to kSlots keys, a block each (other queries' blocks leave at
// once), by merging: a thread sorts V keys in registers, then runs are merged two by
// two, a thread making V consecutive keys of every merge from where their ranks split
// the two runs (the merge path of Green, McColl and Bader).  A key costs some 30
// instructions in the registers' network and 20 a merge; a warp's network of 256 costs
// 300.  Keys sit one past every 16 in shared memory, so that a warp's threads, V keys
// apart, use different banks.  27 lists of 3365 keys 27 us, 2211 of 2344 137; eight lists
// to a block, one after the other by ranks among sorted pieces, and whole calls: 849 us
// (now 115; the two-pass scan with a segmented sort 227) and 760 (398; 484).
__device__ __forceinline__ int list_pos(int e) { return e + (e >> 4); }

template <int V>
__device__ __forceinline__ void sort_list(const uint64_t* __restrict__ in, int n, int metric, uint64_t* s_key) {
  uint64_t v[V];
#pragma unroll
  for (int r = 0; r < V; r++) {
    const int e = (int)threadIdx.x + 256 * r;
    v[r] = e < n ? range_key(in[e], metric) : KEY_NONE;
  }
#pragma unroll
  for (int k2 = 2; k2 <= V; k2 <<= 1)
#pragma unroll
    for (int j = k2 >> 1; j > 0; j >>= 1)
#pragma unroll
      for (int r = 0; r < V; r++) {
        if (r & j) continue;
        const uint64_t x = v[r], y = v[r ^ j];
        const bool sw = (r & k2) == 0 ? x > y : x < y;
        v[r] = sw ? y : x;
        v[r ^ j] = sw ? x : y;
      }
  const int k0 = (int)threadIdx.x * V;  // this thread's keys of every merge: [k0, k0 + V)
#pragma unroll
  for (int r = 0; r < V; r++) s_key[list_pos(k0 + r)] = v[r];
  __syncthreads();
#pragma unroll 1
  for (int w = V; w < 256 * V; w *= 2) {
    const int a = k0 & ~(2 * w - 1), b = a + w, k = k0 - a;  // runs at a and b; k keys of the merge come before
    int lo = max(0, k - w), hi = min(k, w);  // how many of those are of the first run
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (s_key[list_pos(a + mid)] < s_key[list_pos(b + k - 1 - mid)]) lo = mid + 1;
      else hi = mid;
    }
    int i = lo, j = k - lo;
    uint64_t va = i < w ? s_key[list_pos(a + i)] : KEY_NONE, vb = j < w ? s_key[list_pos(b + j)] : KEY_NONE;
#pragma unroll
    for (int r = 0; r < V; r++) {
      const bool first = j >= w || (i < w && va <= vb);
      v[r] = first ? va : vb;
      if (first) i++;
      else j++;
      const uint64_t next = first ? (i < w ? s_key[list_pos(a + i)] : KEY_NONE)
                                  : (j < w ? s_key[list_pos(b + j)] : KEY_NONE);
      va = first ? next : va;
      vb = first ? vb : next;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < V; r++) s_key[list_pos(k0 + r)] = v[r];
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) range_long_kernel(const uint64_t* __restrict__ slots, int64_t cap, int metric,
                                                         const int64_t* __restrict__ offs, int64_t* __restrict__ idx,
                                                         float* __restrict__ dist) {
  static_assert(kSlots == 256 * 16 && kWarpSort == 256, "2 to 16 keys per thread");
  __shared__ uint64_t s_key[kSlots + kSlots / 16];
  const int64_t q = blockIdx.x;
  const int64_t o = offs[q];
  if (offs[q + 1] - o <= kWarpSort) return;
  const int n = (int)(offs[q + 1] - o);
  const uint64_t* in = slots + q * cap;
  if (n <= 512) sort_list<2>(in, n, metric, s_key);
  else if (n <= 1024) sort_list<4>(in, n, metric, s_key);
  else if (n <= 2048) sort_list<8>(in, n, metric, s_key);
  else sort_list<16>(in, n, metric, s_key);
  for (int e = threadIdx.x; e < n; e += 256) {
    const uint64_t key = s_key[list_pos(e)];
    idx[o + e] = key_idx(key);
    dist[o + e] = key_dist(key);
  }
}

// Squared distances to the metric's in place (lists too long for the slots).
__global__ void root_keys_kernel(uint64_t* __restrict__ keys, int64_t total) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < total) keys[e] = range_key(keys[e], METRIC_EUCLIDEAN);
}

}  // namespace

// The result's arrays, both or neither.
static int result_alloc(int64_t** d_idx, float** d_dist, int64_t tot) {
  if (cudaMalloc(d_idx, sizeof(int64_t) * tot) == cudaSuccess) {
    if (cudaMalloc(d_dist, sizeof(float) * tot) == cudaSuccess) return ST_OK;
    cudaFree(*d_idx);
  }
  cudaGetLastError();
  *d_idx = nullptr;
  *d_dist = nullptr;
  set_error("no device memory for a range result of %lld hits", (long long)tot);
  return ST_ENOMEM;
}

bool tile_range_supported(int d) { return d >= 1 && d <= kRangeMaxD; }

int tile_range(const ExactScanParams& p, float radius, int exclude_self, int64_t* d_off, int64_t** d_idx,
               float** d_dist, int64_t* total, cudaStream_t stream, const float* radii, int* passes) {
  Scratch counts, tmp, slots;
  FUELG_TRY(counts.alloc(sizeof(int64_t) * (p.m + 3), stream));
  FUELG_CUDA(cudaMemsetAsync(counts.p, 0, sizeof(int64_t) * (p.m + 3), stream));
  const int64_t cap = std::min<int64_t>(
      p.n, std::clamp<int64_t>((int64_t)(kSlotBytes / sizeof(uint64_t)) / p.m, 32, kSlots));
  FUELG_TRY(slots.alloc(sizeof(uint64_t) * cap * p.m, stream));
  RangeTileArgs a{};
  a.A = p.A;
  a.m = p.m;
  a.B = p.B;
  a.n = p.n;
  a.d = p.d;
  a.nb = p.d / 8;
  a.metric = p.metric;
  a.radius = radius;
  a.radii = radii;
  a.exclude_self = exclude_self;
  a.counts = counts.as<unsigned long long>();
  a.cap = cap;
  a.out = slots.as<uint64_t>();
  a.nz = kNegZero2;
  // two buffers while two CTAs still fit an SM; strips as long as leaves four CTAs
  // for each place on the chip (both as for the pairwise tiles)
  const size_t smem2 = sizeof(float) * p.d * (kTileQS + 2 * kTilePS);
  const size_t smem1 = sizeof(float) * p.d * (kTileQS + kTilePS);
  a.bufs = smem2 <= kTwoCtas ? 2 : 1;
  const size_t smem = a.bufs == 2 ? smem2 : smem1;
  const int64_t qb = (p.m + kRows - 1) / kRows, tb = (p.n + kTileP - 1) / kTileP;
  a.strip = (int)std::max<int64_t>(std::clamp<int64_t>(qb * tb / (kTwoPerSm * 4), 1, kMaxStrip),
                                   (tb + 65534) / 65535);
  auto pass = [&]() -> int {
    auto kern = p.order == ORDER_X86 ? range_tile_kernel<true> : range_tile_kernel<false>;
    FUELG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kTwoCtas));
    kern<<<dim3((unsigned)qb, (unsigned)((tb + a.strip - 1) / a.strip)), 256, smem, stream>>>(a);
    ::fuelg::note_launch();
    FUELG_CUDA(cudaGetLastError());
    ++*passes;
    return ST_OK;
  };
  FUELG_TRY(pass());
  size_t sb = 0;
  FUELG_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, sb, counts.as<int64_t>(), d_off, p.m + 1, stream));
  FUELG_TRY(tmp.alloc(sb, stream));
  FUELG_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, sb, counts.as<int64_t>(), d_off, p.m + 1, stream));
  int64_t tot = 0, flags[2] = {0, 0};
  FUELG_CUDA(cudaMemcpyAsync(&tot, d_off + p.m, sizeof(int64_t), cudaMemcpyDeviceToHost, stream));
  FUELG_CUDA(cudaMemcpyAsync(flags, counts.as<int64_t>() + p.m + 1, sizeof(flags), cudaMemcpyDeviceToHost, stream));
  FUELG_CUDA(cudaStreamSynchronize(stream));
  const bool over = flags[0] != 0, longer = flags[1] != 0;
  *total = tot;
  if (tot == 0) return ST_OK;
  if (!over) {
    FUELG_TRY(result_alloc(d_idx, d_dist, tot));
    range_rows_kernel<<<(unsigned)((p.m + 7) / 8), 256, 0, stream>>>(slots.as<uint64_t>(), cap, p.m, p.metric, d_off,
                                                                     *d_idx, *d_dist);
    ::fuelg::note_launch();
    if (longer) {
      range_long_kernel<<<(unsigned)p.m, 256, 0, stream>>>(slots.as<uint64_t>(), cap, p.metric, d_off, *d_idx, *d_dist);
      ::fuelg::note_launch();
    }
    FUELG_CUDA(cudaGetLastError());
    return ST_OK;
  }
  slots.release();  // the lists take their place
  Scratch keys, sorted, sort_tmp;
  FUELG_TRY(keys.alloc(sizeof(uint64_t) * tot, stream));
  FUELG_TRY(sorted.alloc(sizeof(uint64_t) * tot, stream));
  FUELG_CUDA(cudaMemsetAsync(counts.p, 0, sizeof(int64_t) * p.m, stream));
  a.offs = d_off;
  a.cap = p.n;
  a.out = keys.as<uint64_t>();
  FUELG_TRY(pass());
  if (p.metric == METRIC_EUCLIDEAN) {
    root_keys_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, stream>>>(keys.as<uint64_t>(), tot);
    ::fuelg::note_launch();
    FUELG_CUDA(cudaGetLastError());
  }
  sb = 0;
  FUELG_CUDA(cub::DeviceSegmentedSort::SortKeys(nullptr, sb, keys.as<uint64_t>(), sorted.as<uint64_t>(), tot, p.m,
                                                d_off, d_off + 1, stream));
  FUELG_TRY(sort_tmp.alloc(sb, stream));
  FUELG_CUDA(cub::DeviceSegmentedSort::SortKeys(sort_tmp.p, sb, keys.as<uint64_t>(), sorted.as<uint64_t>(), tot, p.m,
                                                d_off, d_off + 1, stream));
  FUELG_TRY(result_alloc(d_idx, d_dist, tot));  // (120 us or more of host time, beside the sort)
  return split_keys(sorted.as<uint64_t>(), tot, *d_idx, *d_dist, stream);
}

}  // namespace fuelg
