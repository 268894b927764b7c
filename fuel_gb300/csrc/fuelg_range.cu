// fuelg_range.cu -- range search of rows of up to 128 dimensions in register tiles
// (linear_scan_range, src/api/search.rs:154-166).
//
// One pass over all pairs (tile_dists: 64 queries x 128 index rows) counts each
// query's hits and writes their keys into the query's slots in whatever order
// they come; the keys are unique, so the sort by (distance, index) that the result
// needs anyway makes the order definite.  The counts' prefix sums are the result's
// offsets, and one warp (above 256 hits: one block) sorts a query's slots into its
// place.  Only when a query has more hits than slots does a second pass fill the
// lists at their offsets, for a segmented sort.
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
// Most slots of a query: what a block sorts in the shared memory that lets five
// blocks share an SM.  (With 1024 the 300-hit self-join had rows past them and took
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
  unsigned long long* counts;  // [m] hits so far; then [m]: a zero, [m + 1]: set when a query has more than cap
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

// A query's slots sorted into its place of the result: a warp per query, in
// registers.  A query with more than kWarpSort keys by the whole block: pieces of up
// to kWarpSort keys, sorted by a warp each, and every key's rank from its place
// in its own piece and a binary search in each of the others.  0.33 ms for the same
// self-join (a segmented sort over all lists and a split of its keys: 1.25).
// Whole calls: that one 4.32 -> 1.74 ms, 20 000 x 20 000 x 16 with 19 hits a row
// 2.83 -> 1.23, 40 queries on 40 000 x 64 0.92 -> 0.13; with 3900 hits a row, many
// lists past the slots, 11.8 -> 11.7.
__global__ void __launch_bounds__(256) range_rows_kernel(const uint64_t* __restrict__ slots, int64_t cap, int64_t m,
                                                         int metric, const int64_t* __restrict__ offs,
                                                         int64_t* __restrict__ idx, float* __restrict__ dist) {
  __shared__ uint64_t s_key[kSlots];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t q0 = (int64_t)blockIdx.x * 8;
  const int64_t q = q0 + warp;
  int c = 0;
  if (q < m) {
    const int64_t o = offs[q];
    c = (int)(offs[q + 1] - o);
    if (c > 0 && c <= kWarpSort)
      warp_sort_slots(slots + q * cap, c, metric, lane, [&](int e, uint64_t key) {
        idx[o + e] = key_idx(key);
        dist[o + e] = key_dist(key);
      });
  }
  if (!__syncthreads_or(c > kWarpSort)) return;
  for (int w = 0; w < 8 && q0 + w < m; w++) {
    const int64_t o = offs[q0 + w];
    const int n = (int)(offs[q0 + w + 1] - o);
    if (n <= kWarpSort) continue;
    const uint64_t* in = slots + (q0 + w) * cap;
    const int pieces = (n + kWarpSort - 1) / kWarpSort, len = (n + pieces - 1) / pieces;
    __syncthreads();  // the previous query's keys are no longer read
    for (int p = warp; p < pieces; p += 8) {
      const int b = p * len;
      warp_sort_slots(in + b, min(len, n - b), metric, lane, [&](int e, uint64_t key) { s_key[b + e] = key; });
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n; e += 256) {
      const uint64_t key = s_key[e];
      const int own = e / len;
      int rank = e - own * len;
      for (int p = 0; p < pieces; p++) {
        if (p == own) continue;
        const uint64_t* s = s_key + p * len;
        int lo = 0, hi = min(len, n - p * len);  // keys below: [0, lo) are, [hi, ..) are not
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (s[mid] < key) lo = mid + 1;
          else hi = mid;
        }
        rank += lo;
      }
      idx[o + rank] = key_idx(key);
      dist[o + rank] = key_dist(key);
    }
  }
}

// Squared distances to the metric's in place (lists too long for the slots).
__global__ void root_keys_kernel(uint64_t* __restrict__ keys, int64_t total) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < total) keys[e] = range_key(keys[e], METRIC_EUCLIDEAN);
}

}  // namespace

// No memory for the result or the sort: nothing is left of it.
static int no_room(int64_t** d_idx, float** d_dist, int64_t tot) {
  if (*d_idx) cudaFree(*d_idx);
  if (*d_dist) cudaFree(*d_dist);
  *d_idx = nullptr;
  *d_dist = nullptr;
  set_error("no device memory for a range result of %lld hits", (long long)tot);
  return ST_ENOMEM;
}

bool tile_range_supported(int d) { return d >= 1 && d <= kRangeMaxD; }

int tile_range(const ExactScanParams& p, float radius, int exclude_self, int64_t* d_off, int64_t** d_idx,
               float** d_dist, int64_t* total, cudaStream_t stream, const float* radii, int* passes) {
  Scratch counts, tmp, slots;
  FUELG_TRY(counts.alloc(sizeof(int64_t) * (p.m + 2), stream));
  FUELG_CUDA(cudaMemsetAsync(counts.p, 0, sizeof(int64_t) * (p.m + 2), stream));
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
  int64_t tot = 0, over = 0;
  FUELG_CUDA(cudaMemcpyAsync(&tot, d_off + p.m, sizeof(int64_t), cudaMemcpyDeviceToHost, stream));
  FUELG_CUDA(cudaMemcpyAsync(&over, counts.as<int64_t>() + p.m + 1, sizeof(int64_t), cudaMemcpyDeviceToHost, stream));
  FUELG_CUDA(cudaStreamSynchronize(stream));
  *total = tot;
  if (tot == 0) return ST_OK;
  Scratch keys, sorted, sort_tmp;
  if (over) {
    slots.release();  // the lists below take their place
    FUELG_TRY(keys.alloc(sizeof(uint64_t) * tot, stream));
    FUELG_TRY(sorted.alloc(sizeof(uint64_t) * tot, stream));
  }
  if (cudaMalloc(d_idx, sizeof(int64_t) * tot) != cudaSuccess ||
      cudaMalloc(d_dist, sizeof(float) * tot) != cudaSuccess) {
    cudaGetLastError();
    return no_room(d_idx, d_dist, tot);
  }
  if (!over) {
    range_rows_kernel<<<(unsigned)((p.m + 7) / 8), 256, 0, stream>>>(slots.as<uint64_t>(), cap, p.m, p.metric, d_off,
                                                                     *d_idx, *d_dist);
    ::fuelg::note_launch();
    FUELG_CUDA(cudaGetLastError());
    return ST_OK;
  }
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
  if (sort_tmp.alloc(sb, stream) != ST_OK) return no_room(d_idx, d_dist, tot);
  FUELG_CUDA(cub::DeviceSegmentedSort::SortKeys(sort_tmp.p, sb, keys.as<uint64_t>(), sorted.as<uint64_t>(), tot, p.m,
                                                d_off, d_off + 1, stream));
  return split_keys(sorted.as<uint64_t>(), tot, *d_idx, *d_dist, stream);
}

}  // namespace fuelg
