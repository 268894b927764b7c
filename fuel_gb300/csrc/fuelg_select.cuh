// fuelg_select.cuh -- warp-cooperative selection of the smallest (distance,
// index) keys, shared by the tensor-core screen and the FP32 tile scan.
#pragma once
#include "fuelg_common.cuh"

namespace fuelg {

constexpr int kSel = 8;  // keys per lane in a selection (appended or prefix): 256 per warp

// Number of held keys below t over the warp.
__device__ __forceinline__ int warp_count_hi_below(const uint32_t (&hi)[2 * kSel], uint32_t t) {
  int c = 0;
#pragma unroll
  for (int i = 0; i < 2 * kSel; i++) c += hi[i] < t ? 1 : 0;
  return __reduce_add_sync(0xffffffffu, c);
}

// Warp-cooperative selection for one query: the union of its
// na (<= 256) appended keys and its plen (<= kk <= 256) kept keys is reduced
// to its kk smallest, written unsorted back over cur[0, min(kk, na + plen)).
// The kk-th smallest key is found by a bitwise binary search over the
// distance word (counting with a warp reduction) and, only when several keys
// share that distance, over the index word; keys are unique.  Each search
// starts below the bits that the smallest and largest candidate word share.
// In place: every lane has read its keys before the first warp-wide
// exchange, and every store comes after the last.  No shared memory, no sort.
// Returns the kk-th smallest key, or KEY_NONE while fewer than kk are held,
// on every lane.
static __device__ __noinline__ uint64_t warp_select(const uint64_t* __restrict__ app, int na, uint64_t* cur, int plen,
                                             int kk, int lane) {
  uint64_t key[2 * kSel];
#pragma unroll
  for (int i = 0; i < kSel; i++) {
    const int e = lane + 32 * i;
    key[i] = e < na ? app[e] : KEY_NONE;
    key[kSel + i] = e < plen ? cur[e] : KEY_NONE;
  }
  uint32_t hi[2 * kSel];
  uint32_t hmin = 0xffffffffu, hmax = 0;
#pragma unroll
  for (int i = 0; i < 2 * kSel; i++) {
    hi[i] = (uint32_t)(key[i] >> 32);
    if (key[i] != KEY_NONE) {
      hmin = min(hmin, hi[i]);
      hmax = max(hmax, hi[i]);
    }
  }
  const int total = na + plen;
  uint64_t kth = KEY_NONE;
  if (total >= kk) {
    // the kk-th distance word lies in [hmin, hmax]: search the bits below
    // their common prefix only
    hmin = __reduce_min_sync(0xffffffffu, hmin);
    hmax = __reduce_max_sync(0xffffffffu, hmax);
    int top = hmin == hmax ? -1 : 31 - __clz(hmin ^ hmax);
    uint32_t H = top >= 0 ? hmin & ~((2u << top) - 1u) : hmin;
    for (int b = top; b >= 0; b--) {
      const uint32_t t = H | (1u << b);
      if (warp_count_hi_below(hi, t) < kk) H = t;
    }
    // keys below H: fewer than kk; keys with hi == H: the rest is taken from them
    const int below = warp_count_hi_below(hi, H);
    int eq = 0;
    uint32_t lmin = 0xffffffffu, lmax = 0;
#pragma unroll
    for (int i = 0; i < 2 * kSel; i++)
      if (hi[i] == H) {
        eq++;
        lmin = min(lmin, (uint32_t)key[i]);
        lmax = max(lmax, (uint32_t)key[i]);
      }
    eq = __reduce_add_sync(0xffffffffu, eq);
    lmax = __reduce_max_sync(0xffffffffu, lmax);
    const int need = kk - below;
    uint32_t Lo = lmax;
    if (eq != need) {
      lmin = __reduce_min_sync(0xffffffffu, lmin);
      top = lmin == lmax ? -1 : 31 - __clz(lmin ^ lmax);
      Lo = top >= 0 ? lmin & ~((2u << top) - 1u) : lmin;
      for (int b = top; b >= 0; b--) {
        const uint32_t t = Lo | (1u << b);
        int c = 0;
#pragma unroll
        for (int i = 0; i < 2 * kSel; i++) c += (hi[i] == H && (uint32_t)key[i] < t) ? 1 : 0;
        if (__reduce_add_sync(0xffffffffu, c) < need) Lo = t;
      }
    }
    kth = ((uint64_t)H << 32) | Lo;
  }
  // compact the kept keys: lane offsets by a warp scan of per-lane counts
  int mine = 0;
#pragma unroll
  for (int i = 0; i < 2 * kSel; i++) mine += (key[i] != KEY_NONE && key[i] <= kth) ? 1 : 0;
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  int pos = incl - mine;
#pragma unroll
  for (int i = 0; i < 2 * kSel; i++)
    if (key[i] != KEY_NONE && key[i] <= kth) cur[pos++] = key[i];
  __syncwarp();
  return total >= kk ? kth : KEY_NONE;
}

// A distance-word limit t for the keys the lanes hold in hi[] (0xffffffff: no
// key): at least kk of them lie below t, and no more than kk + slack unless more
// share one word.  Returns t, the number below it in *below.  total >= kk keys,
// words in [hmin, hmax].  Where the words are spread evenly, aiming at the rank
// between the two counts takes two or three steps; every third step halves the
// range instead, which bounds them.
template <int N>
__device__ __forceinline__ uint32_t warp_cut(const uint32_t (&hi)[N], int total, int kk, int slack, uint32_t hmin,
                                             uint32_t hmax, int* below) {
  uint32_t lo = hmin, up = hmax + 1;  // count(< lo) = clo < kk <= cnt = count(< up)
  int clo = 0, cnt = total;
#pragma unroll 1
  for (int step = 1; cnt > kk + slack && up - lo > 1; step++) {
    const uint32_t span = up - lo;
    uint32_t mid = lo + span / 2;
    if (step % 3 != 0) {
      const float f = ((float)(kk - clo) + 0.5f * (float)slack) / (float)(cnt - clo);
      mid = lo + min(span - 1, max(1u, (uint32_t)(f * (float)span)));
    }
    int c = 0;
#pragma unroll
    for (int i = 0; i < N; i++) c += hi[i] < mid ? 1 : 0;
    c = __reduce_add_sync(0xffffffffu, c);
    if (c >= kk) {
      up = mid;
      cnt = c;
    } else {
      lo = mid;
      clo = c;
    }
  }
  *below = cnt;
  return up;
}

// v of the lanes sorted ascending over the warp (bitonic network, 15 stages).
__device__ __forceinline__ uint64_t warp_sort32(uint64_t v, int lane) {
#pragma unroll
  for (int k2 = 2; k2 <= 32; k2 <<= 1) {
#pragma unroll
    for (int j = k2 >> 1; j > 0; j >>= 1) {
      const uint64_t o = ((uint64_t)__shfl_xor_sync(0xffffffffu, (uint32_t)(v >> 32), j) << 32) |
                         __shfl_xor_sync(0xffffffffu, (uint32_t)v, j);
      const bool keep_min = ((lane & j) == 0) == ((lane & k2) == 0);
      v = (o < v) == keep_min ? o : v;
    }
  }
  return v;
}

// The 32 smallest of `kept` (ascending over the lanes) and v (any order),
// ascending over the lanes: v is sorted, reversed against kept (the lane-wise
// minima are the 32 smallest, a bitonic sequence) and merged in five stages.
__device__ __forceinline__ uint64_t warp_merge32(uint64_t kept, uint64_t v, int lane) {
  v = warp_sort32(v, lane);
  const uint64_t r = ((uint64_t)__shfl_xor_sync(0xffffffffu, (uint32_t)(v >> 32), 31) << 32) |
                     __shfl_xor_sync(0xffffffffu, (uint32_t)v, 31);
  kept = r < kept ? r : kept;
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) {
    const uint64_t o = ((uint64_t)__shfl_xor_sync(0xffffffffu, (uint32_t)(kept >> 32), j) << 32) |
                       __shfl_xor_sync(0xffffffffu, (uint32_t)kept, j);
    kept = (o < kept) == ((lane & j) == 0) ? o : kept;
  }
  return kept;
}

// One key into the warp's ascending list of 32 (the largest falls out).
__device__ __forceinline__ uint64_t warp_insert32(uint64_t kept, uint64_t key, int lane) {
  const uint64_t up = ((uint64_t)__shfl_up_sync(0xffffffffu, (uint32_t)(kept >> 32), 1) << 32) |
                      __shfl_up_sync(0xffffffffu, (uint32_t)kept, 1);
  return kept < key ? kept : (lane == 0 || up < key) ? key : up;
}

__device__ __forceinline__ uint64_t shfl_u64(uint64_t v, int src) {
  return ((uint64_t)__shfl_sync(0xffffffffu, (uint32_t)(v >> 32), src) << 32) |
         __shfl_sync(0xffffffffu, (uint32_t)v, src);
}

// Ascending bitonic sort of the warp's 32 R keys, element e = lane * R + r in v[r].
template <int R>
__device__ __forceinline__ void warp_sort_keys(uint64_t (&v)[R], int lane) {
#pragma unroll
  for (int k2 = 2; k2 <= 32 * R; k2 <<= 1) {
#pragma unroll
    for (int j = k2 >> 1; j > 0; j >>= 1) {
      if (j >= R) {
#pragma unroll
        for (int r = 0; r < R; r++) {
          const uint64_t o = ((uint64_t)__shfl_xor_sync(0xffffffffu, (uint32_t)(v[r] >> 32), j / R) << 32) |
                             __shfl_xor_sync(0xffffffffu, (uint32_t)v[r], j / R);
          const int e = lane * R + r;
          const bool up = (e & k2) == 0;
          const bool lower = (e & j) == 0;
          v[r] = (lower == up) ? (o < v[r] ? o : v[r]) : (o > v[r] ? o : v[r]);
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; r++) {
          if (r & j) continue;
          const int e = lane * R + r;
          const bool up = (e & k2) == 0;
          const uint64_t x = v[r], y = v[r ^ j];
          const bool sw = up ? (x > y) : (x < y);
          v[r] = sw ? y : x;
          v[r ^ j] = sw ? x : y;
        }
      }
    }
  }
}

}  // namespace fuelg
