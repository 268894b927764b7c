// fuelg_batched.cu -- many independent Lloyd k-means problems in one pass
// per iteration.
//
// Every problem keeps fuel's Lloyd semantics exactly as fuelg_kmeans_lloyd
// does (src/cluster/kmeans/lloyd.rs:12-202 with fixed initial centres): the
// initial assignment in the vec_pairwise_sqdist order, later passes in the
// math::sqdist order, strict < over centres (first index wins), empty
// clusters keep their centre, centres = correctly rounded f32 of the exact
// mean (integer sums at the problem's scale 2^e_lo, 32-bit slices in 64-bit
// counters, order independent), iteration counting with the initial pass as
// iteration 1 and the changed == 0 stop.  Results are bit-identical to one
// fuelg_kmeans_lloyd call per problem.
//
// Layout: all problems' points are packed row-major one after another; work
// items are 256-row slices of one problem, handed to persistent CTAs in
// contiguous ranges so a CTA reloads a problem's centres into shared memory
// only when its range crosses into the next problem.  One kernel per
// iteration assigns every point of every problem and, for points whose label
// changed, adds +x / -x to the cluster sums: per CTA in shared memory when a
// problem's k*d*L counters fit (many points per counter: few global atomics),
// straight to global counters otherwise.  A second kernel turns the sums into
// centres.  The middle iterations are one CUDA graph replayed.
#include <cuda.h>
#include <unistd.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

#include "../../include/fuelg.h"
#include "fuelg_common.cuh"
#include "fuelg_exact.cuh"
#include "fuelg_internal.h"
#include "fuelg_tc_common.cuh"
#include "fuelg_tile.cuh"

namespace fuelg {
namespace {

constexpr int kItemRows = 256;       // rows per work item = threads per CTA
constexpr int kCentreCap = 16384;    // centre floats staged in shared memory (64 KB)
constexpr int kAggCap = 2048;        // per-CTA sum counters in shared memory (16 KB)

struct BProb {
  int64_t x_off;     // float offset of the problem's rows
  int64_t n;
  int64_t lab_off;   // label offset
  int64_t c_off;     // centre float offset (k * d)
  int64_t limb_off;  // counter offset (k * d * L)
  int32_t cnt_off;   // count offset (k)
  int32_t d, k, L, e_lo;
  int32_t item_begin;  // first work item
  int32_t active;      // 0: skipped (bad data)
  int64_t cost_begin;  // cumulative work before this problem's first item
  int64_t item_cost;   // work of one item (~ k * d)
  int32_t all_item_begin;  // first 256-row item over all problems (inertia)
  int32_t tc;              // assigned by the tensor-core screen (no CUDA-core items)
};

// First work item whose work offset is >= c (work offsets: the problem's
// cost_begin + j * item_cost for its item j), so CTAs can take contiguous item
// ranges of equal work instead of equal item counts.
__device__ __forceinline__ int64_t item_at_cost(const BProb* __restrict__ probs, int P, int items_total, int64_t c) {
  int lo = 0, hi = P;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (probs[mid].cost_begin <= c) lo = mid;
    else hi = mid;
  }
  const BProb& pr = probs[lo];
  const int64_t items = (lo + 1 < P ? probs[lo + 1].item_begin : items_total) - pr.item_begin;
  const int64_t j = (c - pr.cost_begin + pr.item_cost - 1) / pr.item_cost;
  return j >= items ? pr.item_begin + items : pr.item_begin + j;
}

template <int D>
struct Dim {
  static constexpr int value = D;
};

// Where a problem's rows and first centres are: the caller's device memory, or
// already in their places in X and C (copied there, host memory).
struct BSrc {
  const float* x;
  const float* c;
  int64_t x_len;  // n d
};

// The problems' rows into X, 64K values per block, and their exponent ranges on the
// way; zeros up to the next problem's 16-byte boundary.  One launch instead of a
// copy per problem, a clear and a pass over X (512 problems, 2.4 GB, in device memory:
// the call 57.2 -> 47.3 ms, with the centres leaving by one copy).
__global__ void __launch_bounds__(256) batched_gather_kernel(const BSrc* __restrict__ src, float* __restrict__ X,
                                                             const int64_t* __restrict__ off,
                                                             const int32_t* __restrict__ blk_begin, int P,
                                                             int* __restrict__ out) {
  int lo_b = 0, hi_b = P;  // problem of this block
  while (hi_b - lo_b > 1) {
    const int mid = (lo_b + hi_b) >> 1;
    if (blk_begin[mid] <= (int)blockIdx.x) lo_b = mid;
    else hi_b = mid;
  }
  const int p = lo_b;
  const BSrc sp = src[p];
  const int64_t s0 = (int64_t)((int)blockIdx.x - blk_begin[p]) * 65536;
  const int64_t s1 = min(s0 + 65536, sp.x_len);
  float* dst = X + off[p];
  const bool copy = sp.x != dst;
  int lo = 1 << 30, hi = -(1 << 30), bad = 0;
  auto see = [&](float v) {
    uint32_t mant;
    int l, h;
    bool z, b;
    f32_parts(v, mant, l, h, z, b);
    if (b) bad = 1;
    if (!z && !b) {
      lo = min(lo, l);
      hi = max(hi, h);
    }
  };
  int64_t e = s0;
  if ((reinterpret_cast<uintptr_t>(sp.x) & 15) == 0) {  // (dst is aligned)
    const int64_t v1 = (s1 - s0) >> 2;
    const float4* s4 = reinterpret_cast<const float4*>(sp.x + s0);
    float4* d4 = reinterpret_cast<float4*>(dst + s0);
#pragma unroll 4
    for (int64_t v = threadIdx.x; v < v1; v += 256) {
      const float4 f = s4[v];
      if (copy) d4[v] = f;
      see(f.x);
      see(f.y);
      see(f.z);
      see(f.w);
    }
    e = s0 + 4 * v1;
  }
  for (e += threadIdx.x; e < s1; e += 256) {
    const float f = sp.x[e];
    if (copy) dst[e] = f;
    see(f);
  }
  // padding up to the next problem (at most 3 values)
  if (s1 == sp.x_len && threadIdx.x < off[p + 1] - off[p] - sp.x_len) dst[sp.x_len + threadIdx.x] = 0.0f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    bad |= __shfl_xor_sync(0xffffffffu, bad, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&out[3 * p], lo);
    atomicMax(&out[3 * p + 1], hi);
    if (bad) atomicOr(&out[3 * p + 2], 1);
  }
}

// The problems' first centres into C, a block per problem.
__global__ void __launch_bounds__(256) batched_centres_kernel(const BSrc* __restrict__ src,
                                                              const BProb* __restrict__ probs, float* __restrict__ C) {
  const BProb& pr = probs[blockIdx.x];
  const float* c = src[blockIdx.x].c;
  float* dst = C + pr.c_off;
  if (c == dst) return;
  for (int64_t e = threadIdx.x; e < (int64_t)pr.k * pr.d; e += 256) dst[e] = c[e];
}

// Adds the exact slices of +-x (coordinate `dim` of a point) to cluster c.
__device__ __forceinline__ void add_coord(unsigned long long* __restrict__ dst, float x, int e_lo, int L, bool neg) {
  const unsigned __int128 v = fixed_of(x, e_lo, neg);
  for (int l = 0; l < L; l++) {
    const unsigned long long sl = (unsigned long long)((v >> (32 * l)) & 0xffffffffu);
    if (sl) atomicAdd(dst + l, sl);
  }
}

// The squared distances from x (each coordinate twice) to two centres c (their
// coordinates interleaved), two lanes of one packed chain: the operation
// sequence of exact_dist_fn<KIND, ORDER, D> for D = 2 or 8.  nz is kNegZero2, as
// an argument: a product plus an explicit -0 stays a product of its own.
template <int KIND, int ORDER, int D>
__device__ __forceinline__ f32x2 exact_dist_pair(const f32x2 (&x)[D], const f32x2* __restrict__ c, f32x2 nz) {
  static_assert(D == 2 || D == 8, "");
  static_assert(KIND == KIND_SQDIST || KIND == KIND_PAIRWISE, "");
  constexpr bool fma_chain = KIND == KIND_PAIRWISE && ORDER == ORDER_X86 && D >= 4;
  constexpr bool tree = KIND == KIND_SQDIST && ORDER == ORDER_X86 && D == 8;
  f32x2 sq[D];
  f32x2 s = 0;
#pragma unroll
  for (int t = 0; t < D; t += 2) {
    const ulonglong2 cc = *reinterpret_cast<const ulonglong2*>(c + t);
    const f32x2 d0 = fma2(cc.x, kNegOne2, x[t]), d1 = fma2(cc.y, kNegOne2, x[t + 1]);
    if (fma_chain) {
      s = t == 0 ? fma2(d0, d0, nz) : fma2(d0, d0, s);
      s = fma2(d1, d1, s);
    } else {
      sq[t] = fma2(d0, d0, nz);
      sq[t + 1] = fma2(d1, d1, nz);
    }
  }
  if constexpr (tree) {
    return add2(add2(add2(sq[0], sq[4]), add2(sq[1], sq[5])), add2(add2(sq[2], sq[6]), add2(sq[3], sq[7])));
  } else if constexpr (!fma_chain) {
    s = sq[0];  // (+0 + a square is the square)
#pragma unroll
    for (int t = 1; t < D; t++) s = add2(s, sq[t]);
  }
  return s;
}

// One iteration over all problems: assignment + sum updates of changed points.
// Problems of 2 or 8 dimensions (two of the four widths whose rows are held in
// registers; others take fuel's order from memory) whose centres fit the stage, up to
// 8192 and 2048: two centres per packed step, their coordinates interleaved in shared
// memory; with more centres one at a time, from global memory (10 passes of 100 000 x 2,
// k = 8200 9.1 ms, 200 000 x 8, k = 2100 9.7; 29.5 and 35.7 through the general loop).
// WIDE: some problem has 32 dimensions or more (rows of 32 and 64 are held in
// registers): 128 registers per thread; 64 without.  Bound by FP32 issue and, in the first
// passes, by the adds of changed rows: a later pass over 10.3 million rows of 2 or
// 8 dimensions, k to 256: 0.90 -> 0.56 ms against one centre at a time.
template <int KIND, int ORDER, bool WIDE>
__global__ void __launch_bounds__(kItemRows) batched_assign_kernel(
    const BProb* __restrict__ probs, int P, int items_total, const float* __restrict__ X,
    const float* __restrict__ C, int32_t* __restrict__ labels, unsigned long long* __restrict__ limbs,
    int32_t* __restrict__ counts, int32_t* __restrict__ pchg, int first, int64_t work_total, int ccap, f32x2 nz) {
  extern __shared__ __align__(16) unsigned char smem_b[];
  float* cs = reinterpret_cast<float*>(smem_b);                                           // [ccap]
  unsigned long long* agg = reinterpret_cast<unsigned long long*>(cs + ccap);            // [kAggCap]
  int* aggc = reinterpret_cast<int*>(agg + kAggCap);                                      // [256]
  __shared__ int s_chg;
  const int64_t it0 = item_at_cost(probs, P, items_total, (int64_t)((__int128)work_total * blockIdx.x / gridDim.x));
  const int64_t it1 =
      blockIdx.x + 1 == gridDim.x ? items_total
                                  : item_at_cost(probs, P, items_total,
                                                 (int64_t)((__int128)work_total * (blockIdx.x + 1) / gridDim.x));
  int p = -1;
  BProb pr{};
  bool staged = false, paired = false, use_agg = false;
  // flush this CTA's partial sums / counts / change count of problem p
  auto flush = [&]() {
    __syncthreads();
    if (p < 0 || !pr.active) return;
    if (threadIdx.x == 0 && s_chg) atomicAdd(&pchg[p], s_chg);
    if (use_agg) {
      for (int e = threadIdx.x; e < pr.k * pr.d * pr.L; e += blockDim.x)
        if (agg[e]) atomicAdd(limbs + pr.limb_off + e, agg[e]);
      for (int e = threadIdx.x; e < pr.k; e += blockDim.x)
        if (aggc[e]) atomicAdd(&counts[pr.cnt_off + e], aggc[e]);
    }
  };
  for (int64_t item = it0; item < it1; item++) {
    if (p < 0 || (p + 1 < P && item >= probs[p + 1].item_begin)) {
      // next problem: flush the previous one, stage this one's centres
      flush();
      int lo = 0, hi = P;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (probs[mid].item_begin <= item) lo = mid;
        else hi = mid;
      }
      __syncthreads();
      p = lo;
      pr = probs[p];
      staged = ((pr.k + 1) & ~1) * pr.d <= ccap;
      paired = staged && (pr.d == 2 || pr.d == 8);
      use_agg = pr.k * pr.d * pr.L <= kAggCap && pr.k <= 256;
      if (pr.active) {
        if (paired) {
          // centres 2 j and 2 j + 1 interleaved; an odd last one with a NaN, which is
          // never nearer
          for (int e = threadIdx.x; e < ((pr.k + 1) & ~1) * pr.d; e += blockDim.x) {
            const int c = e / pr.d, t = e - c * pr.d;
            cs[((c >> 1) * pr.d + t) * 2 + (c & 1)] = c < pr.k ? C[pr.c_off + e] : __int_as_float(0x7fffffff);
          }
        } else if (staged) {
          for (int e = threadIdx.x; e < pr.k * pr.d; e += blockDim.x) cs[e] = C[pr.c_off + e];
        }
        if (use_agg) {
          for (int e = threadIdx.x; e < pr.k * pr.d * pr.L; e += blockDim.x) agg[e] = 0;
          for (int e = threadIdx.x; e < pr.k; e += blockDim.x) aggc[e] = 0;
        }
      }
      if (threadIdx.x == 0) s_chg = 0;
      __syncthreads();
    }
    if (!pr.active) continue;
    const int64_t i = (item - pr.item_begin) * kItemRows + threadIdx.x;
    const bool live = i < pr.n;
    int best = -1;
    const float* xr = X + pr.x_off + (live ? i : 0) * pr.d;
    const float* cbase = staged ? cs : C + pr.c_off;
    if (live) {
      float bd = 0.0f;
      auto scan = [&](auto dimc) {
        constexpr int DD = decltype(dimc)::value;
        float xv[DD];
#pragma unroll
        for (int t = 0; t < DD; t++) xv[t] = __ldg(xr + t);
        for (int c = 0; c < pr.k; c++) {
          const float* cc = cbase + c * DD;
          // centre values by 16-byte (8-byte for d = 2) loads, one per 4 (2) values
          auto cv = [&](int t) -> float {
            if constexpr (DD % 4 == 0) {
              const float4 v = reinterpret_cast<const float4*>(cc)[t >> 2];
              return (t & 3) == 0 ? v.x : (t & 3) == 1 ? v.y : (t & 3) == 2 ? v.z : v.w;
            } else if constexpr (DD % 2 == 0) {
              const float2 v = reinterpret_cast<const float2*>(cc)[t >> 1];
              return (t & 1) == 0 ? v.x : v.y;
            } else {
              return cc[t];
            }
          };
          const float dv = exact_dist_fn<KIND, ORDER, DD>([&](int t) { return xv[t]; }, cv);
          if (best < 0 || dv < bd) {
            bd = dv;
            best = c;
          }
        }
      };
      auto scan_pairs = [&](auto dimc) {
        constexpr int DD = decltype(dimc)::value;
        f32x2 x[DD];
#pragma unroll
        for (int t = 0; t < DD; t++) {
          const float v = __ldg(xr + t);
          x[t] = pack2(v, v);
        }
        const f32x2* cp = reinterpret_cast<const f32x2*>(cs);
        float d0, d1;
        unpack2(exact_dist_pair<KIND, ORDER, DD>(x, cp, nz), d0, d1);
        bd = d0;  // the first centre, whatever its distance
        best = 0;
#pragma unroll 2
        for (int c = 0; c < pr.k; c += 2, cp += DD) {
          unpack2(exact_dist_pair<KIND, ORDER, DD>(x, cp, nz), d0, d1);
          if (d0 < bd) {
            bd = d0;
            best = c;
          }
          if (d1 < bd) {
            bd = d1;
            best = c + 1;
          }
        }
      };
      if (paired && pr.d == 2) scan_pairs(Dim<2>{});
      else if (paired) scan_pairs(Dim<8>{});
      else if (WIDE && pr.d == 32) scan(Dim<32>{});
      else if (WIDE && pr.d == 64) scan(Dim<64>{});
      else if (pr.d == 2) scan(Dim<2>{});  // (centres that are not staged)
      else if (pr.d == 8) scan(Dim<8>{});
      else {
          for (int c = 0; c < pr.k; c++) {
            const float dv = exact_dist_scalar<KIND, ORDER>(xr, C + pr.c_off + (int64_t)c * pr.d, pr.d);
            if (best < 0 || dv < bd) {
              bd = dv;
              best = c;
            }
          }
      }
    }
    const int old = live ? (first ? -1 : labels[pr.lab_off + i]) : -1;
    if (live && best != old) {
      labels[pr.lab_off + i] = best;
      if (!first) atomicAdd(&s_chg, 1);
      unsigned long long* base = use_agg ? agg : limbs + pr.limb_off;
      if (use_agg) {
        atomicAdd(&aggc[best], 1);
        if (old >= 0) atomicAdd(&aggc[old], -1);
      } else {
        atomicAdd(&counts[pr.cnt_off + best], 1);
        if (old >= 0) atomicAdd(&counts[pr.cnt_off + old], -1);
      }
      for (int t = 0; t < pr.d; t++) {
        const float xv = __ldg(xr + t);
        add_coord(base + ((int64_t)best * pr.d + t) * pr.L, xv, pr.e_lo, pr.L, false);
        if (old >= 0) add_coord(base + ((int64_t)old * pr.d + t) * pr.L, xv, pr.e_lo, pr.L, true);
      }
    }
  }
  flush();
}

// Centres from the sums: canonicalise each coordinate's counters (carry
// propagation modulo 2^(32L)) and round the exact mean; empty clusters keep
// their centre.  Also records per-problem convergence: conv[p] = the first
// iteration (counting the initial pass as 1) with no changed label.
__global__ void batched_mean_kernel(const BProb* __restrict__ probs, int P, const int64_t* __restrict__ kd_begin,
                                    int64_t kd_total, unsigned long long* __restrict__ limbs,
                                    const int32_t* __restrict__ counts, float* __restrict__ C, int write_centers) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < kd_total;
       e += (int64_t)gridDim.x * blockDim.x) {
    int lo = 0, hi = P;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (kd_begin[mid] <= e) lo = mid;
      else hi = mid;
    }
    while (lo + 1 < P && kd_begin[lo + 1] <= e) lo++;
    const BProb& pr = probs[lo];
    if (!pr.active) continue;
    const int64_t local = e - kd_begin[lo];
    const int L = pr.L;
    unsigned long long* lp = limbs + pr.limb_off + local * L;
    unsigned __int128 tot = 0;
    for (int l = 0; l < L; l++) tot += (unsigned __int128)lp[l] << (32 * l);
    if (L < 4) tot &= (((unsigned __int128)1) << (32 * (L & 3))) - 1;
    for (int l = 0; l < L; l++) lp[l] = (unsigned long long)((tot >> (32 * l)) & 0xffffffffu);
    const int j = (int)(local / pr.d);
    const int cnt = counts[pr.cnt_off + j];
    if (cnt <= 0 || !write_centers) continue;
    const bool neg = (tot >> (32 * L - 1)) & 1;
    unsigned __int128 mag = tot;
    if (neg) {
      if (L < 4) {
        mag = (((unsigned __int128)1) << (32 * (L & 3))) - tot;
        mag &= (((unsigned __int128)1) << (32 * (L & 3))) - 1;
      } else {
        mag = (unsigned __int128)0 - tot;
      }
    }
    const float v = mag == 0 ? 0.0f : rn_ratio_f32(mag, (unsigned long long)cnt, pr.e_lo);
    C[pr.c_off + local] = neg ? -v : v;
  }
}

// After each pass: record the iteration and convergence, reset the change
// counters.  iter[0] counts passes (the initial one is 1).
__global__ void batched_step_kernel(int P, int32_t* __restrict__ pchg, int32_t* __restrict__ conv,
                                    int32_t* __restrict__ last_chg, int32_t* __restrict__ iter,
                                    int* __restrict__ und_n) {
  const int it = iter[0] + 1;
  for (int p = threadIdx.x; p < P; p += blockDim.x) {
    const int c = pchg[p];
    last_chg[p] = c;
    if (it > 1 && c == 0 && conv[p] == 0) conv[p] = it;
    pchg[p] = 0;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    iter[0] = it;
    *und_n = 0;
  }
}

// Labels as the caller's 64-bit integers.
constexpr int64_t kHostLabels = 16384;  // a problem, and that many more: fewer are widened on the host
__global__ void widen_labels_kernel(const int32_t* __restrict__ labels, int64_t count, int64_t* __restrict__ out) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < count) out[e] = labels[e];
}

// Sum of squared distances to the final centres, per problem (near-FP64: SqDiffAcc
// over the d terms that a thread takes of its item, FP64 across threads).  The
// block reads its item's rows as one run: 512 problems, 20 million rows, 2.60 -> 0.95 ms
// (one row per thread before).  Bound by the accumulator's FP32 steps.
__global__ void batched_inertia_kernel(const BProb* __restrict__ probs, int P, int items_total,
                                       const float* __restrict__ X, const float* __restrict__ C,
                                       const int32_t* __restrict__ labels, double* __restrict__ inertia) {
  for (int64_t item = blockIdx.x; item < items_total; item += gridDim.x) {
    int lo = 0, hi = P;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (probs[mid].all_item_begin <= item) lo = mid;
      else hi = mid;
    }
    const BProb& pr = probs[lo];
    const int64_t i0 = (item - pr.all_item_begin) * kItemRows;
    double s = 0.0;
    if (pr.active) {
      const int rows = (int)min((int64_t)kItemRows, pr.n - i0);
      const float* x = X + pr.x_off + i0 * pr.d;
      const float* c = C + pr.c_off;
      const int32_t* lab = labels + pr.lab_off + i0;
      SqDiffAcc sa;
      int terms = 0;
      if (pr.d > 4096) {  // (32-bit element numbers below)
        for (int r = 0; r < rows; r++)
          for (int q = threadIdx.x; q < pr.d; q += kItemRows) {
            sa.add(__ldg(x + (int64_t)r * pr.d + q), __ldg(c + (int64_t)lab[r] * pr.d + q));
            if ((++terms & 31) == 0) sa.renorm();
          }
      } else if ((pr.d & 3) == 0) {  // 16 bytes per step (x_off and c_off are multiples of 4)
        const unsigned cpr = (unsigned)pr.d >> 2;
        for (unsigned e = threadIdx.x; e < rows * cpr; e += kItemRows) {
          const unsigned r = e / cpr, q = e - r * cpr;
          const float4 xv = __ldg(reinterpret_cast<const float4*>(x) + e);
          const float4 cv = __ldg(reinterpret_cast<const float4*>(c + (int64_t)lab[r] * pr.d) + q);
          sa.add(xv.x, cv.x);
          sa.add(xv.y, cv.y);
          sa.add(xv.z, cv.z);
          sa.add(xv.w, cv.w);
          if ((++terms & 7) == 0) sa.renorm();
        }
      } else {
        for (unsigned e = threadIdx.x; e < (unsigned)rows * pr.d; e += kItemRows) {
          const unsigned r = e / (unsigned)pr.d, q = e - r * pr.d;
          sa.add(__ldg(x + e), __ldg(c + (int64_t)lab[r] * pr.d + q));
          if ((++terms & 31) == 0) sa.renorm();
        }
      }
      s = sa.value();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0 && s != 0.0) atomicAdd(&inertia[lo], s);
  }
}

// ---------------------------------------------------------------------------
// Tensor-core tier for problems with 32 <= d <= 64 and k <= 256: each
// 128-row item of a problem is screened with split-BF16 products (x_hi c_hi +
// x_hi c_lo + x_lo c_hi, one 64-wide K chunk, FP32 accumulators in TMEM)
// against the problem's centres staged in shared memory; a row is decided
// when every other centre's lower bound exceeds the best centre's upper bound
// (the error bound of the single-problem screen), otherwise its candidate
// centres are re-scored with fuel's exact f32 arithmetic.  Labels are
// therefore identical to the CUDA-core tier.
// ---------------------------------------------------------------------------
constexpr int kTcRows = 128;

struct BTcArgs {
  const int32_t* tcp;         // problem ids served here
  const int32_t* item_begin;  // [ntc + 1] first 128-row item of each
  const int64_t* cta_begin;   // [grid + 1] first item of each CTA (ranges of equal estimated cost)
  int ntc, items;
  float alpha;                // operand + accumulation error per |x||c|
  int* status;
  unsigned long long* undecided;  // rows re-scored exactly (count over the call)
  int32_t* und_p;                 // this pass's undecided rows: problem, row
  int32_t* und_i;
  uint32_t* und_m;                // and their candidate centres: und_w bit words per row
  int und_w;
  int* und_n;
  // passes after the first: changed rows (row, new and old global cluster)
  // listed for the bucketed sums while the list has room, and the per-key
  // counts (key 2 gc: rows entering cluster gc, 2 gc + 1: rows leaving it)
  int32_t *chg_row, *chg_new, *chg_old, *hist;
  int* chg_n;
  int chg_cap;
};


// |v|^2 in FP32 as 8 interleaved chains + a 3-level tree (error <= (ceil(d/8) + 3) u |v|^2).
template <class F>
__device__ __forceinline__ float norm2_blocked(F v, int d) {
  float p[8];
#pragma unroll
  for (int l = 0; l < 8; l++) p[l] = 0.0f;
  for (int e = 0; e < d; e += 8) {
#pragma unroll
    for (int l = 0; l < 8; l++)
      if (e + l < d) {
        const float x = v(e + l);
        p[l] = fmaf(x, x, p[l]);
      }
  }
  return ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7]));
}

// Warp-specialised persistent screen over a list of 128-row items:
//   warps 0-7   loaders: convert the current item's rows from one of two staging
//               buffers into BF16 hi / lo (SW128) and |x|^2 into one of two A
//               buffers; on a problem change they stage the problem's centres
//               (hi / lo, SW128), norms and parameters
//   warp 8      TMEM owner; one lane issues the three products per K step
//               (x_hi c_hi + x_hi c_lo + x_lo c_hi) into one of two 256-column
//               accumulators and commits, and copies the rows of the item after
//               next (contiguous in memory) into the staging buffer just converted
//               with one bulk copy
//   warps 9-16  epilogue, four warps per accumulator: screen, labels, sums of
//               changed rows
// so the row copy of item t+1, its conversion, the MMAs and the epilogue of
// item t overlap.  Barriers: stage_full[s] (bulk copy bytes), a_full[b] (eight
// loader warps), acc_full[b] (the MMA commit: A[b] is free again),
// item_done[b] (four epilogue warps: TMEM[b] is free again).  An item's
// parameters and row norms have one of four places: item t's are written after
// the MMAs of item t-2, which were issued after item t-4 retired.  On a
// problem change the loaders first wait for both previous items to retire, so
// the single centre buffer is never replaced under a reader.  Every wait is
// bounded.
//
// Bound by the latency of 17 warps that each depend on few others (1.5 instructions
// a cycle, tensor pipe 4 %).  Screens of 76 900 items (9.8 million rows of 32 or 64
// dimensions, k to 256): 2.38 ms with one group of four epilogue warps that branched
// per column (123 cycles a column) and four loader warps with one row per thread;
// 1.29 now.  On the way: branch-free passes and two groups 1.9, packed steps and the
// problem looked up at a change only 1.75, CTA ranges by the new costs 1.29.  The
// issuer's role on an epilogue warp (16 warps) spilled and was 15 % slower, as was
// holding the screen values of up to 32 columns between the passes (5 %).
constexpr int kTcThreads = 544;
constexpr int kTcLoaders = 256;
constexpr uint32_t kTcA = 32768;   // one A buffer: hi 16 KB + lo 16 KB
constexpr uint32_t kTcB = 65536;   // the centre buffer: hi 32 KB + lo 32 KB (256 centres)
constexpr uint32_t kTcS = 32768;   // one staging buffer: 128 rows x 64 f32
constexpr uint32_t kTcOffB = 2 * kTcA, kTcOffS = kTcOffB + kTcB, kTcSmall = kTcOffS + 2 * kTcS;

struct ItemMeta {  // one item's problem parameters, written by the loaders
  int64_t n, lab_off, limb_off, x_off;
  int32_t p, i0, kp, d, k, L, e_lo, cnt_off;
};

// + norms (2 x 256 floats), maxima (4), row norms (4 x 128), metadata (4), 9 mbarriers,
// TMEM address and abort word, 1 KB alignment
constexpr size_t kTcSmem =
    1024 + kTcSmall + 4 * 2 * 256 + 4 * 4 + 4 * 4 * 128 + sizeof(ItemMeta) * 4 + 8 * 9 + 8 + 64;

// Every loader thread (warps 0-7, named barrier 1) learns whether all of
// them passed `v`.
__device__ __forceinline__ bool loaders_all(bool v) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 q, %1, 0;\n bar.red.and.pred p, 1, 256, q;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(r)
      : "r"((uint32_t)v)
      : "memory");
  return r != 0;
}

template <int KIND, int ORDER>
__global__ void __launch_bounds__(kTcThreads, 1) batched_tc_assign_kernel(
    const BProb* __restrict__ probs, BTcArgs ta, const float* __restrict__ X, const float* __restrict__ C,
    int32_t* __restrict__ labels, unsigned long long* __restrict__ limbs, int32_t* __restrict__ counts,
    int32_t* __restrict__ pchg, int first) {
  extern __shared__ __align__(1024) unsigned char smem_t[];
  unsigned char* base =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_t) + 1023) & ~(uintptr_t)1023);
  unsigned char* sBh = base + kTcOffB;
  unsigned char* sBl = sBh + kTcB / 2;
  float* cn2s = reinterpret_cast<float*>(base + kTcSmall);  // [256] |c|^2 of the staged problem
  float* cns = cn2s + 256;                                   // [256] |c|
  float* cmaxs = cns + 256;                                  // max |c|^2, max |c| (bits)
  float* xn2s = cmaxs + 4;                                   // [4 items][128] |x|^2
  ItemMeta* meta = reinterpret_cast<ItemMeta*>(xn2s + 4 * 128);
  uint64_t* stage_full = reinterpret_cast<uint64_t*>(meta + 4);
  uint64_t* a_full = stage_full + 2;
  uint64_t* acc_full = a_full + 2;
  uint64_t* item_done = acc_full + 2;
  uint64_t* fin = item_done + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(fin + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int b = 0; b < 2; b++) {
      tcx::mbar_init(&stage_full[b], 1);
      tcx::mbar_init(&a_full[b], kTcLoaders / 32);  // one arrival per warp
      tcx::mbar_init(&acc_full[b], 1);
      tcx::mbar_init(&item_done[b], kTcRows / 32);
    }
    tcx::mbar_init(fin, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tcx::smem_u32(tmem_holder)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcx::tc_fence_before();
  __syncthreads();
  tcx::tc_fence_after();
  const uint32_t tmem = *tmem_holder;
  // this CTA's items: a contiguous range of equal estimated cost
  const int64_t it0 = ta.cta_begin[blockIdx.x], it1 = ta.cta_begin[blockIdx.x + 1];
  const int64_t nlt = it1 - it0;
  auto problem_of = [&](int64_t item, int q0) {
    int q = q0 < 0 ? 0 : q0;
    if (q0 < 0 || item >= ta.item_begin[q + 1]) {
      int lo = 0, hi = ta.ntc;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (ta.item_begin[mid] <= item) lo = mid;
        else hi = mid;
      }
      q = lo;
    }
    return q;
  };
  // bytes of an item's rows that one bulk copy brings in (0: the direct-load path)
  auto bulk_bytes = [&](const BProb& pr, int64_t i0) -> uint32_t {
    if (!pr.active || (pr.d & 3) != 0 || (pr.x_off & 3) != 0 || pr.d > 64) return 0u;
    const int64_t rows = min((int64_t)kTcRows, pr.n - i0);
    return (uint32_t)(rows * pr.d * 4);
  };

  if (warp < 8) {
    // ---- loaders ----------------------------------------------------------
    int q = -1;
    BProb pr;                            // the problem, looked up at a change only (three dependent loads)
    int64_t q_begin = 0, q_end = 0;      // its items
    int p = 0, kp = 0;
    for (int64_t lt = 0; lt < nlt; lt++) {
      const int b = (int)(lt & 1), slot = (int)(lt & 3);
      const uint32_t ph = (uint32_t)((lt >> 1) & 1);
      // the products of item lt-2 are made: its A buffer is free, and item lt-4
      // has retired.  The loaders leave together (a vote on their named barrier),
      // so the barriers below never wait for a loader that left.
      bool ok = !*abort_flag && tcx::mbar_wait(&acc_full[b], ph ^ 1u, abort_flag);
      if (!ok && !*abort_flag) atomicOr(ta.status, DEV_TIMEOUT);
      if (!loaders_all(ok)) {
        *abort_flag = 1;
        break;
      }
      const int64_t item = it0 + lt;
      if (item >= q_end) {
        q = problem_of(item, q);
        p = ta.tcp[q];
        pr = probs[p];
        q_begin = ta.item_begin[q];
        q_end = ta.item_begin[q + 1];
        kp = (pr.k + 15) & ~15;
        // the previous items must retire before their centres go (a wait by parity is
        // for the barrier's current phase: item lt-1's products come after item lt-3
        // retired)
        if (lt > 0) {
          const uint32_t ph1 = (uint32_t)(((lt - 1) >> 1) & 1);
          ok = !*abort_flag && tcx::mbar_wait(&acc_full[b ^ 1], ph1, abort_flag) &&
               tcx::mbar_wait(&item_done[b ^ 1], ph1, abort_flag) &&
               tcx::mbar_wait(&item_done[b], ph ^ 1u, abort_flag);
          if (!ok && !*abort_flag) atomicOr(ta.status, DEV_TIMEOUT);
          if (!loaders_all(ok)) {
            *abort_flag = 1;
            break;
          }
        }
        for (int e = tid; e < kp * 8; e += kTcLoaders) {
          const int j = e >> 3, ch = e & 7;
          uint32_t hw[4], lw[4];
#pragma unroll
          for (int l = 0; l < 8; l += 2) {
            const int t0 = 8 * ch + l;
            const float c0 = (j < pr.k && t0 < pr.d) ? C[pr.c_off + (int64_t)j * pr.d + t0] : 0.0f;
            const float c1 = (j < pr.k && t0 + 1 < pr.d) ? C[pr.c_off + (int64_t)j * pr.d + t0 + 1] : 0.0f;
            const __nv_bfloat162 h = __floats2bfloat162_rn(c0, c1);
            const float2 hf = __bfloat1622float2(h);
            const __nv_bfloat162 lo = __floats2bfloat162_rn(c0 - hf.x, c1 - hf.y);
            hw[l / 2] = *reinterpret_cast<const uint32_t*>(&h);
            lw[l / 2] = *reinterpret_cast<const uint32_t*>(&lo);
          }
          const uint32_t off = (uint32_t)j * 128u + ((uint32_t)(ch ^ (j & 7)) << 4);
          *reinterpret_cast<uint4*>(sBh + off) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
          *reinterpret_cast<uint4*>(sBl + off) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
        }
        if (tid == 0) cmaxs[0] = cmaxs[1] = 0.0f;
        asm volatile("bar.sync 1, %0;" ::"n"(kTcLoaders) : "memory");  // loaders only
        float m2 = 0.0f;
        for (int j = tid; j < 256; j += kTcLoaders) {
          float v = 0.0f;
          if (j < pr.k) {
            const float* cj = C + pr.c_off + (int64_t)j * pr.d;
            v = norm2_blocked([&](int t) { return cj[t]; }, pr.d);
          }
          // +inf past k: the epilogue reads them four at a time, and a padding
          // column's screen value is then +inf (never the minimum)
          cn2s[j] = j < pr.k ? v : __int_as_float(0x7f800000);
          cns[j] = sqrtf(v);
          m2 = fmaxf(m2, v);
        }
        // non-negative floats order like their bit patterns
        atomicMax(reinterpret_cast<int*>(cmaxs), __float_as_int(m2));
        atomicMax(reinterpret_cast<int*>(cmaxs) + 1, __float_as_int(sqrtf(m2)));
      }
      const int64_t i0 = (item - q_begin) * kTcRows;
      // this item's rows -> BF16 hi / lo (zero padded), FP32 norms: a thread takes
      // chunks of 8 values, the 4 (d <= 32) or 8 chunks of a row on neighbouring
      // lanes, so a warp reads and writes shared memory in runs
      unsigned char* sAh = base + (uint32_t)b * kTcA;
      unsigned char* sAl = sAh + kTcA / 2;
      ok = !*abort_flag && tcx::mbar_wait(&stage_full[b], ph, abort_flag);
      if (!ok && !*abort_flag) atomicOr(ta.status, DEV_TIMEOUT);
      if (!loaders_all(ok)) {
        *abort_flag = 1;
        break;
      }
      const bool bulk = bulk_bytes(pr, i0) != 0;
      const float* stage = reinterpret_cast<const float*>(base + kTcOffS + (uint32_t)b * kTcS);
      const int lpr = pr.d <= 32 ? 4 : 8;  // lanes per row
      const int j = tid & (lpr - 1);
      auto convert = [&](int row, const float (&x)[8]) {
        uint32_t hw[4], lw[4];
        f32x2 s = 0;
#pragma unroll
        for (int l = 0; l < 8; l += 2) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(x[l], x[l + 1]);
          const float2 hf = __bfloat1622float2(h);
          const f32x2 xx = pack2(x[l], x[l + 1]);
          float2 rest;
          unpack2(fma2(pack2(hf.x, hf.y), kNegOne2, xx), rest.x, rest.y);  // x - hi
          const __nv_bfloat162 lo = __floats2bfloat162_rn(rest.x, rest.y);
          hw[l / 2] = *reinterpret_cast<const uint32_t*>(&h);
          lw[l / 2] = *reinterpret_cast<const uint32_t*>(&lo);
          s = fma2(xx, xx, s);
        }
        const uint32_t off = (uint32_t)row * 128u + ((uint32_t)(j ^ (row & 7)) << 4);
        *reinterpret_cast<uint4*>(sAh + off) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
        *reinterpret_cast<uint4*>(sAl + off) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
        // the norm: two chains of 4 and a tree over the row's lanes (7 roundings on a
        // path for d = 32, 8 above: within (ceil(d/8) + 3) u |x|^2)
        float v, v1;
        unpack2(s, v, v1);
        v += v1;
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        if (lpr == 8) v += __shfl_xor_sync(0xffffffffu, v, 4);
        if (j == 0) xn2s[slot * 128 + row] = v;
      };
      if (bulk && pr.d == 8 * lpr) {  // whole chunks of staged rows (past n: unread)
        const float* src = stage + 8 * j;
        for (int row = tid / lpr; row < kTcRows; row += 2 * (kTcLoaders / lpr)) {
          float x[2][8];
#pragma unroll
          for (int u = 0; u < 2; u++) {
            const float* s = src + (row + u * (kTcLoaders / lpr)) * pr.d;
            const float4 a4 = *reinterpret_cast<const float4*>(s);
            const float4 b4 = *reinterpret_cast<const float4*>(s + 4);
            x[u][0] = a4.x, x[u][1] = a4.y, x[u][2] = a4.z, x[u][3] = a4.w;
            x[u][4] = b4.x, x[u][5] = b4.y, x[u][6] = b4.z, x[u][7] = b4.w;
          }
#pragma unroll
          for (int u = 0; u < 2; u++) convert(row + u * (kTcLoaders / lpr), x[u]);
        }
      } else {
#pragma unroll 1
        for (int row = tid / lpr; row < kTcRows; row += kTcLoaders / lpr) {
          const bool live = pr.active && i0 + row < pr.n;
          const float* xr = X + pr.x_off + (live ? i0 + row : 0) * pr.d;
          float x[8];
#pragma unroll
          for (int l = 0; l < 8; l++) {
            const int t = 8 * j + l;
            x[l] = !live || t >= pr.d ? 0.0f : bulk ? stage[row * pr.d + t] : __ldg(xr + t);
          }
          convert(row, x);
        }
      }
      if (tid == 0) {
        ItemMeta m;
        m.n = pr.n;
        m.lab_off = pr.lab_off;
        m.limb_off = pr.limb_off;
        m.x_off = pr.x_off;
        m.p = p;
        m.i0 = (int32_t)i0;
        m.kp = pr.active ? kp : 0;
        m.d = pr.d;
        m.k = pr.k;
        m.L = pr.L;
        m.e_lo = pr.e_lo;
        m.cnt_off = pr.cnt_off;
        meta[slot] = m;
      }
      // generic-proxy smem writes -> visible to the tensor core's async proxy
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) tcx::mbar_arrive(&a_full[b]);
    }
  } else if (warp == 8) {
    // ---- row copies and MMAs, one lane -----------------------------------------
    if (lane == 0) {
      int issued[2] = {0, 0};  // copies (or plain arrivals) armed per staging buffer
      BProb pr;
      int64_t q_begin = 0, q_end = 0;
      int q = -1;
      // item lt's rows into staging buffer lt & 1
      auto fetch = [&](int64_t lt) {
        const int s = (int)(lt & 1);
        issued[s]++;
        if (it0 + lt >= q_end) {
          q = problem_of(it0 + lt, q);
          pr = probs[ta.tcp[q]];
          q_begin = ta.item_begin[q];
          q_end = ta.item_begin[q + 1];
        }
        const int64_t i0 = (it0 + lt - q_begin) * kTcRows;
        const uint32_t by = bulk_bytes(pr, i0);
        if (by) {
          tcx::mbar_expect_tx(&stage_full[s], by);
          tcx::bulk_load(base + kTcOffS + (uint32_t)s * kTcS, X + pr.x_off + i0 * pr.d, by, &stage_full[s]);
        } else {
          tcx::mbar_arrive(&stage_full[s]);
        }
      };
      for (int64_t lt = 0; lt < 2 && lt < nlt; lt++) fetch(lt);
      for (int64_t lt = 0; lt < nlt && !*abort_flag; lt++) {
        const int b = (int)(lt & 1);
        const uint32_t ph = (uint32_t)((lt >> 1) & 1);
        if (!tcx::mbar_wait(&a_full[b], ph, abort_flag) ||
            !tcx::mbar_wait(&item_done[b], ph ^ 1u, abort_flag)) {
          if (!*abort_flag) atomicOr(ta.status, DEV_TIMEOUT);
          *abort_flag = 1;
          break;
        }
        tcx::tc_fence_after();
        const int kp = meta[lt & 3].kp;
        if (kp > 0) {
          unsigned char* sAh = base + (uint32_t)b * kTcA;
          const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kp >> 3) << 17) |
                                 ((uint32_t)(kTcRows >> 4) << 24);
          const uint64_t ah = tcx::smem_desc_sw128(tcx::smem_u32(sAh));
          const uint64_t al = tcx::smem_desc_sw128(tcx::smem_u32(sAh + kTcA / 2));
          const uint64_t bh = tcx::smem_desc_sw128(tcx::smem_u32(sBh));
          const uint64_t bl = tcx::smem_desc_sw128(tcx::smem_u32(sBl));
          const uint32_t d_tmem = tmem + (uint32_t)b * 256u;
          // K steps of 16 that hold data (the zero columns past d add nothing)
          const int nks = (meta[lt & 3].d + 15) >> 4;
#pragma unroll
          for (int kk = 0; kk < 4; kk++)
            if (kk < nks) tcx::umma_bf16(d_tmem, ah + 2 * kk, bh + 2 * kk, idesc, kk ? 1u : 0u);
#pragma unroll
          for (int kk = 0; kk < 4; kk++)
            if (kk < nks) tcx::umma_bf16(d_tmem, ah + 2 * kk, bl + 2 * kk, idesc, 1u);
#pragma unroll
          for (int kk = 0; kk < 4; kk++)
            if (kk < nks) tcx::umma_bf16(d_tmem, al + 2 * kk, bh + 2 * kk, idesc, 1u);
        }
        tcx::umma_commit(&acc_full[b]);
        // the rows of this staging buffer have been converted (a_full)
        if (lt + 2 < nlt) fetch(lt + 2);
      }
      // every MMA issued here has completed before TMEM is freed
      tcx::umma_commit(fin);
      volatile int never = 0;
      if (!tcx::mbar_wait(fin, 0, &never)) atomicOr(ta.status, DEV_TIMEOUT);
      // a copy still in flight must not outlive the CTA: the last one armed on
      // each staging buffer lands before the exit (also after an abort)
      for (int s = 0; s < 2; s++)
        if (issued[s] > 0 && !tcx::mbar_wait(&stage_full[s], (uint32_t)((issued[s] - 1) & 1), &never))
          atomicOr(ta.status, DEV_TIMEOUT);
    }
  } else {
    // ---- epilogue: warp w reads TMEM lanes 32 * (w % 4) .. +32; warps 9-12 take the
    // items of buffer 0, warps 13-16 those of buffer 1 -------------------------
    const int g = warp & 3;
    const int row = g * 32 + lane;
    const double u24 = 5.9604644775390625e-08;
    const int b = (warp - 9) >> 2;
    int last_d = -1;
    float beta = 0.0f, gamma = 0.0f;  // error terms of a problem's d
    for (int64_t lt = b; lt < nlt; lt += 2) {
      const uint32_t ph = (uint32_t)((lt >> 1) & 1);
      bool ok = !*abort_flag && tcx::mbar_wait(&acc_full[b], ph, abort_flag);
      if (!ok) {
        if (!*abort_flag) atomicOr(ta.status, DEV_TIMEOUT);
        *abort_flag = 1;
      }
      if (!__all_sync(0xffffffffu, ok)) break;  // warp-uniform exit
      tcx::tc_fence_after();
      const int slot = (int)(lt & 3);
      const ItemMeta mt = meta[slot];
      const int kp = mt.kp;
      const int64_t i = (int64_t)mt.i0 + row;
      const bool live = kp > 0 && i < mt.n;
      // the row's current label, fetched while the screen runs
      const int old = live ? (first ? -1 : labels[mt.lab_off + i]) : -1;
      const float cmax0 = cmaxs[0], cmax1 = cmaxs[1];
      const float nx = xn2s[slot * 128 + row];
      if (mt.d != last_d) {
        last_d = mt.d;
        beta = (float)(((mt.d + 7) / 8 + 3 + 9) * u24 * 1.01);
        gamma = (float)((mt.d + 4) * u24 * 1.01);
      }
      const uint32_t taddr = tmem + ((uint32_t)(g * 32) << 16) + (uint32_t)b * 256u;
      const float xl = sqrtf(nx);
      float best = __int_as_float(0x7f800000);
      int bj = 0;
      bool undecided = false;
      // candidate centres of an undecided row: 32-column words (bit w of
      // cm_set: word w holds candidates)
      uint32_t cmask[8];
      uint32_t cm_set = 0;
      if (kp > 0) {
        // Screen over the TMEM columns, 32 per wait, without branches on a column's
        // value.  Pass 1: the smallest screen value (padding columns past k read
        // +inf norms).  The best centre's upper bound hi_b takes the problem's norm
        // maxima (at least its own error term), so it needs no column index, and no
        // column above T reaches it with the largest error of the problem.  Pass 2:
        // the columns up to T.  A row with one such column is decided.  Pass 3, for
        // warps with another row: the first column holding the smallest value is the
        // best centre (first index wins ties, as in a scan), and every other column
        // whose own lower bound reaches the bound is a candidate.
        const f32x2 nx2 = pack2(nx, nx), m2 = pack2(-2.0f, -2.0f);
        uint32_t r[2][16];
        auto columns = [&](int c0) {
#pragma unroll
          for (int h = 0; h < 2; h++)
            if (c0 + 16 * h < kp) tcx::tmem_ld16_nowait(taddr + c0 + 16 * h, r[h]);
          tcx::tmem_ld_wait();
#pragma unroll
          for (int h = 0; h < 2; h++) tcx::tmem_regs_ready(r[h]);
        };
        // screen values fma(-2, dot, |x|^2 + |c|^2) of columns c0 + 16 h + 4 v ..
        auto screen4 = [&](int c, const uint32_t* q, float (&dt)[4], float (&cc)[4]) {
          const float4 c4 = *reinterpret_cast<const float4*>(cn2s + c);
          cc[0] = c4.x, cc[1] = c4.y, cc[2] = c4.z, cc[3] = c4.w;
#pragma unroll
          for (int u = 0; u < 4; u += 2)
            unpack2(fma2(m2, pack2(__uint_as_float(q[u]), __uint_as_float(q[u + 1])),
                         add2(nx2, pack2(cc[u], cc[u + 1]))),
                    dt[u], dt[u + 1]);
        };
        float b4[4] = {best, best, best, best};
        for (int c0 = 0; c0 < kp; c0 += 32) {
          columns(c0);
#pragma unroll
          for (int h = 0; h < 2; h++) {
            if (c0 + 16 * h >= kp) break;
#pragma unroll
            for (int v = 0; v < 4; v++) {
              float dt[4], cc[4];
              screen4(c0 + 16 * h + 4 * v, r[h] + 4 * v, dt, cc);
#pragma unroll
              for (int u = 0; u < 4; u++) b4[u] = fminf(b4[u], dt[u]);
            }
          }
        }
        best = fminf(fminf(b4[0], b4[1]), fminf(b4[2], b4[3]));
        const float amax = (ta.alpha * xl * cmax1 + beta * (nx + cmax0)) * (1.0f + gamma);
        const float hi_b = best + amax + gamma * fabsf(best);
        const float T0 = (hi_b + amax) * (1.0f + 2.0f * gamma) * (1.0f + 9.5367431640625e-07f);
        const float T = T0 > 0.0f ? T0 : __int_as_float(0x7f800000);
        // One instruction per column: the sign of dt - T', T' the next value above T,
        // shifted into a word.  Finite T: every norm, screen value and bound of the
        // row is finite (T covers the largest of each).
        const bool finite = T < __int_as_float(0x7f800000);
        const float nt = -__int_as_float(__float_as_int(T) + (finite ? 1 : 0));
        const f32x2 nt2 = pack2(nt, nt);
        int near = 0;  // columns up to T
        for (int c0 = 0; c0 < kp; c0 += 32) {
          uint32_t bits = 0;  // the last column at bit 0
          columns(c0);
#pragma unroll
          for (int h = 0; h < 2; h++) {
            if (c0 + 16 * h >= kp) break;
#pragma unroll
            for (int v = 0; v < 4; v++) {
              float dt[4], cc[4];
              screen4(c0 + 16 * h + 4 * v, r[h] + 4 * v, dt, cc);
#pragma unroll
              for (int u = 0; u < 4; u += 2) {
                float e0, e1;
                unpack2(add2(pack2(dt[u], dt[u + 1]), nt2), e0, e1);
                bits = __funnelshift_l(__float_as_uint(e0), bits, 1);
                bits = __funnelshift_l(__float_as_uint(e1), bits, 1);
              }
            }
          }
          near += __popc(bits);
          if (bits) bj = min(c0 + 32, kp) - __ffs(bits);
        }
        bool found = finite && near == 1;
        if (__any_sync(0xffffffffu, live && !found)) {
          bj = 0;
          found = false;
          for (int c0 = 0; c0 < kp; c0 += 32) {
            uint32_t bits = 0, eq = 0;
            columns(c0);
#pragma unroll
            for (int h = 0; h < 2; h++) {
              if (c0 + 16 * h >= kp) break;
#pragma unroll
              for (int v = 0; v < 4; v++) {
                float dt[4], cc[4];
                screen4(c0 + 16 * h + 4 * v, r[h] + 4 * v, dt, cc);
                const float4 s4 = *reinterpret_cast<const float4*>(cns + c0 + 16 * h + 4 * v);
                const float ss[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                for (int u = 0; u < 4; u++) {
                  const float e = (ta.alpha * xl * ss[u] + beta * (nx + cc[u])) * (1.0f + gamma) + gamma * fabsf(dt[u]);
                  const uint32_t bit = 1u << (16 * h + 4 * v + u);
                  eq |= dt[u] == best ? bit : 0u;
                  bits |= !(dt[u] > T) && !(dt[u] - e > hi_b) ? bit : 0u;
                }
              }
            }
            if (!found && eq) {
              found = true;
              bj = c0 + __ffs(eq) - 1;
              bits &= ~(eq & (0u - eq));
            }
            if (bits) {
              undecided = true;
              cmask[c0 >> 5] = bits;
              cm_set |= 1u << (c0 >> 5);
            }
          }
        }
        // no column equal to the minimum (a NaN screen value): the re-score
        // decides among every centre
        if (!found) {
          undecided = true;
          for (int w = 0; w < (kp + 31) / 32; w++) cmask[w] = 0xffffffffu;
          cm_set = (1u << ((kp + 31) / 32)) - 1u;
        }
      }
      // the item's accumulator, tile and parameters are no longer read
      tcx::tc_fence_before();
      __syncwarp();
      if (lane == 0) tcx::mbar_arrive(&item_done[b]);
      if (kp == 0) continue;
      const int p = mt.p;
      const int lab = bj;
      const bool chg = live && !undecided && lab != old;
      const unsigned um = __ballot_sync(0xffffffffu, live && undecided);
      const unsigned cm = __ballot_sync(0xffffffffu, chg);
      // places on the undecided and the change list, both asked for before either
      // answer is used
      int u_at = 0, c_at = 0;
      if (lane == 0) {
        if (um) u_at = atomicAdd(ta.und_n, __popc(um));
        if (!first && cm) c_at = atomicAdd(ta.chg_n, __popc(cm));
        if (um) atomicAdd(ta.undecided, (unsigned long long)__popc(um));
        if (!first && cm) atomicAdd(&pchg[p], __popc(cm));
      }
      const unsigned below = (1u << lane) - 1u;
      u_at = __shfl_sync(0xffffffffu, u_at, 0) + __popc(um & below);
      c_at = __shfl_sync(0xffffffffu, c_at, 0) + __popc(cm & below);
      if (live && undecided) {
        // the exact re-score kernel decides this row among its candidates
        // and the screen's best
        ta.und_p[u_at] = p;
        ta.und_i[u_at] = (int32_t)i;
        uint32_t* words = ta.und_m + (int64_t)u_at * ta.und_w;
        for (int w = 0; w < ta.und_w; w++) {
          uint32_t m = ((cm_set >> w) & 1u) ? cmask[w] : 0u;
          if (w == (bj >> 5)) m |= 1u << (bj & 31);
          words[w] = m;
        }
      }
      if (chg) {
        labels[mt.lab_off + i] = lab;
        atomicAdd(&counts[mt.cnt_off + lab], 1);
        if (old >= 0) atomicAdd(&counts[mt.cnt_off + old], -1);
      }
      // the first pass's sums (every row enters) are made after the pass by
      // the bucketed kernels below
      if (first) continue;
      // later passes: the changed rows go to the change list (bucketed and
      // summed after the pass) while it has room
      const bool listed = chg && c_at < ta.chg_cap;
      if (listed) {
        ta.chg_row[c_at] = (int32_t)i;
        ta.chg_new[c_at] = mt.cnt_off + lab;
        ta.chg_old[c_at] = mt.cnt_off + old;
        atomicAdd(&ta.hist[2 * (mt.cnt_off + lab)], 1);
        atomicAdd(&ta.hist[2 * (mt.cnt_off + old) + 1], 1);
      }
      // the others' coordinates into the exact sums: the warp takes the
      // rows that enter one cluster (or leave one) together -- lanes over
      // consecutive coordinates, the group's 32-bit slices summed in 64-bit
      // registers (at most 32 slices: no overflow), one atomic per counter --
      // which gives the counters the same values as one add per row, since the
      // counters add modulo 2^64
      for (int dir = 0; dir < 2; dir++) {
        const bool mine = chg && !listed && (dir == 0 || old >= 0);
        const int key = dir == 0 ? lab : old;
        unsigned pend = __ballot_sync(0xffffffffu, mine);
        while (pend) {
          const int src = __ffs(pend) - 1;
          const int ks = __shfl_sync(0xffffffffu, key, src);
          const unsigned grp = __ballot_sync(0xffffffffu, mine && key == ks);
          pend &= ~grp;
          unsigned long long* dst = limbs + mt.limb_off + (int64_t)ks * mt.d * mt.L;
          for (int tb = 0; tb < mt.d; tb += 32) {
            const int t = tb + lane;
            const bool tv = t < mt.d;
            unsigned long long acc[4] = {0ull, 0ull, 0ull, 0ull};
            unsigned gm = grp;
            while (gm) {
              const int r = __ffs(gm) - 1;
              gm &= gm - 1;
              const int64_t is = __shfl_sync(0xffffffffu, i, r);
              if (tv) {
                const unsigned __int128 v = fixed_of(__ldg(X + mt.x_off + is * mt.d + t), mt.e_lo, dir == 1);
#pragma unroll
                for (int l = 0; l < 4; l++)
                  if (l < mt.L) acc[l] += (unsigned long long)((v >> (32 * l)) & 0xffffffffu);
              }
            }
            if (tv) {
#pragma unroll
              for (int l = 0; l < 4; l++)
                if (l < mt.L && acc[l]) atomicAdd(dst + (int64_t)t * mt.L + l, acc[l]);
            }
          }
        }
      }
    }
  }
  tcx::tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tcx::tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// Exact assignment of the rows the tensor-core screen left undecided: one
// warp per row, lanes over the centres (fuel's f32 operation order), the
// smallest (distance, index) key wins -- the first minimum, as in the
// CUDA-core pass -- then the row's sums move if its label changed.
template <int KIND, int ORDER>
__global__ void __launch_bounds__(256) batched_rescore_kernel(
    const BProb* __restrict__ probs, const int32_t* __restrict__ und_p, const int32_t* __restrict__ und_i,
    const uint32_t* __restrict__ und_m, int und_w, const int* __restrict__ und_n, const float* __restrict__ X,
    const float* __restrict__ C,
    int32_t* __restrict__ labels, unsigned long long* __restrict__ limbs, int32_t* __restrict__ counts,
    int32_t* __restrict__ pchg, int first) {
  const int lane = threadIdx.x & 31;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  const int cnt = *und_n;
  for (int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < cnt; u += nw) {
    const int p = und_p[u];
    const int64_t i = und_i[u];
    const BProb& pr = probs[p];
    const float* xr = X + pr.x_off + i * pr.d;
    uint64_t best = ~0ull;
    // the candidates (every centre whose lower bound reached the screen
    // best's upper bound, and that best): lane t scores the t-th of each 32
    const uint32_t* um = und_m + (int64_t)u * und_w;
    int w = 0;
    uint32_t m = um[0];
    for (;;) {
      int c = -1, got = 0;
      while (got < 32) {
        while (m == 0 && w + 1 < und_w) m = um[++w];
        if (m == 0) break;
        const int b = __ffs(m) - 1;
        m &= m - 1;
        if (got == lane) c = w * 32 + b;
        got++;
      }
      if (c >= 0 && c < pr.k) {
        const float dv = exact_dist_scalar<KIND, ORDER>(xr, C + pr.c_off + (int64_t)c * pr.d, pr.d);
        const uint64_t key = ((uint64_t)__float_as_uint(dv) << 32) | (uint32_t)c;
        best = key < best ? key : best;
      }
      if (got < 32) break;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const uint64_t v = ((uint64_t)__shfl_xor_sync(0xffffffffu, (uint32_t)(best >> 32), o) << 32) |
                         __shfl_xor_sync(0xffffffffu, (uint32_t)best, o);
      best = v < best ? v : best;
    }
    const int lab = (int)(uint32_t)best;
    const int old = first ? -1 : labels[pr.lab_off + i];
    if (lab == old) continue;
    if (lane == 0) {
      labels[pr.lab_off + i] = lab;
      if (!first) atomicAdd(&pchg[p], 1);
      atomicAdd(&counts[pr.cnt_off + lab], 1);
      if (old >= 0) atomicAdd(&counts[pr.cnt_off + old], -1);
    }
    if (first) continue;  // the first pass's sums: tc_first_sum_kernel
    for (int t = lane; t < pr.d; t += 32) {
      const float xv = __ldg(xr + t);
      add_coord(limbs + pr.limb_off + ((int64_t)lab * pr.d + t) * pr.L, xv, pr.e_lo, pr.L, false);
      if (old >= 0) add_coord(limbs + pr.limb_off + ((int64_t)old * pr.d + t) * pr.L, xv, pr.e_lo, pr.L, true);
    }
  }
}

// The first pass's exact sums of the tensor-core problems, after every row
// has its label (so a warp sums runs of rows of one cluster in registers
// instead of one atomic per row and counter): bucket offsets per cluster (one
// warp per problem: exclusive prefix of its final counts, from the problem's
// first row of the bucket array), the rows scattered into their clusters'
// buckets, then one warp per 32 bucket entries.
__global__ void tc_first_offsets_kernel(const BProb* __restrict__ probs, const int32_t* __restrict__ tcp, int ntc,
                                        const int64_t* __restrict__ row_base, const int32_t* __restrict__ counts,
                                        int64_t* __restrict__ boff, int32_t* __restrict__ cursor) {
  const int lane = threadIdx.x & 31;
  const int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (q >= ntc) return;
  const BProb pr = probs[tcp[q]];
  int64_t carry = row_base[q];
  for (int j0 = 0; j0 < pr.k; j0 += 32) {
    const int j = j0 + lane;
    const int c = j < pr.k ? counts[pr.cnt_off + j] : 0;
    int a = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, a, o);
      if (lane >= o) a += u;
    }
    if (j < pr.k) {
      boff[pr.cnt_off + j] = carry + a - c;
      cursor[pr.cnt_off + j] = 0;
    }
    carry += __shfl_sync(0xffffffffu, a, 31);
  }
}

__global__ void __launch_bounds__(kTcRows) tc_first_scatter_kernel(
    const BProb* __restrict__ probs, const int32_t* __restrict__ tcp, const int32_t* __restrict__ item_begin,
    int ntc, const int32_t* __restrict__ labels, const int64_t* __restrict__ boff, int32_t* __restrict__ cursor,
    int32_t* __restrict__ b_row, int32_t* __restrict__ b_gc) {
  const int item = blockIdx.x;
  int lo = 0, hi = ntc;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (item_begin[mid] <= item) lo = mid;
    else hi = mid;
  }
  const BProb pr = probs[tcp[lo]];
  const int64_t i = (int64_t)(item - item_begin[lo]) * kTcRows + threadIdx.x;
  const bool live = pr.active && i < pr.n;
  const int gc = live ? pr.cnt_off + labels[pr.lab_off + i] : -1;
  // one reservation per cluster among the warp's rows
  const unsigned grp = __match_any_sync(0xffffffffu, gc);
  const int lead = __ffs(grp) - 1;
  int at = 0;
  if (live && (int)(threadIdx.x & 31) == lead) at = atomicAdd(&cursor[gc], __popc(grp));
  at = __shfl_sync(0xffffffffu, at, lead) + __popc(grp & ((1u << (threadIdx.x & 31)) - 1u));
  if (live) {
    const int64_t e = boff[gc] + at;
    b_row[e] = (int32_t)i;
    b_gc[e] = gc;
  }
}

__global__ void __launch_bounds__(256) tc_first_sum_kernel(const BProb* __restrict__ probs,
                                                           const int32_t* __restrict__ gc_prob, int64_t entries,
                                                           const int32_t* __restrict__ b_row,
                                                           const int32_t* __restrict__ b_gc,
                                                           const float* __restrict__ X,
                                                           unsigned long long* __restrict__ limbs) {
  const int lane = threadIdx.x & 31;
  const int64_t w0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32;
  if (w0 >= entries) return;
  const int64_t e = w0 + lane;
  const int myrow = e < entries ? b_row[e] : 0;
  const int mygc = e < entries ? b_gc[e] : -1;
  int cur = -1;
  BProb pr{};
  unsigned long long a0[4] = {0ull, 0ull, 0ull, 0ull}, a1[4] = {0ull, 0ull, 0ull, 0ull};
  auto flush = [&]() {
    if (cur < 0) return;
    unsigned long long* dst = limbs + pr.limb_off + (int64_t)(cur - pr.cnt_off) * pr.d * pr.L;
    for (int l = 0; l < pr.L; l++) {
      if (lane < pr.d && a0[l]) atomicAdd(dst + (int64_t)lane * pr.L + l, a0[l]);
      if (lane + 32 < pr.d && a1[l]) atomicAdd(dst + (int64_t)(lane + 32) * pr.L + l, a1[l]);
      a0[l] = 0ull;
      a1[l] = 0ull;
    }
  };
#pragma unroll 4
  for (int t = 0; t < 32; t++) {
    const int gc = __shfl_sync(0xffffffffu, mygc, t);
    if (gc < 0) break;
    const int row = __shfl_sync(0xffffffffu, myrow, t);
    if (gc != cur) {
      flush();
      cur = gc;
      pr = probs[gc_prob[gc]];
    }
    const float* xr = X + pr.x_off + (int64_t)row * pr.d;
    const float x0 = lane < pr.d ? __ldg(xr + lane) : 0.0f;
    const float x1 = lane + 32 < pr.d ? __ldg(xr + lane + 32) : 0.0f;
    const unsigned __int128 v0 = fixed_of(x0, pr.e_lo, false), v1 = fixed_of(x1, pr.e_lo, false);
#pragma unroll
    for (int l = 0; l < 4; l++) {
      if (l < pr.L) {
        a0[l] += (unsigned long long)((v0 >> (32 * l)) & 0xffffffffu);
        a1[l] += (unsigned long long)((v1 >> (32 * l)) & 0xffffffffu);
      }
    }
  }
  flush();
}

// Passes after the first: the listed changes' exact sums.  Bucket offsets per
// key (one warp per problem: its keys' exclusive prefix, the problem's region
// taken from a global counter; the counts and cursors are cleared for the next
// pass), the listed rows scattered under their keys (one reservation per key
// among a warp's rows), then one warp per 32 bucket entries sums runs of one
// key in registers (rows leaving a cluster negated).  ctl: [0] listed rows,
// [1] region counter, [2] bucket entries of the pass.
__global__ void chg_offsets_kernel(const BProb* __restrict__ probs, const int32_t* __restrict__ tcp, int ntc,
                                   int32_t* __restrict__ hist, int64_t* __restrict__ boff,
                                   int32_t* __restrict__ cursor, int* __restrict__ ctl) {
  const int lane = threadIdx.x & 31;
  const int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (q >= ntc) return;
  const BProb pr = probs[tcp[q]];
  const int nk = 2 * pr.k, k0 = 2 * pr.cnt_off;
  int tot = 0;
  for (int j0 = 0; j0 < nk; j0 += 32) tot += (j0 + lane < nk) ? hist[k0 + j0 + lane] : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
  if (tot == 0) return;
  int base = 0;
  if (lane == 0) base = atomicAdd(&ctl[1], tot);
  int64_t carry = __shfl_sync(0xffffffffu, base, 0);
  for (int j0 = 0; j0 < nk; j0 += 32) {
    const int j = j0 + lane;
    const int c = j < nk ? hist[k0 + j] : 0;
    int a = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, a, o);
      if (lane >= o) a += u;
    }
    if (j < nk) {
      boff[k0 + j] = carry + a - c;
      cursor[k0 + j] = 0;
      hist[k0 + j] = 0;
    }
    carry += __shfl_sync(0xffffffffu, a, 31);
  }
}

__global__ void __launch_bounds__(256) chg_scatter_kernel(const int32_t* __restrict__ chg_row,
                                                          const int32_t* __restrict__ chg_new,
                                                          const int32_t* __restrict__ chg_old, int cap,
                                                          const int64_t* __restrict__ boff,
                                                          int32_t* __restrict__ cursor, int32_t* __restrict__ b_row,
                                                          int32_t* __restrict__ b_key, int* __restrict__ ctl) {
  const int lane = threadIdx.x & 31;
  const int n = min(ctl[0], cap);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctl[2] = ctl[1];  // this pass's bucket entries
    ctl[1] = 0;
  }
  const int stride = gridDim.x * blockDim.x;
  for (int e0 = blockIdx.x * blockDim.x; e0 < n; e0 += stride) {
    const int e = e0 + threadIdx.x;
    const bool v = e < n;
    const int row = v ? chg_row[e] : 0;
#pragma unroll
    for (int dir = 0; dir < 2; dir++) {
      const int key = v ? 2 * (dir ? chg_old[e] : chg_new[e]) + dir : -1;
      const unsigned grp = __match_any_sync(0xffffffffu, key);
      const int lead = __ffs(grp) - 1;
      int at = 0;
      if (v && lane == lead) at = atomicAdd(&cursor[key], __popc(grp));
      at = __shfl_sync(0xffffffffu, at, lead) + __popc(grp & ((1u << lane) - 1u));
      if (v) {
        const int64_t b = boff[key] + at;
        b_row[b] = row;
        b_key[b] = key;
      }
    }
  }
}

__global__ void __launch_bounds__(256) chg_sum_kernel(const BProb* __restrict__ probs,
                                                      const int32_t* __restrict__ gc_prob,
                                                      const int32_t* __restrict__ b_row,
                                                      const int32_t* __restrict__ b_key, const float* __restrict__ X,
                                                      unsigned long long* __restrict__ limbs, int* __restrict__ ctl) {
  const int lane = threadIdx.x & 31;
  const int64_t entries = ctl[2];
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl[0] = 0;  // the list, for the next pass
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t w0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; w0 < entries; w0 += nw * 32) {
    const int64_t e = w0 + lane;
    const int myrow = e < entries ? b_row[e] : 0;
    const int mykey = e < entries ? b_key[e] : -1;
    int cur = -1;
    BProb pr{};
    unsigned long long a0[4] = {0ull, 0ull, 0ull, 0ull}, a1[4] = {0ull, 0ull, 0ull, 0ull};
    auto flush = [&]() {
      if (cur < 0) return;
      unsigned long long* dst = limbs + pr.limb_off + (int64_t)((cur >> 1) - pr.cnt_off) * pr.d * pr.L;
#pragma unroll
      for (int l = 0; l < 4; l++) {
        if (l < pr.L) {
          if (lane < pr.d && a0[l]) atomicAdd(dst + (int64_t)lane * pr.L + l, a0[l]);
          if (lane + 32 < pr.d && a1[l]) atomicAdd(dst + (int64_t)(lane + 32) * pr.L + l, a1[l]);
        }
        a0[l] = 0ull;
        a1[l] = 0ull;
      }
    };
#pragma unroll 4
    for (int t = 0; t < 32; t++) {
      const int key = __shfl_sync(0xffffffffu, mykey, t);
      if (key < 0) break;
      const int row = __shfl_sync(0xffffffffu, myrow, t);
      if (key != cur) {
        flush();
        cur = key;
        pr = probs[gc_prob[key >> 1]];
      }
      const float* xr = X + pr.x_off + (int64_t)row * pr.d;
      const bool neg = (key & 1) != 0;
      const float x0 = lane < pr.d ? __ldg(xr + lane) : 0.0f;
      const float x1 = lane + 32 < pr.d ? __ldg(xr + lane + 32) : 0.0f;
      const unsigned __int128 v0 = fixed_of(x0, pr.e_lo, neg), v1 = fixed_of(x1, pr.e_lo, neg);
#pragma unroll
      for (int l = 0; l < 4; l++) {
        if (l < pr.L) {
          a0[l] += (unsigned long long)((v0 >> (32 * l)) & 0xffffffffu);
          a1[l] += (unsigned long long)((v1 >> (32 * l)) & 0xffffffffu);
        }
      }
    }
    flush();
  }
}

struct DevBuf {
  void* p = nullptr;
  cudaStream_t s = nullptr;
  ~DevBuf() {
    if (p) cudaFreeAsync(p, s);
  }
  int alloc(size_t b, cudaStream_t st) {
    s = st;
    if (cudaMallocFromPoolAsync(&p, b ? b : 16, lib_pool(), st) != cudaSuccess) {
      cudaGetLastError();
      p = nullptr;
      set_error("device allocation of %zu bytes failed", b);
      return ST_ENOMEM;
    }
    return ST_OK;
  }
  template <class T>
  T* as() const {
    return static_cast<T*>(p);
  }
};

// What kind of memory an address is: device memory at all, and (kHereInRange) a
// range of bytes, aligned for floats, that lies in one allocation of this device.
constexpr int kDeviceMem = 1, kHereInRange = 2;
int pointer_kind(const void* ptr, size_t bytes, int dev) {
  // (through the runtime: the library loads on machines without a driver)
  using Fn = CUresult (*)(unsigned, CUpointer_attribute*, void**, CUdeviceptr);
  static const Fn attributes = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &f, 7000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      f = nullptr;
    }
    return (Fn)f;
  }();
  CUmemorytype type = (CUmemorytype)0;
  unsigned managed = 0;
  int ord = -1;
  CUdeviceptr start = 0;
  size_t size = 0;
  CUpointer_attribute at[5] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                               CU_POINTER_ATTRIBUTE_DEVICE_ORDINAL, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                               CU_POINTER_ATTRIBUTE_RANGE_SIZE};
  void* out[5] = {&type, &managed, &ord, &start, &size};
  const CUdeviceptr a = (CUdeviceptr)(uintptr_t)ptr;
  if (attributes == nullptr) {
    cudaPointerAttributes pa;
    if (cudaPointerGetAttributes(&pa, ptr) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return pa.type == cudaMemoryTypeDevice ? kDeviceMem : 0;
  }
  if (attributes(5, at, out, a) != CUDA_SUCCESS || type != CU_MEMORYTYPE_DEVICE || managed) return 0;
  const bool here = ord == dev && (a & 3) == 0 && a >= start && bytes <= size && a - start <= size - bytes;
  return kDeviceMem | (here ? kHereInRange : 0);
}

// Launch shapes chosen per problem mix by timing the candidates once (the
// first middle iteration of the first call with that mix), cached per
// process.  Key: the sorted multiset of (d, k bucket) of the problems.
struct Tuned {
  int blocks_per_sm = 0;
};
std::mutex g_tune_mu;
std::map<std::vector<int>, Tuned> g_tuned;

}  // namespace
}  // namespace fuelg

using namespace fuelg;

extern "C" int fuelg_kmeans_batched(fuelg_kmeans_problem* probs, int32_t count, int32_t max_iter, int32_t order,
                                    int32_t precision, int32_t flags, fuelg_stats* stats) {
  if (count < 0 || (count > 0 && !probs) || max_iter < 1) {
    set_error("invalid batched kmeans arguments count=%d max_iter=%d", count, max_iter);
    return ST_EINVAL;
  }
  if (order != FUELG_ORDER_ARM && order != FUELG_ORDER_X86) {
    set_error("unknown summation order %d", order);
    return ST_EINVAL;
  }
  if (precision < FUELG_PREC_AUTO || precision > FUELG_PREC_SPLIT_BF16) {
    set_error("unknown precision tier %d", precision);
    return ST_EINVAL;
  }
  if (precision == FUELG_PREC_AUTO) precision = FUELG_PREC_SPLIT_BF16;  // the screen takes the problems it serves
  for (int p = 0; p < count; p++) {
    const fuelg_kmeans_problem& q = probs[p];
    if (q.n < 1 || q.d < 1 || q.k < 1 || !q.data || !q.init || !q.out_centers || !q.out_labels) {
      set_error("invalid problem %d (n=%lld d=%d k=%d)", p, (long long)q.n, q.d, q.k);
      return ST_EINVAL;
    }
    if (q.n >= (1ll << 31) || (int64_t)q.k * q.d > (1ll << 28)) {
      set_error("problem %d too large for the batched engine", p);
      return ST_ENOTSUP;
    }
  }
  if (stats) memset(stats, 0, sizeof(*stats));
  if (count == 0) return ST_OK;
  cudaStream_t s;
  FUELG_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  struct SG {
    cudaStream_t s;
    ~SG() { cudaStreamDestroy(s); }
  } sg{s};
  // the CUDA-core kernel's stream (forked from s and joined back every pass)
  cudaStream_t s2;
  FUELG_CUDA(cudaStreamCreateWithFlags(&s2, cudaStreamNonBlocking));
  SG sg2{s2};
  cudaEvent_t ev_fork, ev_join;
  FUELG_CUDA(cudaEventCreateWithFlags(&ev_fork, cudaEventDisableTiming));
  FUELG_CUDA(cudaEventCreateWithFlags(&ev_join, cudaEventDisableTiming));
  struct EG2 {
    cudaEvent_t a, b;
    ~EG2() {
      cudaEventDestroy(a);
      cudaEventDestroy(b);
    }
  } eg2{ev_fork, ev_join};
  const int64_t launches0 = launch_count();
  cudaEvent_t ev0, ev1, evh0, evh1;
  cudaEventCreate(&ev0);
  cudaEventCreate(&ev1);
  cudaEventCreate(&evh0);
  cudaEventCreate(&evh1);
  struct EG {
    cudaEvent_t a, b, c, d;
    ~EG() {
      cudaEventDestroy(a);
      cudaEventDestroy(b);
      cudaEventDestroy(c);
      cudaEventDestroy(d);
    }
  } eg{ev0, ev1, evh0, evh1};
  cudaEventRecord(ev0, s);

  // layout
  const int P = count;
  std::vector<BProb> hp(P);
  std::vector<int64_t> xoff(P + 1, 0), kdb(P + 1, 0);
  std::vector<int32_t> rblk(P + 1, 0);
  int64_t xs = 0, cs = 0, ls = 0, ks = 0, kd = 0;
  int64_t items = 0;      // CUDA-core 256-row items
  int64_t all_items = 0;  // 256-row items of every problem (inertia)
  int64_t work = 0;
  std::vector<int32_t> tcp, tc_begin;  // tensor-core problems and their 128-row item starts
  int64_t tc_items = 0, tc_rows = 0;
  int tc_kmax = 1;
  int64_t rb = 0;
  for (int p = 0; p < P; p++) {
    const fuelg_kmeans_problem& q = probs[p];
    hp[p].x_off = xs;
    hp[p].n = q.n;
    hp[p].lab_off = ls;
    hp[p].c_off = cs;
    hp[p].cnt_off = (int32_t)ks;
    hp[p].d = q.d;
    hp[p].k = q.k;
    // tensor-core tier: split-BF16 screen for 32 <= d <= 64, k <= 256
    hp[p].tc = (precision != FUELG_PREC_FP32 && q.d >= 32 && q.d <= 64 && q.k <= 256) ? 1 : 0;
    hp[p].item_begin = (int32_t)items;
    hp[p].all_item_begin = (int32_t)all_items;
    hp[p].cost_begin = work;
    hp[p].item_cost = (int64_t)q.k * q.d + 64;  // distance work + per-row overhead
    const int64_t its = hp[p].tc ? 0 : (q.n + kItemRows - 1) / kItemRows;
    work += hp[p].item_cost * its;
    all_items += (q.n + kItemRows - 1) / kItemRows;
    if (hp[p].tc) {
      tcp.push_back(p);
      tc_begin.push_back((int32_t)tc_items);
      tc_items += (q.n + kTcRows - 1) / kTcRows;
      tc_rows += q.n;
      tc_kmax = std::max(tc_kmax, q.k);
    }
    xoff[p] = xs;
    kdb[p] = kd;
    rblk[p] = (int32_t)rb;
    xs += (q.n * q.d + 3) & ~3ll;  // 16-byte aligned rows for d % 4 == 0
    cs += ((int64_t)q.k * q.d + 3) & ~3ll;
    ls += q.n;
    ks += q.k;
    kd += (int64_t)q.k * q.d;
    items += its;
    rb += (q.n * q.d + 65535) / 65536;
  }
  xoff[P] = xs;
  kdb[P] = kd;
  rblk[P] = (int32_t)rb;
  tc_begin.push_back((int32_t)tc_items);
  // 32-bit item starts; centre keys 2 gc + 1 (gc < ks) of the change list are 32-bit
  if (all_items >= (1ll << 31) || tc_items >= (1ll << 31) || ks >= (1ll << 30)) {
    set_error("batch too large");
    return ST_ENOTSUP;
  }
  DevBuf dX, dC, dLab, dCnt, dOff, dRb, dRange, dProbs, dKdb, dPchg, dConv, dLast, dIter, dInert, dLimbs, dTcp,
      dTcb, dSt, dUnd, dCtaB, dSrc;
  FUELG_TRY(dX.alloc(sizeof(float) * xs, s));
  FUELG_TRY(dC.alloc(sizeof(float) * cs, s));
  FUELG_TRY(dLab.alloc(sizeof(int32_t) * ls, s));
  FUELG_TRY(dCnt.alloc(sizeof(int32_t) * ks, s));
  FUELG_TRY(dOff.alloc(sizeof(int64_t) * (P + 1), s));
  FUELG_TRY(dRb.alloc(sizeof(int32_t) * (P + 1), s));
  FUELG_TRY(dRange.alloc(sizeof(int) * 3 * P, s));
  // rows and first centres: read in place by the gather kernels from this device's
  // memory, else copied to their places first
  std::vector<BSrc> hsrc(P);
  int cur_dev = 0;
  FUELG_CUDA(cudaGetDevice(&cur_dev));
  for (int p = 0; p < P; p++) {
    const size_t xb = sizeof(float) * probs[p].n * probs[p].d, cb = sizeof(float) * probs[p].k * probs[p].d;
    hsrc[p] = {probs[p].data, probs[p].init, probs[p].n * probs[p].d};
    if (!(pointer_kind(probs[p].data, xb, cur_dev) & kHereInRange)) {
      hsrc[p].x = dX.as<float>() + hp[p].x_off;
      FUELG_CUDA(cudaMemcpyAsync(dX.as<float>() + hp[p].x_off, probs[p].data, xb, cudaMemcpyDefault, s));
    }
    if (!(pointer_kind(probs[p].init, cb, cur_dev) & kHereInRange)) {
      hsrc[p].c = dC.as<float>() + hp[p].c_off;
      FUELG_CUDA(cudaMemcpyAsync(dC.as<float>() + hp[p].c_off, probs[p].init, cb, cudaMemcpyDefault, s));
    }
  }
  FUELG_TRY(dSrc.alloc(sizeof(BSrc) * P, s));
  FUELG_CUDA(cudaMemcpyAsync(dSrc.p, hsrc.data(), sizeof(BSrc) * P, cudaMemcpyHostToDevice, s));
  FUELG_CUDA(cudaMemcpyAsync(dOff.p, xoff.data(), sizeof(int64_t) * (P + 1), cudaMemcpyHostToDevice, s));
  FUELG_CUDA(cudaMemcpyAsync(dRb.p, rblk.data(), sizeof(int32_t) * (P + 1), cudaMemcpyHostToDevice, s));
  {
    std::vector<int> init(3 * P);
    for (int p = 0; p < P; p++) {
      init[3 * p] = 1 << 30;
      init[3 * p + 1] = -(1 << 30);
      init[3 * p + 2] = 0;
    }
    FUELG_CUDA(cudaMemcpyAsync(dRange.p, init.data(), sizeof(int) * 3 * P, cudaMemcpyHostToDevice, s));
    FUELG_CUDA(cudaStreamSynchronize(s));  // `init` leaves scope
  }
  if (rb > 0) {
    batched_gather_kernel<<<(unsigned)rb, 256, 0, s>>>(dSrc.as<BSrc>(), dX.as<float>(), dOff.as<int64_t>(),
                                                       dRb.as<int32_t>(), P, dRange.as<int>());
    note_launch();
    FUELG_CUDA(cudaGetLastError());
  }
  std::vector<int> hr(3 * P);
  FUELG_CUDA(cudaMemcpyAsync(hr.data(), dRange.p, sizeof(int) * 3 * P, cudaMemcpyDeviceToHost, s));
  FUELG_CUDA(cudaStreamSynchronize(s));
  int64_t limbs_total = 0;
  for (int p = 0; p < P; p++) {
    int e_lo = hr[3 * p], e_hi = hr[3 * p + 1];
    if (e_lo > e_hi) e_lo = e_hi = 0;  // all zeros
    int logn = 0;
    while ((1ll << logn) <= hp[p].n) logn++;
    const int bits = (e_hi - e_lo + 1) + logn + 1;
    const int L = (bits + 31) / 32;
    hp[p].active = (hr[3 * p + 2] == 0 && L <= 4) ? 1 : 0;
    hp[p].L = std::max(1, std::min(4, L));
    hp[p].e_lo = e_lo;
    hp[p].limb_off = limbs_total;
    limbs_total += (int64_t)hp[p].k * hp[p].d * hp[p].L;
  }
  FUELG_TRY(dLimbs.alloc(sizeof(unsigned long long) * limbs_total, s));
  FUELG_TRY(dProbs.alloc(sizeof(BProb) * P, s));
  FUELG_TRY(dKdb.alloc(sizeof(int64_t) * (P + 1), s));
  FUELG_TRY(dPchg.alloc(sizeof(int32_t) * P, s));
  FUELG_TRY(dConv.alloc(sizeof(int32_t) * P, s));
  FUELG_TRY(dLast.alloc(sizeof(int32_t) * P, s));
  FUELG_TRY(dIter.alloc(sizeof(int32_t), s));
  FUELG_TRY(dInert.alloc(sizeof(double) * P, s));
  FUELG_CUDA(cudaMemcpyAsync(dProbs.p, hp.data(), sizeof(BProb) * P, cudaMemcpyHostToDevice, s));
  batched_centres_kernel<<<(unsigned)P, 256, 0, s>>>(dSrc.as<BSrc>(), dProbs.as<BProb>(), dC.as<float>());
  note_launch();
  FUELG_CUDA(cudaGetLastError());
  const int ntc = (int)tcp.size();
  FUELG_TRY(dTcp.alloc(sizeof(int32_t) * std::max(1, ntc), s));
  FUELG_TRY(dTcb.alloc(sizeof(int32_t) * (ntc + 1), s));
  FUELG_TRY(dSt.alloc(sizeof(int) * 4, s));
  if (ntc) FUELG_CUDA(cudaMemcpyAsync(dTcp.p, tcp.data(), sizeof(int32_t) * ntc, cudaMemcpyHostToDevice, s));
  FUELG_CUDA(cudaMemcpyAsync(dTcb.p, tc_begin.data(), sizeof(int32_t) * (ntc + 1), cudaMemcpyHostToDevice, s));
  FUELG_CUDA(cudaMemsetAsync(dSt.p, 0, sizeof(int) * 4, s));
  FUELG_CUDA(cudaMemcpyAsync(dKdb.p, kdb.data(), sizeof(int64_t) * (P + 1), cudaMemcpyHostToDevice, s));
  FUELG_CUDA(cudaMemsetAsync(dLimbs.p, 0, sizeof(unsigned long long) * limbs_total, s));
  FUELG_CUDA(cudaMemsetAsync(dCnt.p, 0, sizeof(int32_t) * ks, s));
  FUELG_CUDA(cudaMemsetAsync(dPchg.p, 0, sizeof(int32_t) * P, s));
  FUELG_CUDA(cudaMemsetAsync(dConv.p, 0, sizeof(int32_t) * P, s));
  FUELG_CUDA(cudaMemsetAsync(dIter.p, 0, sizeof(int32_t), s));
  FUELG_CUDA(cudaMemsetAsync(dInert.p, 0, sizeof(double) * P, s));

  // centre staging sized for the problems this kernel serves (those without
  // the tensor-core screen): more resident CTAs when their centres are small
  int ccap = 4;
  for (int p = 0; p < P; p++)
    if (!hp[p].tc) ccap = std::max<int64_t>(ccap, std::min<int64_t>(kCentreCap, (int64_t)((hp[p].k + 1) & ~1) * hp[p].d));
  ccap = (ccap + 3) & ~3;
  // With tensor-core problems in the batch the CUDA-core kernel runs beside the
  // screen (its own stream, joined before the centre update): with the centres
  // of the problems it serves (d < 32) one of its CTAs fits beside the
  // screen's on every SM, and its warps use the issue slots the screen's
  // epilogue leaves.
  const bool concurrent = items > 0 && tc_items > 0;
  const size_t smem = sizeof(float) * ccap + sizeof(unsigned long long) * kAggCap + sizeof(int) * 256;
  // With 64 registers twice as many rows are resident, which rows of 32 dimensions and
  // more pay with L1 misses (they are read again for every centre): 10 passes of
  // 20 000 x 100, k = 200 14.1 ms, 13.1 with 128; x 65, k = 100 4.8, 3.4; x 31, k = 100 1.68, 1.69.
  bool wide = false;
  for (int p = 0; p < P; p++) wide = wide || (!hp[p].tc && hp[p].d >= 32);
  auto assign = [&](auto kind, bool x86) {
    constexpr int K = decltype(kind)::value;
    return x86 ? (wide ? batched_assign_kernel<K, ORDER_X86, true> : batched_assign_kernel<K, ORDER_X86, false>)
               : (wide ? batched_assign_kernel<K, ORDER_ARM, true> : batched_assign_kernel<K, ORDER_ARM, false>);
  };
  auto k_init = assign(Dim<KIND_PAIRWISE>{}, order == FUELG_ORDER_X86);
  auto k_iter = assign(Dim<KIND_SQDIST>{}, order == FUELG_ORDER_X86);
  FUELG_CUDA(cudaFuncSetAttribute(k_init, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  FUELG_CUDA(cudaFuncSetAttribute(k_iter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  auto t_init = order == FUELG_ORDER_X86 ? batched_tc_assign_kernel<KIND_PAIRWISE, ORDER_X86>
                                         : batched_tc_assign_kernel<KIND_PAIRWISE, ORDER_ARM>;
  auto t_iter = order == FUELG_ORDER_X86 ? batched_tc_assign_kernel<KIND_SQDIST, ORDER_X86>
                                         : batched_tc_assign_kernel<KIND_SQDIST, ORDER_ARM>;
  const size_t tsmem = kTcSmem;
  FUELG_CUDA(cudaFuncSetAttribute(t_init, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsmem));
  FUELG_CUDA(cudaFuncSetAttribute(t_iter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsmem));
  BTcArgs ta{};
  ta.tcp = dTcp.as<int32_t>();
  ta.item_begin = dTcb.as<int32_t>();
  ta.ntc = ntc;
  ta.items = (int)tc_items;
  {
    // operand rounding of hi + lo (3.01 * 2^-16) + FP32 accumulation of 3 x 64 products
    const double rel = 3.01 * std::ldexp(1.0, -16) + 3.0 * 64 * std::ldexp(1.0, -23) * (1.0 + std::ldexp(1.0, -7));
    ta.alpha = (float)(2.0 * rel * 1.01);
  }
  ta.status = dSt.as<int>();
  ta.undecided = reinterpret_cast<unsigned long long*>(dSt.as<int>() + 2);
  ta.und_n = dSt.as<int>() + 1;
  ta.und_w = (tc_kmax + 31) / 32;
  FUELG_TRY(dUnd.alloc(sizeof(int32_t) * (2 + ta.und_w) * std::max<int64_t>(1, tc_rows), s));
  ta.und_p = dUnd.as<int32_t>();
  ta.und_i = dUnd.as<int32_t>() + std::max<int64_t>(1, tc_rows);
  ta.und_m = reinterpret_cast<uint32_t*>(dUnd.as<int32_t>() + 2 * std::max<int64_t>(1, tc_rows));
  // the first pass's bucketed sums of the tensor-core problems: the bucket
  // array (row, cluster) reuses the undecided list's memory once the first
  // re-score is done; rows of each active problem from row_base[q]
  DevBuf dBoff, dCur, dGcp, dRowB;
  int64_t tc_entries = 0;
  if (tc_items > 0) {
    std::vector<int64_t> rowb(ntc + 1);
    for (int q = 0; q < ntc; q++) {
      rowb[q] = tc_entries;
      if (hp[tcp[q]].active) tc_entries += hp[tcp[q]].n;
    }
    rowb[ntc] = tc_entries;
    std::vector<int32_t> gcp(std::max<int64_t>(1, ks));
    for (int p = 0; p < P; p++)
      for (int j = 0; j < hp[p].k; j++) gcp[hp[p].cnt_off + j] = p;
    FUELG_TRY(dBoff.alloc(sizeof(int64_t) * std::max<int64_t>(1, ks), s));
    FUELG_TRY(dCur.alloc(sizeof(int32_t) * std::max<int64_t>(1, ks), s));
    FUELG_TRY(dGcp.alloc(sizeof(int32_t) * std::max<int64_t>(1, ks), s));
    FUELG_TRY(dRowB.alloc(sizeof(int64_t) * (ntc + 1), s));
    FUELG_CUDA(cudaMemcpyAsync(dGcp.p, gcp.data(), sizeof(int32_t) * gcp.size(), cudaMemcpyHostToDevice, s));
    FUELG_CUDA(cudaMemcpyAsync(dRowB.p, rowb.data(), sizeof(int64_t) * (ntc + 1), cudaMemcpyHostToDevice, s));
  }
  // later passes: the change list (room for half the tensor-core rows; the
  // rest of a pass's changes take the epilogue's direct sums), its per-key
  // counts, offsets and cursors, the buckets and three control words
  DevBuf dChg, dHist, dKoff, dKcur, dBk, dCtl;
  // (bucket positions and the region counter are 32-bit: at most 2^29 listed rows)
  const int chg_cap = (int)std::max<int64_t>(1, std::min<int64_t>(tc_rows / 2, 1ll << 29));
  if (tc_items > 0) {
    FUELG_TRY(dChg.alloc(sizeof(int32_t) * 3 * (size_t)chg_cap, s));
    FUELG_TRY(dHist.alloc(sizeof(int32_t) * 2 * std::max<int64_t>(1, ks), s));
    FUELG_TRY(dKoff.alloc(sizeof(int64_t) * 2 * std::max<int64_t>(1, ks), s));
    FUELG_TRY(dKcur.alloc(sizeof(int32_t) * 2 * std::max<int64_t>(1, ks), s));
    FUELG_TRY(dBk.alloc(sizeof(int32_t) * 4 * (size_t)chg_cap, s));
    FUELG_TRY(dCtl.alloc(sizeof(int) * 4, s));
    FUELG_CUDA(cudaMemsetAsync(dHist.p, 0, sizeof(int32_t) * 2 * std::max<int64_t>(1, ks), s));
    FUELG_CUDA(cudaMemsetAsync(dCtl.p, 0, sizeof(int) * 4, s));
    ta.chg_row = dChg.as<int32_t>();
    ta.chg_new = ta.chg_row + chg_cap;
    ta.chg_old = ta.chg_new + chg_cap;
    ta.hist = dHist.as<int32_t>();
    ta.chg_n = dCtl.as<int>();
    ta.chg_cap = chg_cap;
  }
  auto r_init = order == FUELG_ORDER_X86 ? batched_rescore_kernel<KIND_PAIRWISE, ORDER_X86>
                                         : batched_rescore_kernel<KIND_PAIRWISE, ORDER_ARM>;
  auto r_iter = order == FUELG_ORDER_X86 ? batched_rescore_kernel<KIND_SQDIST, ORDER_X86>
                                         : batched_rescore_kernel<KIND_SQDIST, ORDER_ARM>;
  int sms = 152;
  {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  // tuned launch shape for this mix of (d, k) buckets
  std::vector<int> key;
  for (int p = 0; p < P; p++) key.push_back(hp[p].d * 16 + std::min(15, (int)std::log2((double)hp[p].k)));
  std::sort(key.begin(), key.end());
  int bps = 0;
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tuned.find(key);
    if (it != g_tuned.end()) bps = it->second.blocks_per_sm;
  }
  auto grid_for = [&](int b) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>(items, (int64_t)sms * b)); };
  // one persistent screen CTA per SM, each over a contiguous range of items of
  // equal estimated cost (cycles per item by k: 3200 at 30, 3700 at 48, 4700 at 113)
  const unsigned tc_grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(tc_items, (int64_t)sms));
  {
    std::vector<double> icost(ntc);
    double total = 0.0;
    for (int q = 0; q < ntc; q++) {
      const int kp = (hp[tcp[q]].k + 15) & ~15;
      icost[q] = 200.0 + 2.0 * kp;
      total += icost[q] * (tc_begin[q + 1] - tc_begin[q]);
    }
    std::vector<int64_t> cb(tc_grid + 1, 0);
    cb[tc_grid] = tc_items;
    double acc = 0.0;
    int q = 0;
    for (unsigned c = 1; c < tc_grid; c++) {
      const double target = total * c / tc_grid;
      while (q < ntc && acc + icost[q] * (tc_begin[q + 1] - tc_begin[q]) < target) {
        acc += icost[q] * (tc_begin[q + 1] - tc_begin[q]);
        q++;
      }
      int64_t at = tc_items;
      if (q < ntc) at = std::min<int64_t>(tc_begin[q + 1], tc_begin[q] + (int64_t)std::ceil((target - acc) / icost[q]));
      cb[c] = std::max(cb[c - 1], at);
    }
    FUELG_TRY(dCtaB.alloc(sizeof(int64_t) * (tc_grid + 1), s));
    FUELG_CUDA(cudaMemcpyAsync(dCtaB.p, cb.data(), sizeof(int64_t) * (tc_grid + 1), cudaMemcpyHostToDevice, s));
    ta.cta_begin = dCtaB.as<int64_t>();
  }
  const unsigned mean_grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>((kd + 255) / 256, (int64_t)sms * 8));
  const int fixed = (flags & FUELG_LLOYD_FIXED_ITERS) ? 1 : 0;
  (void)fixed;  // every pass runs; the reported count follows the changed == 0 stop unless fixed

  auto pass = [&](bool first, bool write, unsigned grid) -> int {
    cudaStream_t sc = s;
    if (concurrent) {
      FUELG_CUDA(cudaEventRecord(ev_fork, s));
      FUELG_CUDA(cudaStreamWaitEvent(s2, ev_fork, 0));
      sc = s2;
    }
    if (items > 0) {
      if (first)
        k_init<<<grid, kItemRows, smem, sc>>>(dProbs.as<BProb>(), P, (int)items, dX.as<float>(), dC.as<float>(),
                                             dLab.as<int32_t>(), dLimbs.as<unsigned long long>(), dCnt.as<int32_t>(),
                                             dPchg.as<int32_t>(), 1, work, ccap, kNegZero2);
      else
        k_iter<<<grid, kItemRows, smem, sc>>>(dProbs.as<BProb>(), P, (int)items, dX.as<float>(), dC.as<float>(),
                                             dLab.as<int32_t>(), dLimbs.as<unsigned long long>(), dCnt.as<int32_t>(),
                                             dPchg.as<int32_t>(), 0, work, ccap, kNegZero2);
      note_launch();
    }
    if (tc_items > 0) {
      (first ? t_init : t_iter)<<<tc_grid, kTcThreads, tsmem, s>>>(dProbs.as<BProb>(), ta, dX.as<float>(),
                                                                 dC.as<float>(), dLab.as<int32_t>(),
                                                                 dLimbs.as<unsigned long long>(),
                                                                 dCnt.as<int32_t>(), dPchg.as<int32_t>(),
                                                                 first ? 1 : 0);
      note_launch();
      (first ? r_init : r_iter)<<<sms * 8, 256, 0, s>>>(dProbs.as<BProb>(), ta.und_p, ta.und_i, ta.und_m, ta.und_w,
                                                        ta.und_n,
                                                        dX.as<float>(), dC.as<float>(), dLab.as<int32_t>(),
                                                        dLimbs.as<unsigned long long>(), dCnt.as<int32_t>(),
                                                        dPchg.as<int32_t>(), first ? 1 : 0);
      note_launch();
      if (first) {
        int32_t* b_row = dUnd.as<int32_t>();
        int32_t* b_gc = b_row + std::max<int64_t>(1, tc_rows);
        tc_first_offsets_kernel<<<(unsigned)((ntc * 32 + 255) / 256), 256, 0, s>>>(
            dProbs.as<BProb>(), ta.tcp, ntc, dRowB.as<int64_t>(), dCnt.as<int32_t>(), dBoff.as<int64_t>(),
            dCur.as<int32_t>());
        note_launch();
        tc_first_scatter_kernel<<<(unsigned)tc_items, kTcRows, 0, s>>>(dProbs.as<BProb>(), ta.tcp, ta.item_begin, ntc,
                                                                       dLab.as<int32_t>(), dBoff.as<int64_t>(),
                                                                       dCur.as<int32_t>(), b_row, b_gc);
        note_launch();
        if (tc_entries > 0) {
          tc_first_sum_kernel<<<(unsigned)((tc_entries + 255) / 256), 256, 0, s>>>(
              dProbs.as<BProb>(), dGcp.as<int32_t>(), tc_entries, b_row, b_gc, dX.as<float>(),
              dLimbs.as<unsigned long long>());
          note_launch();
        }
      } else {
        int32_t* b_row = dBk.as<int32_t>();
        int32_t* b_key = b_row + 2 * (size_t)chg_cap;
        chg_offsets_kernel<<<(unsigned)((ntc * 32 + 255) / 256), 256, 0, s>>>(
            dProbs.as<BProb>(), ta.tcp, ntc, dHist.as<int32_t>(), dKoff.as<int64_t>(), dKcur.as<int32_t>(),
            dCtl.as<int>());
        note_launch();
        chg_scatter_kernel<<<(unsigned)(sms * 4), 256, 0, s>>>(ta.chg_row, ta.chg_new, ta.chg_old, chg_cap,
                                                               dKoff.as<int64_t>(), dKcur.as<int32_t>(), b_row, b_key,
                                                               dCtl.as<int>());
        note_launch();
        chg_sum_kernel<<<(unsigned)(sms * 8), 256, 0, s>>>(dProbs.as<BProb>(), dGcp.as<int32_t>(), b_row, b_key,
                                                           dX.as<float>(), dLimbs.as<unsigned long long>(),
                                                           dCtl.as<int>());
        note_launch();
      }
    }
    if (concurrent) {
      FUELG_CUDA(cudaEventRecord(ev_join, s2));
      FUELG_CUDA(cudaStreamWaitEvent(s, ev_join, 0));
    }
    // canonical counters every pass; new centres only when another pass follows
    batched_mean_kernel<<<mean_grid, 256, 0, s>>>(dProbs.as<BProb>(), P, dKdb.as<int64_t>(), kd,
                                                  dLimbs.as<unsigned long long>(), dCnt.as<int32_t>(), dC.as<float>(),
                                                  write ? 1 : 0);
    note_launch();
    batched_step_kernel<<<1, 512, 0, s>>>(P, dPchg.as<int32_t>(), dConv.as<int32_t>(), dLast.as<int32_t>(),
                                          dIter.as<int32_t>(), dSt.as<int>() + 1);
    note_launch();
    FUELG_CUDA(cudaGetLastError());
    return ST_OK;
  };
  cudaEventRecord(evh0, s);
  // iteration 1: initial assignment (pairwise order), every point enters
  FUELG_TRY(pass(true, max_iter > 1, grid_for(bps ? bps : 3)));
  int done = 1;
  // autotune: time the candidate shapes on the first middle iterations
  if (!bps && max_iter > 2) {
    float best_ms = 1e30f;
    int best_b = 3;
    for (int b : {2, 4, 8}) {
      if (done >= max_iter - 1) break;
      cudaEvent_t t0, t1;
      cudaEventCreate(&t0);
      cudaEventCreate(&t1);
      cudaEventRecord(t0, s);
      FUELG_TRY(pass(false, true, grid_for(b)));
      cudaEventRecord(t1, s);
      FUELG_CUDA(cudaEventSynchronize(t1));
      float ms = 0.0f;
      cudaEventElapsedTime(&ms, t0, t1);
      cudaEventDestroy(t0);
      cudaEventDestroy(t1);
      done++;
      if (ms < best_ms) {
        best_ms = ms;
        best_b = b;
      }
    }
    bps = best_b;
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tuned[key].blocks_per_sm = bps;
  }
  if (!bps) bps = 3;
  // middle iterations: one captured graph, replayed
  const int middle = std::max(0, max_iter - 1 - done);
  if (middle > 0) {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    FUELG_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    const int64_t l0 = launch_count();
    const int rc = pass(false, true, grid_for(bps));
    cudaError_t ce = cudaStreamEndCapture(s, &graph);
    if (rc != ST_OK) return rc;
    if (ce != cudaSuccess) {
      set_error("graph capture failed: %s", cudaGetErrorString(ce));
      return ST_ECUDA;
    }
    const int64_t per_pass = launch_count() - l0;
    note_launch((int)(-per_pass));  // counted per replay below
    ce = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ce != cudaSuccess) {
      set_error("graph instantiate failed: %s", cudaGetErrorString(ce));
      return ST_ECUDA;
    }
    for (int i = 0; i < middle; i++) {
      ce = cudaGraphLaunch(exec, s);
      if (ce != cudaSuccess) break;
      note_launch((int)per_pass);
    }
    cudaGraphExecDestroy(exec);
    FUELG_CUDA(ce);
    done += middle;
  }
  // last iteration: assignment, no centre update
  if (done < max_iter) {
    FUELG_TRY(pass(false, false, grid_for(bps)));
    done++;
  }
  cudaEventRecord(evh1, s);
  {
    const unsigned ig = (unsigned)std::max<int64_t>(1, std::min<int64_t>(all_items, (int64_t)sms * 8));
    batched_inertia_kernel<<<ig, kItemRows, 0, s>>>(dProbs.as<BProb>(), P, (int)all_items, dX.as<float>(),
                                                    dC.as<float>(), dLab.as<int32_t>(), dInert.as<double>());
    note_launch();
    FUELG_CUDA(cudaGetLastError());
  }
  // results
  std::vector<int32_t> conv(P);
  std::vector<double> inert(P);
  FUELG_CUDA(cudaMemcpyAsync(conv.data(), dConv.p, sizeof(int32_t) * P, cudaMemcpyDeviceToHost, s));
  FUELG_CUDA(cudaMemcpyAsync(inert.data(), dInert.p, sizeof(double) * P, cudaMemcpyDeviceToHost, s));
  // Many labels are widened here and copied straight to the caller's arrays: as
  // 32-bit integers through a host array, the copy, that array's fresh pages and one
  // host loop took 18 ms of 71 for 20 million rows (6 now).  Few come with the other
  // results instead, in one copy, and the host widens them (as it does without room for
  // the wide ones): a copy to an array costs 8 us, a label on the host 0.6 ns.  Calls, us,
  // device / host: one problem of 3000 rows 303 / 291, 30 000 340 / 347, 65 000 332 / 365; 10
  // of 10 000 554 / 530, of 30 000 629 / 719; 60 of 300 1012 / 516, of 5000 1658 / 1329, of
  // 20 000 1945 / 2183.
  Scratch dLab64;
  std::vector<int32_t> lab32;
  if (ls > kHostLabels * (P + 1) && dLab64.alloc(sizeof(int64_t) * ls, s) == ST_OK) {
    widen_labels_kernel<<<(unsigned)((ls + 255) / 256), 256, 0, s>>>(dLab.as<int32_t>(), ls, dLab64.as<int64_t>());
    note_launch();
    FUELG_CUDA(cudaGetLastError());
  } else {
    lab32.resize(ls);
    FUELG_CUDA(cudaMemcpyAsync(lab32.data(), dLab.p, sizeof(int32_t) * ls, cudaMemcpyDeviceToHost, s));
  }
  // host centres leave by one copy (512 pageable ones take 4 ms)
  std::vector<float> hc((size_t)cs);
  FUELG_CUDA(cudaMemcpyAsync(hc.data(), dC.p, sizeof(float) * cs, cudaMemcpyDeviceToHost, s));
  std::vector<char> c_dev(P);
  for (int p = 0; p < P; p++) {
    c_dev[p] = (pointer_kind(probs[p].out_centers, 0, cur_dev) & kDeviceMem) != 0;
    if (c_dev[p])
      FUELG_CUDA(cudaMemcpyAsync(probs[p].out_centers, dC.as<float>() + hp[p].c_off,
                                 sizeof(float) * probs[p].k * probs[p].d, cudaMemcpyDefault, s));
  }
  int hst4[4] = {0, 0, 0, 0};
  FUELG_CUDA(cudaMemcpyAsync(hst4, dSt.p, sizeof(hst4), cudaMemcpyDeviceToHost, s));
  cudaEventRecord(ev1, s);
  FUELG_CUDA(cudaStreamSynchronize(s));
  for (int p = 0; p < P; p++)
    if (!c_dev[p]) memcpy(probs[p].out_centers, hc.data() + hp[p].c_off, sizeof(float) * probs[p].k * probs[p].d);
  const int hst = hst4[0];
  unsigned long long undecided_rows = 0;
  memcpy(&undecided_rows, hst4 + 2, sizeof(undecided_rows));
  if (hst & DEV_TIMEOUT) {
    set_error("a device wait timed out");
    return ST_ETIMEOUT;
  }
  int64_t d2h = (int64_t)sizeof(float) * kd;
  const size_t page = (size_t)std::max<long>(sysconf(_SC_PAGESIZE), 4096);
  for (int p = 0; p < P; p++) {
    fuelg_kmeans_problem& q = probs[p];
    if (!hp[p].active) {
      q.status = ST_ENOTSUP;
      q.out_iters = 0;
      q.out_inertia = 0.0;
      continue;
    }
    if (dLab64.p == nullptr) {
      for (int64_t i = 0; i < q.n; i++) q.out_labels[i] = lab32[hp[p].lab_off + i];
      d2h += (int64_t)sizeof(int32_t) * q.n;
    } else {
      // The pages of an array that was never written are made here, by stores: the
      // copy would have them made one by one on the device's side (54 ms for 160 MB;
      // stores 5, and 5 the copy into present pages).
      const size_t bytes = sizeof(int64_t) * (size_t)q.n;
      volatile char* c = reinterpret_cast<volatile char*>(q.out_labels);
      for (size_t e = 0; e < bytes; e += page) c[e] = 0;
      c[bytes - 1] = 0;
      FUELG_CUDA(cudaMemcpyAsync(q.out_labels, dLab64.as<int64_t>() + hp[p].lab_off, bytes, cudaMemcpyDefault, s));
      d2h += (int64_t)bytes;
    }
    const int it = (!(flags & FUELG_LLOYD_FIXED_ITERS) && conv[p] > 0) ? conv[p] : max_iter;
    q.out_iters = it;
    q.out_inertia = inert[p];
    q.status = ST_OK;
  }
  if (dLab64.p != nullptr) FUELG_CUDA(cudaStreamSynchronize(s));
  if (stats) {
    float ms = 0.0f, hms = 0.0f;
    cudaEventElapsedTime(&ms, ev0, ev1);
    cudaEventElapsedTime(&hms, evh0, evh1);
    stats->device_ms = ms;
    stats->hot_kernel_ms = hms;
    stats->hot_kernel_launches = max_iter;
    stats->h2d_bytes = (int64_t)sizeof(float) * (xs + kd);
    stats->d2h_bytes = d2h;
    int64_t evals = 0;
    for (int p = 0; p < P; p++) evals += hp[p].n * hp[p].k;
    stats->distance_evals = evals * max_iter;
    stats->iterations = max_iter;
    stats->rescored = (int64_t)undecided_rows;
    stats->precision_used = tc_items > 0 ? precision : 0;
    stats->kernel_launches = (int32_t)(launch_count() - launches0);
  }
  return ST_OK;
}
