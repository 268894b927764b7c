// fuelg_knn_tc.cu -- tensor-core (tcgen05 / TMEM / TMA) linear-scan kNN.
//
// A CTA (one per SM) works on blocks of 256 query rows in two halves of 128.  The
// index streams through shared memory in 128-row tiles that both halves share; one
// warp per half issues tcgen05.mma (M=128, N=128, K=16, 16-bit operands, FP32
// accumulators in TMEM) with the query rows as the A operand (in shared memory
// for rows of up to two 64-column chunks, in TMEM for longer ones) and, as a last K
// step, -1 against three BF16 parts of every index row's |x|^2 / 2, so that an
// accumulator holds q.x - |x|^2 / 2 and the screened distance is D~ = |q|^2 minus
// twice it.  Eight epilogue warps compare accumulators with their rows' limits and
// log the few columns that pass; three selection warps fold the logs into each
// query's kk2 best (D~, index) keys and lower its limit.
//
// What bounds it (10^6-point self-join, d = 128, k = 100): with the epilogue's work
// left out the loads and products take 158 ms (256 TFLOP, 1620 TFLOP/s; the MMA
// peak measured here is 2370), with everything but hits 174, in all 238; the form
// before this one, 128 queries per CTA, one lane issuing and norms added in the
// epilogue, 373.  Steps, measured on that workload: issuing from one lane inside a
// divergent branch kept the operands out of uniform registers and took 1170 cycles
// a chunk (446 ms without epilogue); reading norms from shared memory cost 64 ms of
// epilogue; selecting in the epilogue warps stalled both halves' accumulators; a
// larger unrolled epilogue ran into instruction-cache misses.
//
// Exact mode (exact_screen): when every value of the index and the queries is an
// integer of magnitude <= 256 and small enough, every BF16 product, every FP32 partial
// sum (in halves, at most 2^23) and D~ itself are exact, D~ an integer of at most 2^24 --
// D~ then IS fuel's f32 distance (src/distance/squared_euclidean.rs sums the same
// exact integers), whatever the summation order, and the screen keys are final.
// Otherwise the kk2 = kk + margin best screened keys are re-scored with the
// reference's f32 operation order and kept only when a rigorous bound proves
// every unscreened point is strictly worse than the kk-th re-scored key; the
// queries that fail the proof are re-run through the exact scan.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include <cuda_fp16.h>

#include "fuelg_common.cuh"
#include "fuelg_internal.h"
#include "fuelg_select.cuh"
#include "fuelg_tc_common.cuh"

namespace fuelg {

using namespace tcx;

namespace {

constexpr int QM = 128;        // queries per half block (UMMA M)
constexpr int QB = 2 * QM;     // queries per block: two halves share every index tile
constexpr int XN = 128;        // index rows per tile (UMMA N)
constexpr int kEpiWarps = 8;   // epilogue warps: one per half and TMEM lane quarter
constexpr int kSelWarps = 3;   // selection warps
constexpr int kThreadsKT = 32 * (1 + kEpiWarps + kSelWarps + 2);  // producer, epilogue, selection, two issuers
constexpr int kIssue2 = 2 + kEpiWarps + kSelWarps;  // the second half's issuing warp (the first's: 1)
constexpr int kTmemCols = 512;
constexpr int kSmemPerCta = 226 * 1024;
constexpr int kNB = 16;         // columns of the norm operand: one K step
constexpr uint32_t kNormBytes = XN * kNB * 2;  // its 4 KB tile
constexpr int kMaxStages = 12;  // index tiles in shared memory, at most
constexpr int kMinQuantum = 16;  // tiles of a piece, at least
// Index tiles below which a piece may have two: 300 queries, FP16, k = 20 / 150, on 1400 x 100
// 360 / 1129 us in one piece a block, 319 / 892 in four, 333 / 552 in eleven; on 3000 x 100 476 /
// 1100 and, twelve pieces, 327 / 612; 10 000 queries, k = 150, on 3000 x 200 1747 and, three, 1451.
constexpr int kSmallIndex = 64;
// Each query row has two logs of screened (value, column) pairs: its epilogue lane
// fills one while a selection warp folds the other into the row's kept keys.
constexpr int kLog = 192;      // pairs per log: a step adds up to 32
constexpr int kReq = 96;     // pairs from which a log is handed over
constexpr int kSlack = 16;     // keys kept beyond kk so that a selection ends early (kk > 32)
constexpr int kKeep = 256;     // room for kept keys per row
constexpr int kWarmMax = 512;  // groups per row in a warm-up

struct KnnTcArgs {
  int64_t m, n;
  int kc;        // K chunks of 64
  int ks_last;   // K steps of 16 with data in the last chunk (1..4)
  int kk2;       // keys kept per query (the list stride)
  int kout;      // keys written per row: kk2, or kKeep where kk2 > 32
  const int32_t* row_k;  // per query row k (rows keep kk2_of(row_k[q]) <= kk2 keys), or nullptr
  int margin_mode;  // kk2_of mode of this launch
  int exact;     // D~ is exact (integer data)
  int split;     // hi + lo BF16 operands (three products)
  int stages;    // index tiles in shared memory
  int acols;     // TMEM columns of one half's query operand (hi, then lo in split mode)
  int ss;        // query operand in shared memory (two accumulators per half), else in TMEM (one)
  const uint4* qhi;  // BF16 / FP16 query rows [.., dp]
  const uint4* qlo;  // their residuals (split)
  const float* qn2;  // |q|^2 per query row
  float xmax_n2;     // max |x|^2 over the index (filter slack)
  uint64_t* lists;     // [CTA][QB][kKeep + 2 kLog]: kept keys and logs of the rows a CTA works on
  uint64_t* out_keys;  // [piece][QB][kout]: each piece's kept keys
  int spread;          // one block: the epilogue warps its queries are dealt to (spread_query), or 0
  // Work decomposition: CTA c works through pieces [cta_pb[c], cta_pb[c+1]);
  // piece p = query block piece_qb[p] against index tiles [piece_t0[p], piece_t1[p]).
  const int32_t* piece_qb;
  const int32_t* piece_t0;
  const int32_t* piece_t1;
  const int32_t* cta_pb;
  const int32_t* qb_pb;   // first piece of each query block
  unsigned* pub;          // [piece][QB] limit each piece vouches for (vouch), or nullptr
  int concurrent;         // every piece has a CTA of its own
  uint32_t idesc;
  uint32_t idesc_n;  // of the norm step: BF16 in every tier
  int* status;
  const volatile int* cancel;
  uint64_t wait_ns;  // limit of the pipeline waits (pipeline_wait_ns)
};


constexpr float kF16Max = 65504.0f;  // largest finite FP16 value

// Screened keys kept for a query of k neighbours: k plus the margin the
// error-bound proof needs.  Margin modes: 0 exact screened squared distances
// (none), 1 BF16 / split BF16 (max(8, k/8)), 2 FP16 (max(8, k/4): its larger
// screen error needs more ranks between the k-th and the last kept key).
__host__ __device__ __forceinline__ int kk2_of(int k, int mode) {
  const int m = mode == 0 ? 0 : (mode == 1 ? k / 8 : k / 4);
  return mode == 0 ? k : k + (m > 8 ? m : 8);
}


template <int R>
__device__ __forceinline__ void sort_row(uint64_t* __restrict__ kr, int kk2, int lane) {
  uint64_t v[R];
#pragma unroll
  for (int r = 0; r < R; r++) v[r] = lane * R + r < kk2 ? kr[lane * R + r] : KEY_NONE;
  warp_sort_keys<R>(v, lane);
#pragma unroll
  for (int r = 0; r < R; r++)
    if (lane * R + r < kk2) kr[lane * R + r] = v[r];
}

// Sort each row of kk2 (<= 256) keys ascending, one warp per row, over the part of
// it that holds keys (a piece that shares its limit with others keeps few).
__global__ void __launch_bounds__(256) sort_rows_kernel(uint64_t* __restrict__ keys, int64_t rows, int kk2) {
  const int lane = threadIdx.x & 31;
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (row >= rows) return;
  uint64_t* kr = keys + row * kk2;
  int last = 0;  // last run of 32 entries with a key
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int e = 32 * i + lane;
    if (__any_sync(0xffffffffu, e < kk2 && kr[e] != KEY_NONE)) last = i;
  }
  if (last == 0) sort_row<1>(kr, kk2, lane);
  else if (last == 1) sort_row<2>(kr, kk2, lane);
  else if (last <= 3) sort_row<4>(kr, kk2, lane);
  else sort_row<8>(kr, kk2, lane);
}

// The query of row r where the queries of one block are dealt to `warps` epilogue
// warps (four: one half, or all eight), each an equal share: limits after the warm-up
// and lists out are work of 4 to 6 us a row, one row at a time.
__device__ __forceinline__ int spread_query(int r, int warps) { return (r & 31) * warps + (r >> 5); }

constexpr int kMaxSplits = 160;

// k-way merge by one warp of S <= kMaxSplits sorted lists of kk2 keys, list s at
// in + s * stride, into out[0, kk2); lane l owns lists l, l+32, ...
__device__ __forceinline__ void merge_sorted_lists(const uint64_t* __restrict__ in, size_t stride, int S, int kk2,
                                                   uint64_t* __restrict__ out, int lane) {
  int pos[kMaxSplits / 32];
  uint64_t head[kMaxSplits / 32];
#pragma unroll
  for (int t = 0; t < kMaxSplits / 32; t++) {
    const int sp = lane + 32 * t;
    pos[t] = 0;
    head[t] = sp < S ? in[(size_t)sp * stride] : KEY_NONE;
  }
  for (int j = 0; j < kk2; j++) {
    uint64_t mn = head[0];
#pragma unroll
    for (int t = 1; t < kMaxSplits / 32; t++) mn = head[t] < mn ? head[t] : mn;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const uint64_t v = ((uint64_t)__shfl_xor_sync(0xffffffffu, (uint32_t)(mn >> 32), o) << 32) |
                         __shfl_xor_sync(0xffffffffu, (uint32_t)mn, o);
      mn = v < mn ? v : mn;
    }
    if (lane == 0) out[j] = mn;
    if (mn == KEY_NONE) continue;
#pragma unroll
    for (int t = 0; t < kMaxSplits / 32; t++)
      if (head[t] == mn) {  // keys are unique: one list advances
        const int sp = lane + 32 * t;
        pos[t]++;
        head[t] = pos[t] < kk2 ? in[(size_t)sp * stride + pos[t]] : KEY_NONE;
      }
  }
}

// One warp per query: the sorted lists its query block's pieces kept -- piece
// p holds rows in[p][0, QB)[0, stride); the block's pieces are [qb_pb[qb],
// qb_pb[qb + 1]), at most kMaxSplits -- merged into out[q][0, kk2).
__global__ void __launch_bounds__(256) merge_tc_splits_kernel(const uint64_t* __restrict__ in, int64_t m,
                                                              const int32_t* __restrict__ qb_pb, int stride, int kk2,
                                                              uint64_t* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (q >= m) return;
  const int64_t qb = q / QB, row = q - qb * QB;
  const int p0 = qb_pb[qb], S = qb_pb[qb + 1] - p0;
  merge_sorted_lists(in + ((size_t)p0 * QB + row) * stride, (size_t)QB * stride, S, kk2, out + (size_t)q * kk2, lane);
}

// The same for the runs of the FP32 tile scan (sort_and_merge_runs).
__global__ void __launch_bounds__(256) merge_runs_kernel(const uint64_t* __restrict__ in, int64_t m, int qm,
                                                         int64_t nt, int64_t T, int64_t G, int J, int kk,
                                                         uint64_t* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (q >= m) return;
  const int64_t qb = q / qm, row = q - qb * qm;
  const int S = (int)(scan_run_of((qb + 1) * nt - 1, T, G) - scan_run_of(qb * nt, T, G)) + 1;
  merge_sorted_lists(in + ((size_t)qb * J * qm + row) * kk, (size_t)qm * kk, S, kk, out + (size_t)q * kk, lane);
}

// A handed-over log: its length, which of the two, handed over, being folded.
constexpr unsigned kReqCount = 0xffffu, kReqBuf = 0x10000u, kReqSet = 0x20000u, kReqTaken = 0x40000u;

// Key of a logged (q.x - |x|^2 / 2, column) pair, or KEY_NONE where it cannot enter
// (columns past the index, distances above the row's limit).
__device__ __forceinline__ uint64_t log_key(const KnnTcArgs& a, uint2 e, float nq, uint64_t tau) {
  float dt = fmaf(-2.0f, __uint_as_float(e.x), nq);  // D~ = |q|^2 + (|x|^2 - 2 q.x)
  if (!a.exact && dt == dt) dt = fmaxf(dt, 0.0f);
  const float lim = tau == KEY_NONE ? __int_as_float(0x7f800000) : key_dist(tau - 1);
  const uint64_t key = dt <= lim && (int64_t)e.y < a.n ? make_key(dt, e.y) : KEY_NONE;
  return key < tau ? key : KEY_NONE;
}

// A column can enter only if |x|^2 - 2 q.x <= D - |q|^2 (+ slack covering the
// rounding of both forms when the data are not exact integers), D the largest
// distance that can: the limit of q.x - |x|^2 / 2.
__device__ __forceinline__ float screen_limit(const KnnTcArgs& a, float D, float nq) {
  const float th = D - nq;
  return -0.5f * (a.exact ? th : th + (nq + a.xmax_n2 + D) * 3.814697265625e-06f);  // 2^-18
}

// Distance words held by the lanes: their number and range.
template <int N>
__device__ __forceinline__ int word_range(const uint32_t (&hi)[N], uint32_t* hmin, uint32_t* hmax) {
  int total = 0;
  uint32_t lo = 0xffffffffu, up = 0;
#pragma unroll
  for (int i = 0; i < N; i++)
    if (hi[i] != 0xffffffffu) {
      lo = min(lo, hi[i]);
      up = max(up, hi[i]);
      total++;
    }
  *hmin = __reduce_min_sync(0xffffffffu, lo);
  *hmax = __reduce_max_sync(0xffffffffu, up);
  return __reduce_add_sync(0xffffffffu, total);
}

// The S pieces of one query block scan its rows against disjoint parts of the
// index at the same time.  Each vouches for a distance that `rank` = ceil(kk / S)
// of its columns do not exceed; the ceil(kk / rank)-th smallest of these bounds
// the kk-th of the whole index -- about the limit that one scan of all parts so
// far would have, where a piece's own kk-th key is the limit of its part alone.
// A piece's word only comes down; 0xffffffff: nothing to vouch for yet.
__device__ __forceinline__ void vouch(const KnnTcArgs& a, int r, int p, unsigned mine, int lane) {
  if (lane == 0) atomicMin(a.pub + (size_t)p * QB + r, mine);
}
constexpr int kVouch = kMaxSplits / 32;
__device__ __forceinline__ void vouched_words(const KnnTcArgs& a, int r, int p, int lane, uint32_t (&v)[kVouch]) {
  const int p0 = a.qb_pb[a.piece_qb[p]], p1 = a.qb_pb[a.piece_qb[p] + 1];
#pragma unroll
  for (int i = 0; i < kVouch; i++) {
    const int s = p0 + 32 * i + lane;
    v[i] = s < p1 ? *((volatile unsigned*)a.pub + (size_t)s * QB + r) : 0xffffffffu;
  }
}
// The limit that the words vouch for, or 0xffffffff while too few do.
__device__ __forceinline__ uint32_t vouched_cut(const uint32_t (&v)[kVouch], int kk, int rank) {
  const int j = (kk + rank - 1) / rank;
  uint32_t lo, up;
  const int total = word_range(v, &lo, &up);
  int below;
  return total < j ? 0xffffffffu : warp_cut(v, total, j, j / 16, lo, up, &below);
}

// Folds cnt <= kLog logged pairs of row r of piece p into its kept keys (whole warp)
// and lowers the row's limits, to what the block's pieces vouch for too (rank > 0).
__device__ __noinline__ void select_row(const KnnTcArgs& a, uint64_t* list, const uint2* log, int cnt, int r, int p,
                                        int rank, uint64_t* s_tau, volatile float* s_thr, const float* s_nq, const int* s_kk,
                                        volatile int* s_len, int lane) {
  const float nq = s_nq[r];
  const int kk = s_kk[r], len = s_len[r];
  const uint64_t old = s_tau[r];
  uint64_t tau = old;
  int held = len;
  uint32_t vw[kVouch];  // (on their way during the selection)
  if (rank > 0) vouched_words(a, r, p, lane, vw);
  unsigned mine = 0xffffffffu;
  if (kk <= 32) {
    // a sorted list of 32
    uint2 e[kLog / 32];
#pragma unroll
    for (int i = 0; i < kLog / 32; i++)
      e[i] = 32 * i + lane < cnt ? log[32 * i + lane] : make_uint2(0, 0xffffffffu);
    uint64_t kept = len > 0 ? list[lane] : KEY_NONE;
#pragma unroll
    for (int i = 0; i < kLog / 32; i++) {
      if (32 * i >= cnt) break;
      const uint64_t key = 32 * i + lane < cnt ? log_key(a, e[i], nq, tau) : KEY_NONE;
      unsigned in = __ballot_sync(0xffffffffu, key < tau);
      if (__popc(in) > 10) {
        kept = warp_merge32(kept, key, lane);
        const uint64_t kth = shfl_u64(kept, kk - 1);
        tau = kth < tau ? kth : tau;
        continue;
      }
      while (in) {
        const uint64_t nk = shfl_u64(key, __ffs(in) - 1);
        in &= in - 1;
        if (nk < tau) {
          kept = warp_insert32(kept, nk, lane);
          const uint64_t kth = shfl_u64(kept, kk - 1);
          tau = kth < tau ? kth : tau;
        }
      }
    }
    list[lane] = kept;
    held = 1;
    if (rank > 0) mine = (uint32_t)(shfl_u64(kept, rank - 1) >> 32);
  } else {
    constexpr int NL = kLog / 32, NK = kKeep / 32;
    uint64_t key[NL + NK];
#pragma unroll
    for (int i = 0; i < NL; i++) {
      const int o = 32 * i + lane;
      const uint2 e = o < cnt ? log[o] : make_uint2(0, 0);
      key[i] = o < cnt ? log_key(a, e, nq, old) : KEY_NONE;
    }
#pragma unroll
    for (int i = 0; i < NK; i++) {
      const int o = 32 * i + lane;
      key[NL + i] = o < len ? list[o] : KEY_NONE;
    }
    uint32_t hi[NL + NK];
    uint32_t hmin, hmax;
#pragma unroll
    for (int i = 0; i < NL + NK; i++) hi[i] = (uint32_t)(key[i] >> 32);
    const int total = word_range(hi, &hmin, &hmax);
    uint64_t cut = KEY_NONE;  // keys below it are kept
    held = total;
    int below;
    if (rank > 0 && total >= rank) mine = warp_cut(hi, total, rank, rank / 8, hmin, hmax, &below) - 1;
    if (total >= kk) {
      const uint32_t t = warp_cut(hi, total, kk, min(kSlack, kKeep - kk), hmin, hmax, &below);
      cut = (uint64_t)t << 32;
      if (below > kKeep) {
        // more keys share the kk-th distance than there is room for: the kk-th by index
        const uint32_t H = t - 1;
        int less = 0;
#pragma unroll
        for (int i = 0; i < NL + NK; i++) less += hi[i] < H ? 1 : 0;
        less = __reduce_add_sync(0xffffffffu, less);
        uint32_t L = 0;  // largest index word with fewer than kk - less of the tied keys below it
        for (int b = 31; b >= 0; b--) {
          const uint32_t m = L | (1u << b);
          int c = 0;
#pragma unroll
          for (int i = 0; i < NL + NK; i++) c += hi[i] == H && (uint32_t)key[i] < m ? 1 : 0;
          if (__reduce_add_sync(0xffffffffu, c) < kk - less) L = m;
        }
        cut = (((uint64_t)H << 32) | L) + 1;
        below = kk;
      }
      held = below;
      tau = cut < tau ? cut : tau;  // at least kk keys are held below it
    }
    // compact the kept keys: lane offsets by a warp scan of per-lane counts
    int mine = 0;
#pragma unroll
    for (int i = 0; i < NL + NK; i++) mine += key[i] < cut ? 1 : 0;
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    int pos = incl - mine;
#pragma unroll
    for (int i = 0; i < NL + NK; i++)
      if (key[i] < cut) list[pos++] = key[i];
  }
  if (rank > 0) {
    if (mine != 0xffffffffu) vouch(a, r, p, mine, lane);
    const uint32_t t = vouched_cut(vw, kk, rank);  // keys at the distance itself may still enter
    if (t != 0xffffffffu && ((uint64_t)t << 32) < tau) tau = (uint64_t)t << 32;
  }
  __syncwarp();
  if (lane == 0) {
    s_len[r] = held;
    if (tau < old) {
      s_tau[r] = tau;
      s_thr[r] = screen_limit(a, key_dist(tau - 1), nq);
    }
  }
  __syncwarp();
}

// First limits of the warp's rows r0 .. r0 + rows - 1, from the maxima of
// q.x - |x|^2 / 2 over nv <= kWarmMax groups of the piece's first columns, kept where
// the rows' logs will be: each is some column's value, so the kk-th of them bounds
// the kk-th column's.  One row at a time by the whole warp, the next row's values
// on their way.
__device__ __noinline__ void warm_limits(const KnnTcArgs& a, const uint64_t* lists_w, int nv, int rows, int r0, int p,
                                         uint64_t* s_tau, volatile float* s_thr, const float* s_nq, const int* s_kk,
                                         const int* s_rank, int lane) {
  constexpr int N = kWarmMax / 32;
  constexpr size_t qstride = kKeep + 2 * kLog;
  static_assert(kWarmMax * sizeof(float) <= 2 * kLog * sizeof(uint2), "the warm-up's values share the logs' room");
  auto values = [&](int i, float (&f)[N]) {
    const float* vals = reinterpret_cast<const float*>(lists_w + i * qstride + kKeep);
#pragma unroll
    for (int k = 0; k < N; k++)
      f[k] = i < rows && 32 * k + lane < nv ? vals[32 * k + lane] : __int_as_float(0x7fffffff);
  };
  float next[N];
  values(0, next);
  for (int i = 0; i < rows; i++) {
    const int r = r0 + i;
    const float nq = s_nq[r];
    uint32_t hi[N], hmin, hmax;
#pragma unroll
    for (int k = 0; k < N; k++) {
      float dt = fmaf(-2.0f, next[k], nq);
      if (!a.exact) dt = fmaxf(dt, 0.0f);
      hi[k] = next[k] == next[k] && dt == dt ? __float_as_uint(dt) : 0xffffffffu;
    }
    values(i + 1, next);
    const int total = word_range(hi, &hmin, &hmax);
    const int kk = s_kk[r], rank = s_rank[r];
    int below;
    if (total >= kk) {
      // (where pieces share limits, a coarse cut: half as many steps, and the vouched
      // limit replaces it soon: 256 queries on 200 000 x 128, the call 352 us, 374 with
      // kk / 8; where they don't, 10^6 queries at 241.5 ms, 238.6 with kk / 8)
      const int slack = a.pub != nullptr ? kk / 2 : kk / 8;
      const uint32_t t = warp_cut(hi, total, kk, slack, hmin, hmax, &below);
      if (lane == 0) {
        s_tau[r] = (uint64_t)t << 32;
        s_thr[r] = screen_limit(a, __uint_as_float(t - 1), nq);
      }
    }
    if (rank > 0 && total >= rank)
      vouch(a, r, p, rank == 1 ? hmin : warp_cut(hi, total, rank, rank / 8, hmin, hmax, &below) - 1, lane);
  }
  __syncwarp();
  if (a.pub == nullptr) return;
  // what the block's other pieces vouch for; where each has a CTA of its own they
  // got here at about the same time, which is worth a short wait, never more
  const uint64_t since = globaltimer();
  uint32_t vnext[kVouch];
  vouched_words(a, r0, p, lane, vnext);
  for (int i = 0; i < rows; i++) {
    const int r = r0 + i;
    uint32_t v[kVouch];
#pragma unroll
    for (int k = 0; k < kVouch; k++) v[k] = vnext[k];
    if (i + 1 < rows) vouched_words(a, r + 1, p, lane, vnext);
    uint32_t t;
    while ((t = vouched_cut(v, s_kk[r], s_rank[r])) == 0xffffffffu) {
      if (!a.concurrent || __any_sync(0xffffffffu, globaltimer() - since > 10000)) break;
      vouched_words(a, r, p, lane, v);
    }
    if (t != 0xffffffffu && lane == 0 && ((uint64_t)t << 32) < s_tau[r]) {
      s_tau[r] = (uint64_t)t << 32;
      s_thr[r] = screen_limit(a, __uint_as_float(t - 1), s_nq[r]);
    }
  }
  __syncwarp();
}

// Tiles of a piece of `tiles` that are scanned twice, first for the maxima of
// groups of *g columns alone (4 need of them or more where there are as many,
// kWarmMax at most): a limit before any column is logged.  A scan that starts with
// no limit logs kk ln(columns) of them, most in its first tiles.  A tile costs about
// as much as some 30 logged columns, and w tiles leave tiles need / w of them per
// row, which puts the least sum near sqrt(tiles need).  None where the groups would
// be fewer than 5/4 of the `need` that the limit takes.
__device__ __forceinline__ int warm_tiles(int tiles, int need, int* g) {
  int w = (int)(sqrtf((float)tiles * (float)need) * 0.67f);
  w = max(1, min(w, tiles / 2));
  int lg = 2;
  while (((128 * w) >> lg) > kWarmMax || (((128 * w) >> (lg + 1)) >= 4 * need && ((128 * w) >> (lg + 1)) >= 32)) lg++;
  *g = 1 << lg;
  return tiles >= 2 && ((128 * w) >> lg) >= need + need / 4 ? w : 0;
}
// Whether the block of queries from q0 on has rows in its second half.
__device__ __forceinline__ bool second_half(const KnnTcArgs& a, int64_t q0) {
  return a.spread ? a.spread == 8 : q0 + QM < a.m;
}

// The need of piece p: its rank, or kk where a block is one piece.
__device__ __forceinline__ int piece_need(const KnnTcArgs& a, int p) {
  if (a.pub == nullptr) return a.kk2;
  const int S = a.qb_pb[a.piece_qb[p] + 1] - a.qb_pb[a.piece_qb[p]];
  return (a.kk2 + S - 1) / S;
}

// Takes row r's handed-over log, if no other warp has: folds it into the row's kept
// keys and lowers its limits (whole warp).
__device__ __noinline__ void serve_row(const KnnTcArgs& a, uint64_t* lists_cta, int r, volatile unsigned* s_req,
                                       uint64_t* s_tau, volatile float* s_thr, const float* s_nq, const int* s_kk,
                                       volatile int* s_len, const int* s_rank, const int* s_piece, int lane) {
  unsigned v = 0;
  if (lane == 0) {
    v = s_req[r];
    if (v == 0 || (v & kReqTaken) || atomicCAS(const_cast<unsigned*>(s_req) + r, v, v | kReqTaken) != v) v = 0;
  }
  v = __shfl_sync(0xffffffffu, v, 0);
  if (v == 0) return;
  __threadfence_block();
  uint64_t* list = lists_cta + (size_t)r * (kKeep + 2 * kLog);
  const uint2* log = reinterpret_cast<const uint2*>(list + kKeep) + (v & kReqBuf ? kLog : 0);
  select_row(a, list, log, (int)(v & kReqCount), r, s_piece[r], s_rank[r], s_tau, s_thr, s_nq, s_kk, s_len, lane);
  __threadfence_block();
  __syncwarp();
  if (lane == 0) s_req[r] = 0;
}

// Blocks of 256 query rows against ranges of index tiles; warp 0 loads, warps 1 and
// kIssue2 issue one half's products each, warps 2..9 read accumulators, the rest
// select.  Every wait is bounded.
__global__ void __launch_bounds__(kThreadsKT, 1)
    knn_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmQlo,
                  const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmXlo,
                  const __grid_constant__ CUtensorMap tmN, KnnTcArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t b_bytes = XN * BK * 2;  // 16 KB per stage
  const int NS = a.stages;
  const int nb = a.split ? 2 * a.kc : a.kc;  // chunks of a tile, and of a half's operand: hi (then lo)
  const int nacc = a.ss ? 2 : 1;             // accumulators per half
  const uint32_t tile_bytes = nb * b_bytes + kNormBytes;  // x chunks, then the norm operand
  uint8_t* sA = base;                                     // [2][nb] query chunks (a.ss)
  uint8_t* sB = base + (a.ss ? 2 * nb * b_bytes : 0);     // [NS] tiles
  uint8_t* sN = sB + (size_t)NS * tile_bytes;             // the query side of the norm operand
  uint64_t* full = reinterpret_cast<uint64_t*>(sN + kNormBytes);
  uint64_t* empty = full + kMaxStages;
  uint64_t* accf = empty + kMaxStages;
  uint64_t* acce = accf + 4;
  uint64_t* afull = acce + 4;    // [2] a half's query operand is in place
  uint64_t* aempty = afull + 2;  // [2] the products reading it are done (a.ss)
  uint64_t* fin = aempty + 2;    // [2]
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(fin + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  // per query row of the block
  uint64_t* s_tau = reinterpret_cast<uint64_t*>(tmem_holder + 2);  // no key at or above this enters
  volatile float* s_thr = reinterpret_cast<float*>(s_tau + QB);  // least q.x - |x|^2 / 2 that can enter
  volatile unsigned* s_req = reinterpret_cast<unsigned*>(s_tau + QB) + QB;  // 0, or a log handed over (kReq*)
  float* s_nq = reinterpret_cast<float*>(s_tau + QB) + 2 * QB;
  int* s_kk = reinterpret_cast<int*>(s_tau + QB) + 3 * QB;    // keys the row keeps
  volatile int* s_len = reinterpret_cast<int*>(s_tau + QB) + 4 * QB;  // keys kept so far
  int* s_rank = reinterpret_cast<int*>(s_tau + QB) + 5 * QB;  // rank the piece vouches for (0: none)
  int* s_piece = reinterpret_cast<int*>(s_tau + QB) + 6 * QB;  // the row's piece
  volatile int* s_done = s_piece + QB;                         // epilogue warps that have left

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // this CTA's pieces: (query block, index tile range), worked through in order
  const int pb = a.cta_pb[blockIdx.x], pe = a.cta_pb[blockIdx.x + 1];
  constexpr size_t qstride = kKeep + 2 * kLog;
  uint64_t* const lists_cta = a.lists + (size_t)blockIdx.x * QB * qstride;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NS; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 2);  // both halves' products
    }
    for (int b = 0; b < 2 * nacc; b++) {
      mbar_init(&accf[b], 1);
      mbar_init(&acce[b], kEpiWarps / 2);
    }
    for (int h = 0; h < 2; h++) {
      mbar_init(&afull[h], a.ss ? 1 : kEpiWarps / 2);
      mbar_init(&aempty[h], 1);
      mbar_init(&fin[h], 1);
    }
    *abort_flag = 0;
    *s_done = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = threadIdx.x; i < QB; i += kThreadsKT) s_req[i] = 0;
  // Query side of the norm operand: -1 (BF16) against the three parts of every index
  // row's |x|^2 / 2, rows of 32 bytes with their 16-byte halves swapped in rows 4..7
  // of every 8 (32-byte swizzle).
  for (int i = threadIdx.x; i < (int)kNormBytes / 16; i += kThreadsKT) {
    const int row = i >> 1, chunk = (i & 1) ^ ((row >> 2) & 1);
    reinterpret_cast<uint4*>(sN)[i] = chunk == 0 ? make_uint4(0xbf80bf80u, 0xbf80u, 0u, 0u) : make_uint4(0u, 0u, 0u, 0u);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  const uint32_t tmem_acc = tmem_base + (a.ss ? 0 : 2 * a.acols);  // after the two query operands

  if (warp == 0) {
    // The producer and the MMA issuer run as whole warps, so that their addresses
    // stay in uniform registers, and one elected lane issues: as single lanes they
    // took longer to issue a tile than the tensor core to multiply it.
    const bool issue = elect_one();
    if (issue) prefetch_tmap(&tmX);
    const uint64_t pol_q = policy_evict_first(), pol_x = policy_evict_last();
    const uint32_t sa0 = smem_u32(sA), sb0 = smem_u32(sB);
    uint32_t stage = 0, phase = 0, armed = 0, last_ph = 0;
    int loads_a[2] = {0, 0};
    bool ok = true;
    for (int p = pb; ok && p < pe; p++) {
      const int t0 = a.piece_t0[p], t1 = a.piece_t1[p];
      const int q0 = a.piece_qb[p] * QB;
      for (int h = 0; h < 2 && a.ss && (h == 0 || second_half(a, q0)); h++) {
        // the half's query operand, once the last piece's products have read theirs
        ok = loads_a[h] == 0 || mbar_wait(&aempty[h], (uint32_t)((loads_a[h] - 1) & 1), abort_flag, a.wait_ns);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (issue && !*abort_flag) atomicOr(a.status, DEV_TIMEOUT);
          *abort_flag = 1;
          break;
        }
        if (issue) {
          mbar_expect_tx(&afull[h], nb * b_bytes);
          for (int c = 0; c < nb; c++)
            tma_load_2d_hint(sa0 + (h * nb + c) * b_bytes, c < a.kc ? &tmQ : &tmQlo, (c < a.kc ? c : c - a.kc) * BK,
                             q0 + h * QM, &afull[h], pol_q);
        }
        loads_a[h]++;
      }
      if (!ok) break;
      int g;
      const int warm = warm_tiles(t1 - t0, piece_need(a, p), &g);
      for (int i = 0; i < warm + t1 - t0; i++) {
        const int t = t0 + (i < warm ? i : i - warm);
        if ((t & 63) == 63 && a.cancel != nullptr && __any_sync(0xffffffffu, *a.cancel)) {
          if (issue) atomicOr(a.status, DEV_CANCELLED);
          *abort_flag = 1;
        }
        ok = mbar_wait(&empty[stage], phase ^ 1, abort_flag, a.wait_ns);
        ok = __all_sync(0xffffffffu, ok && !*abort_flag);
        if (!ok) {
          if (issue && !*abort_flag) atomicOr(a.status, DEV_TIMEOUT);
          *abort_flag = 1;
          break;
        }
        if (issue) {
          const uint32_t dst = sb0 + stage * tile_bytes;
          mbar_expect_tx(&full[stage], tile_bytes);
          for (int c = 0; c < a.kc; c++)
            tma_load_2d_hint(dst + c * b_bytes, &tmX, c * BK, t * XN, &full[stage], pol_x);
          if (a.split)
            for (int c = 0; c < a.kc; c++)
              tma_load_2d_hint(dst + (a.kc + c) * b_bytes, &tmXlo, c * BK, t * XN, &full[stage], pol_x);
          tma_load_2d_hint(dst + nb * b_bytes, &tmN, 0, t * XN, &full[stage], pol_x);
        }
        armed |= 1u << stage;
        last_ph = (last_ph & ~(1u << stage)) | (phase << stage);
        if (++stage == (uint32_t)NS) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    // never leave a TMA copy writing shared memory: wait (bounded) for the last
    // operand load of each half and the last load armed on every stage
    volatile int never = 0;
    for (int h = 0; h < 2; h++)
      if (loads_a[h] > 0 && !mbar_wait(&afull[h], (uint32_t)((loads_a[h] - 1) & 1), &never))
        atomicOr(a.status, DEV_TIMEOUT);
    for (int s2 = 0; s2 < NS; s2++)
      if (armed & (1u << s2))
        if (!mbar_wait(&full[s2], (last_ph >> s2) & 1u, &never)) atomicOr(a.status, DEV_TIMEOUT);
  } else if (warp == 1 || warp == kIssue2) {
    // One issuing warp per half: a tile's waits, products and commits of both halves
    // in one warp took 1570 cycles, the products themselves 1042 (d = 128).
    const int h = warp == 1 ? 0 : 1;
    const bool issue = elect_one();
    const uint64_t bd0 = smem_desc_sw128(smem_u32(sB));
    const int kc = a.kc, nks_last = a.ks_last;
    const bool split = a.split != 0, ss = a.ss != 0;
    const uint64_t ad0 = smem_desc_sw128(smem_u32(sA)) + h * nb * (b_bytes >> 4);
    const uint64_t an = smem_desc_sw32(smem_u32(sN)), bn0 = smem_desc_sw32(smem_u32(sB) + nb * b_bytes);
    const uint32_t idesc = a.idesc;
    const uint32_t a_tmem = tmem_base + h * a.acols;
    uint32_t stage = 0, phase = 0;
    uint32_t acc = 0, accph = 0;  // this half's next accumulator and its phase
    bool ok = true;
    for (int p = pb; ok && p < pe; p++) {
      const int li = p - pb;
      const int nh = second_half(a, (int64_t)a.piece_qb[p] * QB) ? 2 : 1;  // halves with query rows
      int g;
      const int tiles = a.piece_t1[p] - a.piece_t0[p];
      const int ntile = tiles + warm_tiles(tiles, piece_need(a, p), &g);
      if (h >= nh) break;  // (only the last piece can lack its second half)
      ok = __all_sync(0xffffffffu, mbar_wait(&afull[h], (uint32_t)(li & 1), abort_flag, a.wait_ns));
      for (int t = 0; t < ntile; t++) {
        ok = ok && mbar_wait(&full[stage], phase, abort_flag, a.wait_ns) &&
             mbar_wait(&acce[h * nacc + acc], accph ^ 1, abort_flag, a.wait_ns);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_acc + (h * nacc + acc) * XN;
        const uint64_t bt = bd0 + stage * (tile_bytes >> 4);
        // q_hi . x_hi, split mode: + q_lo . x_hi + q_hi . x_lo; K steps of 16 (8 TMEM
        // columns) that hold data: the zero columns past d add nothing
        for (int j = 0; j < nb; j++) {
          const int c = j < kc ? j : j - kc;
          const uint64_t bd = bt + j * (b_bytes >> 4);
          const uint32_t at = a_tmem + c * (BK / 2);
          const int nks = c == kc - 1 ? nks_last : BK / 16;
          if (issue) {
            if (ss) {
              const uint64_t ad = ad0 + c * (b_bytes >> 4);
              umma_bf16(d_tmem, ad, bd, idesc, j != 0);
              if (nks > 1) umma_bf16(d_tmem, ad + 2, bd + 2, idesc, 1u);
              if (nks > 2) umma_bf16(d_tmem, ad + 4, bd + 4, idesc, 1u);
              if (nks > 3) umma_bf16(d_tmem, ad + 6, bd + 6, idesc, 1u);
              if (split && j < kc) {
                const uint64_t al = ad + kc * (b_bytes >> 4);
                umma_bf16(d_tmem, al, bd, idesc, 1u);
                if (nks > 1) umma_bf16(d_tmem, al + 2, bd + 2, idesc, 1u);
                if (nks > 2) umma_bf16(d_tmem, al + 4, bd + 4, idesc, 1u);
                if (nks > 3) umma_bf16(d_tmem, al + 6, bd + 6, idesc, 1u);
              }
            } else {
              umma_bf16_ta(d_tmem, at, bd, idesc, j != 0);
              if (nks > 1) umma_bf16_ta(d_tmem, at + 8, bd + 2, idesc, 1u);
              if (nks > 2) umma_bf16_ta(d_tmem, at + 16, bd + 4, idesc, 1u);
              if (nks > 3) umma_bf16_ta(d_tmem, at + 24, bd + 6, idesc, 1u);
              if (split && j < kc) {
                const uint32_t al = at + kc * (BK / 2);
                umma_bf16_ta(d_tmem, al, bd, idesc, 1u);
                if (nks > 1) umma_bf16_ta(d_tmem, al + 8, bd + 2, idesc, 1u);
                if (nks > 2) umma_bf16_ta(d_tmem, al + 16, bd + 4, idesc, 1u);
                if (nks > 3) umma_bf16_ta(d_tmem, al + 24, bd + 6, idesc, 1u);
              }
            }
          }
        }
        if (issue) {
          // - |x|^2 / 2, last: the sums before it round as without it
          umma_bf16(d_tmem, an, bn0 + stage * (tile_bytes >> 4), a.idesc_n, 1u);
          umma_commit(&accf[h * nacc + acc]);
          umma_commit(&empty[stage]);
          if (ss && t == ntile - 1) umma_commit(&aempty[h]);
          if (nh == 1) mbar_arrive(&empty[stage]);  // for the half that has no rows
        }
        if (++acc == (uint32_t)nacc) {
          acc = 0;
          accph ^= 1;
        }
        if (++stage == (uint32_t)NS) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    if (!ok) {
      if (issue && !*abort_flag) atomicOr(a.status, DEV_TIMEOUT);
      *abort_flag = 1;
    }
    __syncwarp();
    if (issue) umma_commit(&fin[h]);
    volatile int never = 0;
    if (!mbar_wait(&fin[h], 0, &never)) atomicOr(a.status, DEV_TIMEOUT);
  } else if (warp < 2 + kEpiWarps) {
    // Epilogue: warp w reads query rows 32*(w%4).. (its TMEM lane quarter) of its
    // half over every column and logs the few that pass their row's limit.  It never
    // selects: a selection takes as long as several tiles, and the accumulators of
    // both halves wait for every epilogue warp.
    const int g = warp & 3;
    const int ew = warp - 2;
    const int half = ew >> 2;
    const int row = half * QM + g * 32 + lane;  // query row of the block; TMEM lane g * 32 + lane
    uint64_t* const lists_w = lists_cta + (half * QM + g * 32) * qstride;
    uint2* const logs = reinterpret_cast<uint2*>(lists_w + lane * qstride + kKeep);  // this row's two logs
    const uint32_t lane_addr = (uint32_t)(g * 32) << 16;
    uint32_t acc = 0, accph = 0;  // this half's next accumulator and its phase
    bool alive = true;
    for (int p = pb; alive && p < pe; p++) {
      const int64_t q0 = (int64_t)a.piece_qb[p] * QB;
      const int64_t t0 = a.piece_t0[p], t1 = a.piece_t1[p];
      const int nh = second_half(a, q0) ? 2 : 1;
      int wg;
      const int warm = warm_tiles((int)(t1 - t0), piece_need(a, p), &wg);
      if (half >= nh) continue;
      const int64_t qi = a.spread ? spread_query(row, a.spread) : q0 + row;
      // this warp's rows with a query (may be <= 0)
      const int64_t rows_left = a.spread ? (a.m + a.spread - 1 - (half * 4 + g)) / a.spread : a.m - (q0 + half * QM + g * 32);
      const bool valid = qi < a.m;
      {
        // (!ss) this row's operand into TMEM: the products that read the last
        // piece's are done, their accumulators have been read
        const size_t rowb = (size_t)(q0 + row) * a.kc * (BK * 2 / 16);
        for (int c = 0; c < nb && !a.ss; c++) {
          const uint4* from = (c < a.kc ? a.qhi : a.qlo) + rowb + (c < a.kc ? c : c - a.kc) * (BK * 2 / 16);
          uint32_t v[32];
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const uint4 w = __ldg(from + i);
            v[4 * i] = w.x, v[4 * i + 1] = w.y, v[4 * i + 2] = w.z, v[4 * i + 3] = w.w;
          }
          tmem_st32(tmem_base + lane_addr + half * a.acols + c * (BK / 2), v);
        }
        if (!a.ss) {
          tmem_st_wait();
          tc_fence_before();
        }
        // the row's selection state (its last request is done: see the end of a piece)
        const int kkr = (a.row_k != nullptr && valid) ? kk2_of(a.row_k[qi], a.margin_mode) : a.kk2;
        s_tau[row] = KEY_NONE;
        s_thr[row] = valid ? -__int_as_float(0x7f800000) : __int_as_float(0x7f800000);
        s_nq[row] = valid ? a.qn2[qi] : 0.0f;
        s_kk[row] = kkr;
        s_len[row] = 0;
        const int S = a.qb_pb[a.piece_qb[p] + 1] - a.qb_pb[a.piece_qb[p]];  // pieces of the block
        s_rank[row] = a.pub != nullptr ? (kkr + S - 1) / S : 0;
        s_piece[row] = p;
        __syncwarp();
        if (lane == 0 && !a.ss) mbar_arrive(&afull[half]);
      }
      int na = 0, buf = 0;
      // hands the log over once the row's last request is done
      auto submit = [&]() {
        if (s_req[row] != 0) return;
        __threadfence_block();
        s_req[row] = (unsigned)na | (buf ? kReqBuf : 0u) | kReqSet;
        buf ^= 1;
        na = 0;
      };
      // serves one of this warp's own rows, where it would only wait for the
      // selection warps
      auto help = [&]() {
        const unsigned v = s_req[row];
        const unsigned b = __ballot_sync(0xffffffffu, v != 0 && !(v & kReqTaken));
        if (b)
          serve_row(a, lists_cta, half * QM + g * 32 + __ffs(b) - 1, s_req, s_tau, s_thr, s_nq, s_kk, s_len, s_rank,
                    s_piece, lane);
      };
      const int tiles = (int)(t1 - t0);
      float* wvals = reinterpret_cast<float*>(logs);  // group maxima of the warm-up
      float wmax = -__int_as_float(0x7f800000);
      int nv = 0;
      // a tile's accumulator, and its release
      auto tile_begin = [&]() -> bool {
        const bool ok = mbar_wait(&accf[half * nacc + acc], accph, abort_flag, a.wait_ns);
        if (__any_sync(0xffffffffu, !ok || *abort_flag)) {  // warp-uniform exit
          if (lane == 0 && !*abort_flag) atomicOr(a.status, DEV_TIMEOUT);
          *abort_flag = 1;
          return false;
        }
        tc_fence_after();
        return true;
      };
      auto tile_end = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acce[half * nacc + acc]);
        if (++acc == (uint32_t)nacc) {
          acc = 0;
          accph ^= 1;
        }
      };
      // maxima of q.x - |x|^2 / 2 over 4 and over 16 of 32 columns
      auto maxima = [&](const uint32_t (&r)[32], float (&m4)[8], float& m16a, float& m16b) {
#pragma unroll
        for (int v = 0; v < 8; v++)
          m4[v] = fmaxf(max3_f32(__uint_as_float(r[4 * v]), __uint_as_float(r[4 * v + 1]),
                                 __uint_as_float(r[4 * v + 2])),
                        __uint_as_float(r[4 * v + 3]));
        m16a = fmaxf(max3_f32(m4[0], m4[1], m4[2]), m4[3]);
        m16b = fmaxf(max3_f32(m4[4], m4[5], m4[6]), m4[7]);
      };
      const uint32_t tacc0 = tmem_acc + lane_addr + half * nacc * XN;
      for (int i = 0; i < warm; i++) {
        if (!tile_begin()) {
          alive = false;
          break;
        }
#pragma unroll 1
        for (int c0 = 0; c0 < XN; c0 += 32) {
          uint32_t r[32];
          tmem_ld32_nowait(tacc0 + acc * XN + c0, r);
          tmem_ld_wait();
          tmem_regs_ready32(r);
          float m4[8], m16a, m16b;
          maxima(r, m4, m16a, m16b);
          if (wg <= 8) {
#pragma unroll
            for (int v = 0; v < 8; v += 2) {
              wvals[nv++] = wg == 8 ? fmaxf(m4[v], m4[v + 1]) : m4[v];
              if (wg == 4) wvals[nv++] = m4[v + 1];
            }
          } else if (wg == 16) {
            wvals[nv++] = m16a;
            wvals[nv++] = m16b;
          } else {
            wmax = max3_f32(m16a, m16b, wmax);
            if (((i * XN + c0 + 32) & (wg - 1)) == 0) {
              wvals[nv++] = wmax;
              wmax = -__int_as_float(0x7f800000);
            }
          }
        }
        tile_end();
      }
      if (!alive) break;
      if (warm > 0) {
        warm_limits(a, lists_w, nv, (int)(rows_left < 32 ? (rows_left > 0 ? rows_left : 0) : 32), half * QM + g * 32, p, s_tau, s_thr,
                    s_nq, s_kk, s_rank, lane);
      }
      for (int i = 0; i < tiles; i++) {
        const int p0 = (int)(t0 + i) * XN;
        if (!tile_begin()) {
          alive = false;
          break;
        }
        const uint32_t taddr = tacc0 + acc * XN;
        const float thr = s_thr[row];
        // The loop is kept short (its instructions, the other roles' and the
        // selections' share one cache): 32 columns a step, and a 4-column group with
        // a hit in any row is read again from TMEM.
#pragma unroll 1
        for (int c0 = 0; c0 < XN; c0 += 32) {
          uint32_t r[32];
          tmem_ld32_nowait(taddr + c0, r);
          tmem_ld_wait();
          tmem_regs_ready32(r);
          float m4[8], m16a, m16b;
          maxima(r, m4, m16a, m16b);
          if (!__any_sync(0xffffffffu, fmaxf(m16a, m16b) >= thr)) continue;
          unsigned hits = 0;
#pragma unroll
          for (int v = 0; v < 8; v++) hits |= m4[v] >= thr ? 1u << v : 0u;
          hits = __reduce_or_sync(0xffffffffu, hits);
          uint2* const log = logs + buf * kLog;
#pragma unroll 1
          while (hits) {
            const int c = c0 + 4 * (__ffs(hits) - 1);
            hits &= hits - 1;
            uint32_t f[4];
            tmem_ld4_nowait(taddr + c, f);
            tmem_ld_wait();
            tmem_regs_ready4(f);
#pragma unroll
            for (int j = 0; j < 4; j++)
              if (__uint_as_float(f[j]) >= thr) log[na++] = make_uint2(f[j], p0 + c + j);
          }
          if (__any_sync(0xffffffffu, na >= kReq)) {
            if (na >= kReq) submit();
            // a step adds up to 32 pairs: without that much room, wait for the selection
            if (__any_sync(0xffffffffu, na > kLog - 32)) {
              const uint64_t since = globaltimer();
              while (__any_sync(0xffffffffu, na > kLog - 32)) {
                if (na > kLog - 32) submit();
                help();
                if (*abort_flag || globaltimer() - since > kWaitNs) {
                  if (!*abort_flag) atomicOr(a.status, DEV_TIMEOUT);
                  *abort_flag = 1;
                  alive = false;
                }
                alive = __all_sync(0xffffffffu, alive);
                if (!alive) break;
              }
            }
          }
          if (!alive) break;
        }
        if (!alive) break;
        tile_end();
      }
      if (!alive) break;
      // the rows' last selections
      {
        const uint64_t since = globaltimer();
        while (__any_sync(0xffffffffu, s_req[row] != 0)) {
          help();
          if (*abort_flag || globaltimer() - since > kWaitNs) {
            if (!*abort_flag) atomicOr(a.status, DEV_TIMEOUT);
            *abort_flag = 1;
            alive = false;
          }
          alive = __all_sync(0xffffffffu, alive);
          if (!alive) break;
        }
      }
      if (!alive) break;
      __threadfence_block();
      __syncwarp();
      // kept keys out, one query at a time per warp: a sorted list, or (kk > 32)
      // the kept keys and what is left in the log, unsorted; slots past them are
      // KEY_NONE.  Piece p's lists sit at rows [p*QB, p*QB + QB) of the output, in
      // query order.
      constexpr int NK = kKeep / 32, NL = kLog / 32;
      uint64_t nkey[NK];
      uint2 nent[NL];
      const int rows = (int)(rows_left < 32 ? rows_left : 32);  // (may be <= 0)
      auto fetch = [&](int src) {  // a row's kept keys and what is left in its log
        const uint64_t* list = lists_w + src * qstride;
        const int len = src < rows ? s_len[half * QM + g * 32 + src] : 0;
        const int sna = __shfl_sync(0xffffffffu, na, src & 31), sbuf = __shfl_sync(0xffffffffu, buf, src & 31);
        const uint2* log = reinterpret_cast<const uint2*>(list + kKeep) + sbuf * kLog;
        const bool sorted = src < rows && s_kk[half * QM + g * 32 + src] <= 32;
#pragma unroll
        for (int k = 0; k < NK; k++)
          nkey[k] = (sorted ? k == 0 && len > 0 : 32 * k + lane < len) ? list[32 * k + lane] : KEY_NONE;
#pragma unroll
        for (int k = 0; k < NL; k++)
          nent[k] = src < rows && 32 * k + lane < sna ? log[32 * k + lane] : make_uint2(0x7fffffffu, 0xffffffffu);
      };
      fetch(0);
      for (int src = 0; src < rows; src++) {
        const int r = half * QM + g * 32 + src;
        const int left = __shfl_sync(0xffffffffu, na, src);
        const int sbuf = __shfl_sync(0xffffffffu, buf, src);
        const int skk = s_kk[r];
        uint64_t* list = lists_w + src * qstride;
        uint64_t* to = a.out_keys + ((size_t)p * QB + (a.spread ? spread_query(r, a.spread) : r)) * a.kout;
        uint64_t key[NK], add[NL];
        const uint64_t stau = s_tau[r];
        const float snq = s_nq[r];
#pragma unroll
        for (int k = 0; k < NK; k++) key[k] = nkey[k];
#pragma unroll
        for (int k = 0; k < NL; k++) add[k] = log_key(a, nent[k], snq, stau);  // (a NaN value: no key)
        fetch(src + 1);
        if (skk <= 32) {
          uint64_t kept = key[0];
#pragma unroll
          for (int k = 0; k < NL; k++)
            if (32 * k < left && __any_sync(0xffffffffu, add[k] < stau)) kept = warp_merge32(kept, add[k], lane);
          for (int o = lane; o < a.kout; o += 32) to[o] = o < skk ? kept : KEY_NONE;  // (o < skk: o == lane)
        } else if (s_len[r] + left > a.kout) {
          const uint2* log = reinterpret_cast<const uint2*>(list + kKeep) + sbuf * kLog;
          select_row(a, list, log, left, r, p, 0, s_tau, s_thr, s_nq, s_kk, s_len, lane);
          const int len = s_len[r];
          for (int o = lane; o < a.kout; o += 32) to[o] = o < len ? list[o] : KEY_NONE;
        } else {
          // kept keys, then the log's (kout == kKeep)
          const int len = s_len[r];
#pragma unroll
          for (int k = 0; k < NK; k++)
            if (32 * k + lane < len || 32 * k + lane >= len + left) to[32 * k + lane] = key[k];
#pragma unroll
          for (int k = 0; k < NL; k++)
            if (32 * k + lane < left) to[len + 32 * k + lane] = add[k];
        }
      }
      __syncwarp();
    }
    __syncwarp();
    if (lane == 0) atomicAdd(const_cast<int*>(s_done), 1);
  } else {
    // Selection warps: take any row's log that was handed over.
    const int sw = warp - 2 - kEpiWarps;
    int at = sw * (QB / kSelWarps);  // start at different rows
    while (!*abort_flag) {
      // rows at + lane, + 32, ...: the first one with an unclaimed request
      int pick = -1;
#pragma unroll
      for (int i = 0; i < QB / 32; i++) {
        const int r = (at + i * 32 + lane) & (QB - 1);
        const unsigned v = s_req[r];
        const unsigned b = __ballot_sync(0xffffffffu, v != 0 && !(v & kReqTaken));
        if (b) {
          pick = (at + i * 32 + __ffs(b) - 1) & (QB - 1);
          break;
        }
      }
      if (pick < 0) {
        if (*s_done == kEpiWarps) break;
        __nanosleep(200);
        continue;
      }
      at = (pick + 1) & (QB - 1);
      serve_row(a, lists_cta, pick, s_req, s_tau, s_thr, s_nq, s_kk, s_len, s_rank, s_piece, lane);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

// Rows -> BF16 copy padded to dp columns and rows_pad rows (zeros), |row|^2 in
// FP32, plus an integer-data census: flags[0] |= 1 for a non-integer or |v| > 256, 2
// for a negative value, flags[1] = max |v| (as float bits; non-negative so integer
// order works).
template <bool F16>
__global__ void knn_prep_kernel(const float* __restrict__ X, int64_t rows, int64_t rows_pad, int d, int dp,
                                void* __restrict__ out, __nv_bfloat16* __restrict__ out_lo,
                                float* __restrict__ n2, int* __restrict__ flags, int spread) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  int bad = 0;
  float vmax = 0.0f;
  for (int64_t r = (int64_t)blockIdx.x * nw + warp; r < rows_pad; r += (int64_t)gridDim.x * nw) {
    const int64_t src = spread ? spread_query((int)r, spread) : r;
    float acc = 0.0f;
    for (int c = lane; c < dp; c += 32) {
      const float x = (src < rows && c < d) ? __ldg(X + src * d + c) : 0.0f;
      if (F16) {
        static_cast<__half*>(out)[r * dp + c] = __float2half_rn(x);
      } else {
        const __nv_bfloat16 hi = __float2bfloat16_rn(x);
        static_cast<__nv_bfloat16*>(out)[r * dp + c] = hi;
        if (out_lo) out_lo[r * dp + c] = __float2bfloat16_rn(x - __bfloat162float(hi));
      }
      acc = fmaf(x, x, acc);
      if (x != rintf(x) || fabsf(x) > 256.0f) bad |= 1;
      if (x < 0.0f) bad |= 2;
      vmax = fmaxf(vmax, fabsf(x));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane == 0) n2[src] = acc;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    bad |= __shfl_xor_sync(0xffffffffu, bad, off);
    vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, off));
  }
  if (lane == 0) {
    if (bad) atomicOr(&flags[0], bad);
    atomicMax(&flags[1], __float_as_int(vmax));
  }
}

// |x|^2 / 2 as three BF16 parts, the leading bits first (together all 24 bits of the
// FP32 value), in the first three of a row's kNB columns.  A norm that is not finite
// goes whole into the first part.
__global__ void norm_parts_kernel(const float* __restrict__ n2, int64_t rows, uint16_t* __restrict__ out) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  float v = 0.5f * n2[r];
  uint32_t part[3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    part[i] = __bfloat16_as_ushort(h);
    v = isfinite(v) ? v - __bfloat162float(h) : 0.0f;
  }
  uint4* o = reinterpret_cast<uint4*>(out + r * kNB);
  o[0] = make_uint4(part[0] | part[1] << 16, part[2], 0u, 0u);
  o[1] = make_uint4(0u, 0u, 0u, 0u);
}

// Re-score the kk2 screened candidates of every query with the reference's
// own f32 order (8-lane groups = fuel's SIMD lanes, 4 candidates per warp
// step), sort them by (distance, index) in the metric's domain, and prove that
// no unscreened point can displace the kk-th: every unscreened point has
// D~ >= D~_last, so its reference distance is >= D~_last - E_max.  Queries that
// fail the proof are flagged for the exact scan.
template <int ORDER>
__global__ void knn_rescore_kernel(const float* __restrict__ Q, const float* __restrict__ X, int64_t n, int d,
                                   int64_t m, int kk, int kk2, const int32_t* __restrict__ row_k, int margin_mode,
                                   int metric, const uint64_t* __restrict__ keys_in, int in_stride,
                                   uint64_t* __restrict__ keys_out, const float* __restrict__ qn2, float xmax_norm,
                                   float xmax_n2, float alpha, float beta, float gamma, float abs_a, float abs_u,
                                   int32_t* __restrict__ redo, int32_t* __restrict__ nredo) {
  extern __shared__ __align__(16) float qsm[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int64_t qi = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (qi >= m) return;
  float* qs = qsm + (size_t)wib * (d + 4);
  for (int e = lane; e < d; e += 32) qs[e] = __ldg(Q + qi * d + e);
  __syncwarp();
  const uint64_t* kin = keys_in + qi * in_stride;
  uint64_t* kout = keys_out + qi * kk2;
  // this row's k and kept keys (the list stride stays kk2)
  const int kq = row_k != nullptr ? row_k[qi] : kk;
  const int kk2q = row_k != nullptr ? kk2_of(kq, margin_mode) : kk2;
  for (int c = kk2q + lane; c < kk2; c += 32) kout[c] = KEY_NONE;
  // exact keys of the candidates, written in place of the screened ones
  const int l = lane & 7, grp = lane >> 3;
  float last_screen = 0.0f;
  for (int c0 = 0; c0 < kk2q; c0 += 4) {
    const int c = c0 + grp;
    const uint64_t sk = c < kk2q ? kin[c] : KEY_NONE;
    // a key that names no index row (never produced by a completed screen)
    // is treated as empty, so no read leaves X
    const bool real = sk != KEY_NONE && (int64_t)key_idx(sk) < n;
    const uint32_t idx = real ? key_idx(sk) : 0u;
    const float* x = X + (int64_t)idx * d;
    const int sd = d & ~7;
    float acc = 0.0f;
    for (int i = l; i < sd; i += 8) {
      const float df = __fsub_rn(qs[i], __ldg(x + i));
      acc = ORDER == ORDER_X86 ? __fmaf_rn(df, df, acc) : __fadd_rn(sq_rn(df), acc);
    }
    float s = __shfl_sync(0xffffffffu, acc, lane & ~7);
#pragma unroll
    for (int t = 1; t < 8; t++) s = __fadd_rn(s, __shfl_sync(0xffffffffu, acc, (lane & ~7) + t));
    for (int i = sd; i < d; i++) {
      const float df = __fsub_rn(qs[i], __ldg(x + i));
      s = ORDER == ORDER_X86 ? __fmaf_rn(df, df, s) : __fadd_rn(s, sq_rn(df));
    }
    if (metric == METRIC_EUCLIDEAN) s = __fsqrt_rn(s);
    if (l == 0 && c < kk2q) kout[c] = real ? make_key(s, idx) : KEY_NONE;
    if (real) last_screen = fmaxf(last_screen, key_dist(sk));
  }
  // the largest screened distance kept (candidates are sorted by screened key)
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) last_screen = fmaxf(last_screen, __shfl_xor_sync(0xffffffffu, last_screen, off));
  __syncwarp();
  // sort the kk2 exact keys (small: insertion sort by lane 0)
  if (lane == 0) {
    for (int a1 = 1; a1 < kk2q; a1++) {
      const uint64_t v = kout[a1];
      int b = a1 - 1;
      while (b >= 0 && kout[b] > v) {
        kout[b + 1] = kout[b];
        b--;
      }
      kout[b + 1] = v;
    }
    // proof: needed unless every point was kept; a list that is neither full nor the
    // whole index missed points whose screened value was NaN
    const int64_t room = n < kk2q ? n : kk2q;
    if (kin[room - 1] == KEY_NONE) {
      redo[atomicAdd(nredo, 1)] = (int32_t)qi;
    } else if (n > kk2q) {
      const float nq = qn2[qi];
      const float qn = sqrtf(nq);
      const float e = (alpha * qn * xmax_norm + beta * (nq + xmax_n2)) * (1.0f + gamma) + gamma * last_screen +
                      abs_a * (qn + xmax_norm) + abs_u;
      const float lower = last_screen - e;  // every unscreened point's reference squared distance is >= this
      const uint64_t kth = kout[kq - 1];
      bool ok;
      if (metric == METRIC_EUCLIDEAN) ok = kth != KEY_NONE && lower > 0.0f && key_dist(kth) < __fsqrt_rd(lower);
      else ok = kth != KEY_NONE && key_dist(kth) < lower;
      if (!ok) redo[atomicAdd(nredo, 1)] = (int32_t)qi;
    }
  }
}

__global__ void gather_rows_kernel(const float* __restrict__ Q, int d, const int32_t* __restrict__ rows,
                                   const int32_t* __restrict__ nrows, float* __restrict__ out) {
  const int cnt = *nrows;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < (int64_t)cnt * d;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e / d, c = e - r * d;
    out[e] = Q[(int64_t)rows[r] * d + c];
  }
}

__global__ void scatter_keys_kernel(const uint64_t* __restrict__ src, int kk, int kk2,
                                    const int32_t* __restrict__ rows, int cnt, uint64_t* __restrict__ dst) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (int64_t)cnt * kk2) return;
  const int64_t r = e / kk2, j = e - r * kk2;
  dst[(int64_t)rows[r] * kk2 + j] = j < kk ? src[r * kk + j] : KEY_NONE;
}

}  // namespace

int sort_and_merge_runs(uint64_t* lists, int64_t m, int qm, int64_t nt, int64_t T, int64_t G, int J, int kk,
                        uint64_t* keys, cudaStream_t stream) {
  const int64_t rows = lists == keys ? m : (m + qm - 1) / qm * J * qm;
  sort_rows_kernel<<<(unsigned)((rows * 32 + 255) / 256), 256, 0, stream>>>(lists, rows, kk);
  note_launch();
  if (lists != keys) {
    merge_runs_kernel<<<(unsigned)((m * 32 + 255) / 256), 256, 0, stream>>>(lists, m, qm, nt, T, G, J, kk, keys);
    note_launch();
  }
  FUELG_CUDA(cudaGetLastError());
  return ST_OK;
}

namespace {
// Shared memory of knn_tc_kernel beside the query chunks and the index tiles.
constexpr size_t kFixedSmem = 1024 + kNormBytes + 8 * (2 * kMaxStages + 16) + 16 + QB * 36 + 16;
// Whether the screened distances of integers up to qmax and xmax in magnitude, in d
// dimensions (dp with padding), are fuel's f32 distances: partial sums and norms are
// exact below 2 dp V^2 < 2^24, V the larger, and so is |q - x|^2 <= d V^2 where no value
// is negative.  With both signs it can reach d (qmax + xmax)^2, up to 4 d V^2: fuel's sums
// round once they pass 2^24, in an order that D~ does not follow (d = 128, values of
// 255 and -254: a third of the distances differ).  Up to 2^24 nothing rounds: the
// products' sums in halves stay within (qmax + xmax)^2 d / 2.
bool exact_screen(int d, int dp, double qmax, double xmax, bool negative) {
  const double v = std::max(qmax, xmax);
  return 2.0 * dp * v * v < 16777216.0 && (!negative || d * (qmax + xmax) * (qmax + xmax) <= 16777216.0);
}
// TMEM columns of one half's query operand: two 16-bit values per column.
int query_cols(int d, int split) { return (split ? 2 : 1) * ((d + BK - 1) / BK) * (BK / 2); }
int margin_mode_of(int tier) { return tier == TC_F16 ? 2 : 1; }
}  // namespace

bool knn_tc_supported(int64_t n, int d, int kk, int tier) {
  if (d < 32 || d > 256 || kk < 1) return false;
  // TMA row coordinates are signed 32-bit: the padded index must stay below 2^31 rows
  if (n >= (1ll << 31) - 4096) return false;
  // kept keys per query are selected 8 per lane by one warp
  if (kk2_of(kk, margin_mode_of(tier)) > 32 * kSel) return false;
  // both halves' query operands beside two accumulators
  return 2 * query_cols(d, tier == TC_SPLIT) + 2 * XN <= kTmemCols;
}

// Top-kk keys of every query via the tensor-core screen.  out_keys: [m, kk]
// (device).  X32/Q32: the f32 rows (for the exact re-score).
struct TcIndex {
  int64_t n = 0, npad = 0;
  int d = 0, dp = 0;
  __nv_bfloat16* xb = nullptr;  // [npad, dp] BF16, zero padded
  __nv_bfloat16* xlo = nullptr; // [npad, dp] BF16 of x - xb (split tier; built on first use)
  __half* xh = nullptr;         // [npad, dp] FP16 (FP16 tier; built on first use)
  float* xn2 = nullptr;         // [npad] FP32 |x|^2 (padded rows 0)
  bool integer = false;         // every value an integer with |v| <= 256
  bool negative = false;        // some value below 0
  float vmax = 0.0f;            // max |v|
  float xmax_n2 = 0.0f;         // max |x|^2
  uint16_t* xnorm = nullptr;    // [npad, 16] |x|^2 / 2 as three BF16 parts, then zeros
  CUtensorMap tmX, tmXlo, tmXh, tmN;
};

int knn_tc_index_class(const TcIndex* t) {
  if (t->integer) return TC_CLASS_INTEGER;
  return t->vmax <= kF16Max ? TC_CLASS_F16_RANGE : TC_CLASS_WIDE;
}

bool knn_tc_index_screens(const TcIndex* t) { return t->xmax_n2 < 1e37f; }

void knn_tc_index_free(TcIndex* t) {
  if (!t) return;
  if (t->xb) cudaFree(t->xb);
  if (t->xn2) cudaFree(t->xn2);
  if (t->xlo) cudaFree(t->xlo);
  if (t->xh) cudaFree(t->xh);
  if (t->xnorm) cudaFree(t->xnorm);
  delete t;
}

int knn_tc_index_build(const float* X32, int64_t n, int d, cudaStream_t stream, TcIndex** out) {
  *out = nullptr;
  TcIndex* t = new TcIndex();
  struct Guard {
    TcIndex*& t;
    ~Guard() { knn_tc_index_free(t); }
  } guard{t};
  t->n = n;
  t->d = d;
  t->dp = ((d + BK - 1) / BK) * BK;
  t->npad = ((n + XN - 1) / XN) * XN;
  FUELG_CUDA(cudaMalloc(&t->xb, (size_t)t->npad * t->dp * 2));
  FUELG_CUDA(cudaMalloc(&t->xn2, sizeof(float) * t->npad));
  FUELG_CUDA(cudaMalloc(&t->xnorm, (size_t)t->npad * kNB * 2));
  Scratch flags;
  FUELG_TRY(flags.alloc(sizeof(int) * 2, stream));
  FUELG_CUDA(cudaMemsetAsync(flags.p, 0, sizeof(int) * 2, stream));
  knn_prep_kernel<false><<<8 * 152, 256, 0, stream>>>(X32, n, t->npad, d, t->dp, t->xb, nullptr, t->xn2,
                                                      flags.as<int>(), 0);
  ::fuelg::note_launch();
  FUELG_CUDA(cudaGetLastError());
  int hf[2];
  FUELG_CUDA(cudaMemcpyAsync(hf, flags.p, sizeof(hf), cudaMemcpyDeviceToHost, stream));
  std::vector<float> h((size_t)t->npad);
  FUELG_CUDA(cudaMemcpyAsync(h.data(), t->xn2, sizeof(float) * t->npad, cudaMemcpyDeviceToHost, stream));
  FUELG_CUDA(cudaStreamSynchronize(stream));
  t->integer = (hf[0] & 1) == 0;
  t->negative = (hf[0] & 2) != 0;
  memcpy(&t->vmax, &hf[1], sizeof(float));
  for (float v : h) t->xmax_n2 = std::max(t->xmax_n2, v);
  norm_parts_kernel<<<(unsigned)((t->npad + 255) / 256), 256, 0, stream>>>(t->xn2, t->npad, t->xnorm);
  ::fuelg::note_launch();
  FUELG_CUDA(cudaGetLastError());
  FUELG_TRY(make_map_norm(&t->tmN, t->xnorm, t->npad, XN));
  FUELG_TRY(make_map_bf16(&t->tmX, t->xb, t->npad, t->dp, XN));
  *out = t;
  t = nullptr;  // owned by the caller now
  return ST_OK;
}

// Adds the BF16 residual copy x - BF16(x) of the index (split tier), once.
int knn_tc_index_add_lo(TcIndex* t, const float* X32, cudaStream_t stream) {
  if (t->xlo) return ST_OK;
  FUELG_CUDA(cudaMalloc(&t->xlo, (size_t)t->npad * t->dp * 2));
  Scratch hi, n2, flags;
  FUELG_TRY(hi.alloc((size_t)t->npad * t->dp * 2, stream));
  FUELG_TRY(n2.alloc(sizeof(float) * t->npad, stream));
  FUELG_TRY(flags.alloc(sizeof(int) * 2, stream));
  knn_prep_kernel<false><<<8 * 152, 256, 0, stream>>>(X32, t->n, t->npad, t->d, t->dp, hi.as<__nv_bfloat16>(),
                                                      t->xlo, n2.as<float>(), flags.as<int>(), 0);
  ::fuelg::note_launch();
  FUELG_CUDA(cudaGetLastError());
  FUELG_TRY(make_map_bf16(&t->tmXlo, t->xlo, t->npad, t->dp, XN));
  FUELG_CUDA(cudaStreamSynchronize(stream));
  return ST_OK;
}

int knn_tc_index_add_f16(TcIndex* t, const float* X32, cudaStream_t stream) {
  if (t->xh) return ST_OK;
  if (!(t->vmax <= kF16Max)) {
    set_error("index values exceed the FP16 range (max |v| = %g)", (double)t->vmax);
    return ST_ENOTSUP;
  }
  FUELG_CUDA(cudaMalloc(&t->xh, (size_t)t->npad * t->dp * 2));
  Scratch n2, flags;
  FUELG_TRY(n2.alloc(sizeof(float) * t->npad, stream));
  FUELG_TRY(flags.alloc(sizeof(int) * 2, stream));
  knn_prep_kernel<true><<<8 * 152, 256, 0, stream>>>(X32, t->n, t->npad, t->d, t->dp, t->xh, nullptr,
                                                     n2.as<float>(), flags.as<int>(), 0);
  ::fuelg::note_launch();
  FUELG_CUDA(cudaGetLastError());
  FUELG_TRY(make_map_bf16(&t->tmXh, t->xh, t->npad, t->dp, XN));  // 2-byte elements: same box geometry
  FUELG_CUDA(cudaStreamSynchronize(stream));
  return ST_OK;
}

int knn_tc_topk(const TcIndex* ti, const float* Q32, int64_t m, const float* X32, int kk, int order, int metric,
                int tier, uint64_t* out_keys, int* dev_status, cudaStream_t stream, int64_t* rescored,
                int* exact_out, const int32_t* row_k) {
  const int64_t n = ti->n;
  const int d = ti->d;
  const int dp = ti->dp;
  if (!knn_tc_index_screens(ti)) {
    // norms near or past the FP32 range have no useful screen: the exact scan answers
    set_error("index norms exceed the tensor-core screen's range (max |x|^2 = %g)", (double)ti->xmax_n2);
    return ST_ENOTSUP;
  }
  const int kc = dp / BK;
  // One block's queries are dealt to the epilogue warps: to all eight where that saves
  // more than the second half's products and tests cost.  Kernel, us, 2 10^6 x 96, k = 10,
  // rows in order / four / eight warps: FP16 16 queries 178 / 125 / -, 32 253 / 146 / 138,
  // 128 281 / 284 / 214; split BF16, three products, 32 328 / 223 / 263, 64 353 / 269 / 288,
  // 128 366 / 368 / 339.  200 000 x 128, 32 queries: the call 315 -> 199.
  const int spread = m > QB ? 0 : m > (tier == TC_SPLIT ? 64 : 16) ? 8 : 4;
  const int64_t mpad = spread == 8 ? QB : ((m + QM - 1) / QM) * QM;
  const bool f16 = tier == TC_F16;
  int split = tier == TC_SPLIT ? 1 : 0;
  if (split && !ti->xlo) {
    set_error("split-BF16 kNN needs the index residual copy");
    return ST_ENOTSUP;
  }
  if (f16 && !ti->xh) {
    set_error("FP16 kNN needs the index FP16 copy");
    return ST_ENOTSUP;
  }
  Scratch qb, qlo, qn2, flags;
  FUELG_TRY(qb.alloc((size_t)mpad * dp * 2, stream));
  if (split) FUELG_TRY(qlo.alloc((size_t)mpad * dp * 2, stream));
  FUELG_TRY(qn2.alloc(sizeof(float) * mpad, stream));
  FUELG_TRY(flags.alloc(sizeof(int) * 2, stream));
  FUELG_CUDA(cudaMemsetAsync(flags.p, 0, sizeof(int) * 2, stream));
  if (f16)
    knn_prep_kernel<true><<<8 * 152, 256, 0, stream>>>(Q32, m, mpad, d, dp, qb.p, nullptr, qn2.as<float>(),
                                                       flags.as<int>(), spread);
  else
    knn_prep_kernel<false><<<8 * 152, 256, 0, stream>>>(Q32, m, mpad, d, dp, qb.p,
                                                        split ? qlo.as<__nv_bfloat16>() : nullptr, qn2.as<float>(),
                                                        flags.as<int>(), spread);
  ::fuelg::note_launch();
  FUELG_CUDA(cudaGetLastError());
  int hf[2];
  FUELG_CUDA(cudaMemcpyAsync(hf, flags.p, sizeof(hf), cudaMemcpyDeviceToHost, stream));
  FUELG_CUDA(cudaStreamSynchronize(stream));
  float qmax;
  memcpy(&qmax, &hf[1], sizeof(float));
  if (f16 && !(qmax <= kF16Max)) {
    set_error("query values exceed the FP16 range (max |q| = %g)", (double)qmax);
    return ST_ENOTSUP;
  }
  const bool integer = (hf[0] & 1) == 0 && ti->integer;
  const bool exact = integer && exact_screen(d, dp, qmax, ti->vmax, (hf[0] & 2) != 0 || ti->negative);
  *exact_out = exact ? 1 : 0;
  if (exact) split = 0;  // integer data: the one-product screen (BF16 or FP16) is already exact
  // screened keys kept per query: exact sqeuclidean needs none extra
  const int mmode = (exact && metric == METRIC_SQEUCLIDEAN) ? 0 : margin_mode_of(tier);
  const int margin = kk2_of(kk, mmode) - kk;
  const int kk2 = kk + margin;

  const int kout = kk2 > 32 ? kKeep : kk2;
  const int acols = query_cols(d, split);
  // Rows of up to two chunks (d <= 128, split d <= 64): the query operand in shared
  // memory leaves room for four tiles beside it and all of TMEM for accumulators,
  // two per half.  Longer rows: in TMEM, and one accumulator per half.
  const int chunks = (split ? 2 : 1) * kc;
  const int ss = chunks <= 2 ? 1 : 0;
  const size_t b_bytes = (size_t)XN * BK * 2;
  const size_t tile_bytes = chunks * b_bytes + kNormBytes;
  const size_t fixed = kFixedSmem + (ss ? 2 * chunks * b_bytes : 0);
  const int stages = std::min(kMaxStages, (int)((kSmemPerCta - fixed) / tile_bytes));
  const size_t smem = fixed + stages * tile_bytes;

  // Work decomposition.  The queries run in batches.  A batch of whole waves
  // (a multiple of the GPU's CTA slots in query blocks) has one CTA per
  // block: the hardware hands blocks to free slots as they come, which
  // evens out blocks of unequal cost.  A batch of less than a wave (a small
  // query count, or the last part of a large one) would leave slots idle, so
  // there each block's index scan is cut into s equal tile ranges (quanta);
  // the quanta, block-major, are dealt out L at a time to consecutive CTAs,
  // L = ceil(quanta / slots).  s is the count (quanta of >= kMinQuantum tiles, or 2, at most
  // kMaxSplits - 2 pieces per block) that minimises the longest CTA's work,
  // L (ntiles / s + 4) tiles with 4 tiles' worth charged per piece for its
  // pipeline refill and its list's start, and 15% more for pieces that a CTA works
  // through one after the other, which cannot share limits.  A CTA's quanta fall into pieces at
  // query-block boundaries; a block cut into several pieces gets one kept
  // list per piece, merged afterwards.
  const int64_t ntiles_all = (n + XN - 1) / XN;
  const int64_t slots = 152;  // one CTA per SM
  const int64_t wave_q = slots * QB;
  constexpr int kMaxQuanta = kMaxSplits - 2;
  auto quanta_of = [&](int64_t qbl) -> int {
    int best = 1;
    double best_cost = 0.0;
    for (int sq = 1; sq <= kMaxQuanta; sq++) {
      // (a small index is all first tiles, whose columns are logged: what bounds it is
      // each CTA's selection, so it is spread as far as every piece has a CTA of its own)
      const bool spread_out = ntiles_all < kSmallIndex && qbl * sq <= slots;
      if (sq > 1 && ntiles_all / sq < (spread_out ? 2 : kMinQuantum)) break;
      const int64_t L = (qbl * sq + slots - 1) / slots;
      const double cost = (double)L * ((double)ntiles_all / sq + 4.0) * (L > 1 ? 1.15 : 1.0);
      if (sq == 1 || cost < best_cost) best = sq, best_cost = cost;
    }
    // tunable: FUELG_KNN_QUANTA fixes s
    if (const char* e = getenv("FUELG_KNN_QUANTA"))
      best = (int)std::max<int64_t>(1, std::min<int64_t>({(int64_t)atoi(e), (int64_t)kMaxQuanta, ntiles_all}));
    return best;
  };
  struct Batch {
    int64_t b0, mcur, G, P;
    bool merge;
    std::vector<int32_t> tab;  // piece_qb[P] piece_t0[P] piece_t1[P] cta_pb[G+1] qb_pb[blocks+1]
  };
  // Bound scratch: whole-wave batches whose lists take at most ~1 GiB.
  const int64_t mb_waves =
      std::max<int64_t>(1, (int64_t)((1ull << 30) / ((size_t)(kKeep + 2 * kLog + kout + 2 * kk2) * 8)) / wave_q) * wave_q;
  std::vector<Batch> batches;
  size_t lists_rows = 0, kept_rows = 0, merge_rows = 0, tab_max = 0;
  int64_t mb = 0;  // largest batch
  for (int64_t b0 = 0; b0 < m;) {
    const int64_t rem = m - b0;
    Batch bt;
    bt.b0 = b0;
    bt.mcur = rem >= wave_q ? std::min<int64_t>(mb_waves, rem / wave_q * wave_q) : rem;
    const int64_t qbl = (bt.mcur + QB - 1) / QB;
    const int sq = bt.mcur >= wave_q ? 1 : quanta_of(qbl);
    const int64_t nq_all = qbl * sq;
    const int64_t L = bt.mcur >= wave_q ? 1 : (nq_all + slots - 1) / slots;
    bt.G = (nq_all + L - 1) / L;
    std::vector<int32_t> pq, pt0, pt1, cpb(1, 0), qpb(1, 0);
    for (int64_t c = 0; c < bt.G; c++) {
      const int64_t qe = std::min<int64_t>(nq_all, (c + 1) * L);
      for (int64_t qu = c * L; qu < qe;) {
        // a run of this CTA's quanta inside one block is one piece
        const int64_t blk = qu / sq, j0 = qu - blk * sq;
        const int64_t j1 = std::min<int64_t>(sq, j0 + (qe - qu));
        pq.push_back((int32_t)blk);
        pt0.push_back((int32_t)(ntiles_all * j0 / sq));
        pt1.push_back((int32_t)(ntiles_all * j1 / sq));
        qu += j1 - j0;
      }
      cpb.push_back((int32_t)pq.size());
    }
    bt.P = (int64_t)pq.size();
    bt.merge = false;
    for (int64_t p = 0, blk = 0; p < bt.P; p++) {
      if (pt0[p] != 0 || pt1[p] != ntiles_all) bt.merge = true;
      while (blk < pq[p]) qpb.push_back((int32_t)p), blk++;
      if (p + 1 == bt.P) qpb.push_back((int32_t)bt.P);
    }
    for (int64_t blk = 0; blk < qbl; blk++)
      if (qpb[blk + 1] - qpb[blk] > kMaxSplits) {
        set_error("kNN work decomposition cuts a query block into more than %d pieces", kMaxSplits);
        return ST_EINVAL;
      }
    bt.tab.reserve(3 * bt.P + bt.G + 1 + qbl + 1);
    bt.tab.insert(bt.tab.end(), pq.begin(), pq.end());
    bt.tab.insert(bt.tab.end(), pt0.begin(), pt0.end());
    bt.tab.insert(bt.tab.end(), pt1.begin(), pt1.end());
    bt.tab.insert(bt.tab.end(), cpb.begin(), cpb.end());
    bt.tab.insert(bt.tab.end(), qpb.begin(), qpb.end());
    lists_rows = std::max(lists_rows, (size_t)bt.G * QB);
    kept_rows = std::max(kept_rows, (size_t)bt.P * QB);
    if (bt.merge) merge_rows = std::max(merge_rows, (size_t)bt.mcur);
    tab_max = std::max(tab_max, bt.tab.size());
    mb = std::max(mb, bt.mcur);
    b0 += bt.mcur;
    batches.push_back(std::move(bt));
  }
  Scratch lists, kept_sp, kept_m, kept2, redo, nredo, plan, pub;
  FUELG_TRY(lists.alloc(lists_rows * (kKeep + 2 * kLog) * 8, stream));
  FUELG_TRY(kept_sp.alloc(kept_rows * kout * 8, stream));
  if (merge_rows) {
    FUELG_TRY(kept_m.alloc(merge_rows * kk2 * 8, stream));
    FUELG_TRY(pub.alloc(kept_rows * sizeof(unsigned), stream));
  }
  FUELG_TRY(plan.alloc(sizeof(int32_t) * tab_max, stream));
  if (margin) {
    FUELG_TRY(kept2.alloc((size_t)mb * kk2 * 8, stream));
    FUELG_TRY(redo.alloc(sizeof(int32_t) * mb, stream));
    FUELG_TRY(nredo.alloc(sizeof(int32_t), stream));
  }
  auto kern = knn_tc_kernel;
  // (one limit for every shape: calls on other threads may set it at the same time)
  FUELG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemPerCta));
  // exact screens aside, the error-bound constants of the Lloyd screen
  const double u8 = std::ldexp(1.0, -8), u23 = std::ldexp(1.0, -23), u24 = std::ldexp(1.0, -24);
  // operand rounding (2u + u^2 per BF16 product with u = 2^-8; 3.01 * 2^-16
  // with hi + lo; u = 2^-11 per FP16 value in the normal range) plus FP32
  // accumulation in the tensor core over dp (3 dp) products.  FP16 values below
  // 2^-14 round with an absolute error of at most 2^-25 instead: the distance
  // (2 q.x) takes 2^-24 (|q|_1 + |x|_1) <= 2^-24 sqrt(dp) (|q| + |x|) more.
  const double u11 = std::ldexp(1.0, -11);
  // (the norm step adds kNB products, the last ones, at the size of both sums).
  // Integers up to 256 are held exactly by either format.
  const double rel = integer ? (3.0 * dp + kNB) * u23
                     : split ? 3.01 * std::ldexp(1.0, -16) + (3.0 * dp + kNB) * u23 * (1.0 + 2 * u8)
                     : f16 ? (2 * u11 + u11 * u11) + (dp + kNB) * u23 * (1.0 + 2 * u11)
                           : (2 * u8 + u8 * u8) + (dp + kNB) * u23 * (1.0 + 2 * u8);
  const float abs_a = (f16 && !exact) ? (float)(u24 * std::sqrt((double)dp) * 1.01) : 0.0f;
  // products, parts of a norm and sums below the FP32 normal range may be flushed
  const float abs_u = exact ? 0.0f : (float)(4.0 * (3.0 * dp + kNB) * std::ldexp(1.0, -126));
  // exact integer data: the screen and fuel's own f32 sum are both exact
  const float alpha = exact ? 0.0f : (float)(2.0 * rel * 1.01);
  // (+3 u: the screened value is rounded as fl(|q|^2 + fl(|x|^2 - 2 q.x)))
  const float beta = exact ? 0.0f : (float)(((d + 31) / 32 + 9) * u24 * 1.01 + 4 * u24 + kNB * u23 * 1.01);
  const float gamma = exact ? 0.0f : (float)((d + 4) * u24 * 1.01);
  // max |x|^2 over the index, for the proof
  const float xmax_n2 = ti->xmax_n2;
  const float xmax_norm = sqrtf(xmax_n2) * (1.0f + 1e-6f);
  int64_t total_redo = 0;
  HotTimer* ht = hot_timer();
  for (const Batch& bt : batches) {
    const int64_t b0 = bt.b0, mcur = bt.mcur, G = bt.G, P = bt.P;
    const bool merge = bt.merge;
    KnnTcArgs a{};
    a.m = mcur;
    a.n = n;
    a.kc = kc;
    a.ks_last = ((d + 15) / 16) - (kc - 1) * (BK / 16);
    a.kk2 = kk2;
    a.kout = kout;
    a.acols = acols;
    a.ss = ss;
    a.qhi = reinterpret_cast<const uint4*>(qb.as<__nv_bfloat16>() + b0 * dp);
    a.qlo = split ? reinterpret_cast<const uint4*>(qlo.as<__nv_bfloat16>() + b0 * dp) : nullptr;
    a.row_k = row_k != nullptr ? row_k + b0 : nullptr;
    a.margin_mode = mmode;
    a.exact = exact ? 1 : 0;
    a.split = split;
    a.spread = spread;
    a.stages = stages;
    a.qn2 = qn2.as<float>() + b0;
    a.xmax_n2 = xmax_n2;
    a.lists = lists.as<uint64_t>();
    a.out_keys = kept_sp.as<uint64_t>();
    // this batch's pieces
    FUELG_CUDA(cudaMemcpyAsync(plan.p, bt.tab.data(), bt.tab.size() * sizeof(int32_t), cudaMemcpyHostToDevice,
                               stream));
    const int32_t* dtab = plan.as<int32_t>();
    a.piece_qb = dtab;
    a.piece_t0 = dtab + P;
    a.piece_t1 = dtab + 2 * P;
    a.cta_pb = dtab + 3 * P;
    const int32_t* qb_pb = dtab + 3 * P + G + 1;
    a.qb_pb = qb_pb;
    a.pub = merge ? pub.as<unsigned>() : nullptr;
    a.concurrent = P <= slots && P == G;
    if (merge) FUELG_CUDA(cudaMemsetAsync(pub.p, 0xff, (size_t)P * QB * sizeof(unsigned), stream));
    // instruction descriptor: D=F32, A=B=BF16 (format 1) or FP16 (format 0), K-major, N=XN, M=QM
    a.idesc = (1u << 4) | (f16 ? 0u : (1u << 7) | (1u << 10)) | ((uint32_t)(XN >> 3) << 17) |
              ((uint32_t)(QM >> 4) << 24);
    a.idesc_n = a.idesc | (1u << 7) | (1u << 10);
    a.status = dev_status;
    a.cancel = cancel_word_device();
    a.wait_ns = pipeline_wait_ns();
    const dim3 grid((unsigned)G);
    if (ht) ht->begin(stream);
    const CUtensorMap& tmXs = f16 ? ti->tmXh : ti->tmX;
    // the query maps address rows b0.. through the y coordinate
    CUtensorMap tmQb, tmQl;
    FUELG_TRY(make_map_bf16(&tmQb, qb.as<__nv_bfloat16>() + b0 * dp, mpad - b0, dp, QM));
    if (split) FUELG_TRY(make_map_bf16(&tmQl, qlo.as<__nv_bfloat16>() + b0 * dp, mpad - b0, dp, QM));
    else tmQl = tmQb;
    kern<<<grid, kThreadsKT, smem, stream>>>(tmQb, tmQl, tmXs, split ? ti->tmXlo : tmXs, ti->tmN, a);
    ::fuelg::note_launch();
    if (ht) ht->end(stream);
    FUELG_CUDA(cudaGetLastError());
    uint64_t* dst = out_keys + b0 * kk;
    // each piece's kept keys in (distance, index) order; with one piece per
    // block the pieces' rows are the queries' rows
    const int64_t srows = merge ? P * QB : mcur;
    if (kk2 > 32) {  // (lists of up to 32 keys are kept sorted)
    sort_rows_kernel<<<(unsigned)((srows * 32 + 255) / 256), 256, 0, stream>>>(kept_sp.as<uint64_t>(), srows, kout);
    ::fuelg::note_launch();
    }
    uint64_t* kept = kept_sp.as<uint64_t>();
    const int kstride = merge ? kk2 : kout;
    if (merge) {
      merge_tc_splits_kernel<<<(unsigned)((mcur * 32 + 255) / 256), 256, 0, stream>>>(kept_sp.as<uint64_t>(), mcur,
                                                                                      qb_pb, kout, kk2, kept_m.as<uint64_t>());
      ::fuelg::note_launch();
      kept = kept_m.as<uint64_t>();
    }
    FUELG_CUDA(cudaGetLastError());
    if (margin == 0) {
      FUELG_CUDA(cudaMemcpy2DAsync(dst, (size_t)kk * 8, kept, (size_t)kstride * 8, (size_t)kk * 8, (size_t)mcur,
                                   cudaMemcpyDeviceToDevice, stream));
      continue;
    }
    FUELG_CUDA(cudaMemsetAsync(nredo.p, 0, sizeof(int32_t), stream));
    const size_t rsm = (size_t)8 * (d + 4) * sizeof(float);
    const unsigned rg = (unsigned)((mcur * 32 + 255) / 256);
    if (order == ORDER_X86)
      knn_rescore_kernel<ORDER_X86><<<rg, 256, rsm, stream>>>(Q32 + b0 * d, X32, n, d, mcur, kk, kk2,
                                                              row_k != nullptr ? row_k + b0 : nullptr, mmode, metric,
                                                              kept, kstride, kept2.as<uint64_t>(),
                                                              qn2.as<float>() + b0, xmax_norm, xmax_n2, alpha, beta,
                                                              gamma, abs_a, abs_u, redo.as<int32_t>(), nredo.as<int32_t>());
    else
      knn_rescore_kernel<ORDER_ARM><<<rg, 256, rsm, stream>>>(Q32 + b0 * d, X32, n, d, mcur, kk, kk2,
                                                              row_k != nullptr ? row_k + b0 : nullptr, mmode, metric,
                                                              kept, kstride, kept2.as<uint64_t>(),
                                                              qn2.as<float>() + b0, xmax_norm, xmax_n2, alpha, beta,
                                                              gamma, abs_a, abs_u, redo.as<int32_t>(), nredo.as<int32_t>());
    ::fuelg::note_launch();
    FUELG_CUDA(cudaGetLastError());
    // first kk exact keys of every query
    FUELG_CUDA(cudaMemcpy2DAsync(dst, (size_t)kk * 8, kept2.p, (size_t)kk2 * 8, (size_t)kk * 8, (size_t)mcur,
                                 cudaMemcpyDeviceToDevice, stream));
    int h_redo = 0;
    FUELG_CUDA(cudaMemcpyAsync(&h_redo, nredo.p, sizeof(int32_t), cudaMemcpyDeviceToHost, stream));
    FUELG_CUDA(cudaStreamSynchronize(stream));
    if (h_redo > 0) {
      // queries the proof could not certify: exact scan
      Scratch qre, kre;
      FUELG_TRY(qre.alloc(sizeof(float) * (size_t)h_redo * d, stream));
      FUELG_TRY(kre.alloc(sizeof(uint64_t) * (size_t)h_redo * kk, stream));
      gather_rows_kernel<<<4 * 152, 256, 0, stream>>>(Q32 + b0 * d, d, redo.as<int32_t>(), nredo.as<int32_t>(),
                                                      qre.as<float>()); ::fuelg::note_launch();
      ExactScanParams sp;
      sp.A = qre.as<float>();
      sp.m = h_redo;
      sp.B = X32;
      sp.n = n;
      sp.d = d;
      sp.kind = KIND_KNN;
      sp.order = order;
      sp.metric = metric;
      sp.kk = kk;
      FUELG_TRY(exact_topk(sp, kre.as<uint64_t>(), dev_status, stream));
      scatter_keys_kernel<<<(unsigned)(((int64_t)h_redo * kk + 255) / 256), 256, 0, stream>>>(
          kre.as<uint64_t>(), kk, kk, redo.as<int32_t>(), h_redo, dst); ::fuelg::note_launch();
      FUELG_CUDA(cudaGetLastError());
      total_redo += h_redo;
    }
  }
  if (rescored) *rescored = margin ? m * (int64_t)kk2 + total_redo * n : 0;
  return ST_OK;
}

}  // namespace fuelg
