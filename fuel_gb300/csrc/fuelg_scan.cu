// fuelg_scan.cu -- exact FP32 linear-scan top-k in register tiles.
//
// The work is qblocks x nt tiles (W * 8 query rows against 128 index rows),
// query-block-major, cut into G contiguous equal runs, one per resident CTA;
// a run that crosses a query block starts new lists there.  A warp owns 8
// query rows, so its selection needs no other warp: the distances stay in
// registers, a row's 128 distances of a tile are tested against its running
// kk-th key with one vote, the few that pass are appended to the row's log, and
// the log is folded into the row's kept keys by the warp (a sorted list of
// 32 keys merged bitonically for kk <= 32, few keys one by one, warp_select above).  The lists of a
// query block's runs are merged afterwards.
//
// Bound: FP32 issue (3 operations per pair and dimension, one fold per 8): 47
// operations a pair at d = 16.  20 000-point self-join, d = 16, k = 10: 0.95 ms
// (the per-thread-list scan of fuelg_knn.cu: 2.15 ms; 0.48 ms of FP32 issue), of
// which selection 0.27 ms.  16 queries against 10^6 rows, d = 16: 0.20 ms a call
// (4.5), 64 queries, k = 200: 1.05 ms (44).
#include <algorithm>

#include "fuelg_common.cuh"
#include "fuelg_internal.h"
#include "fuelg_select.cuh"
#include "fuelg_tile.cuh"

namespace fuelg {
namespace {

struct TileScanArgs {
  const float* A;  // queries [m, d]
  int64_t m;
  const float* B;  // points [n, d]
  int64_t n;
  int d, nb;
  int kk, metric;
  int64_t nt;        // tiles per query block
  int64_t T;         // tiles in all
  uint64_t* lists;   // [CTA][8 W][lstride]: kept keys, then the append log (kk > 32)
  int lstride;       // kk + kTileLogCap + kTileP (kk > 32)
  int tps;           // tiles staged per barrier
  uint64_t* out;     // [qblocks][J][8 W][kk]
  int J;
  unsigned* gthr;    // [m] squared-distance limits (s_thr) shared by a query's runs, or nullptr
  f32x2 nz;          // kNegZero2 (tile_dists)
  int* status;
  const volatile int* cancel;
};

constexpr int kTileMaxD = 128;
constexpr int kFewKeys = 8;  // keys of the kFew lists, at most
// log entries that trigger a selection: a tile adds up to 128, warp_select takes 256
constexpr int kTileLogCap = 32 * kSel - kTileP;
constexpr int kTileSmemMax =
    (int)sizeof(float) * kTileMaxD * (kTileQS + 2 * kTilePS);  // 167 KB

// kSorted: kk <= 32, each row's keys as a sorted list in shared memory that every
// passing key enters at once (the limit is never stale, so the fewest tiles
// take the slow path); kFew: the same for kk <= kFewKeys, where a tile with many
// candidates for a row hands in its smallest keys one by one until one does not enter,
// in place of sorting them all (100 000 queries, k = 2, on 5000 x 2 rows ever closer to
// them 4503 -> 1720 us, the per-thread lists 1499); kLogs: kept keys and an append log in
// global memory.
enum ScanLists { kLogs, kSorted, kFew };
template <bool FMA8, ScanLists LISTS>
__global__ void __launch_bounds__(32 * kTileMaxWarps, 2) scan_tile_kernel(TileScanArgs a) {
  constexpr bool SMALL = LISTS != kLogs, FEW = LISTS == kFew;
  extern __shared__ __align__(16) float tsm[];
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int QM = kTileQ * warps;
  float* qT = tsm;                                  // [d][kTileQS]
  float* xT = qT + (size_t)a.d * kTileQS;                // [2][tps][d][kTilePS]
  const size_t xtile = (size_t)a.d * kTilePS;
  const size_t xbuf = a.tps * xtile;
  constexpr int R = kTileQ * kTileMaxWarps;
  // per query row: above the bits of every squared distance that can still enter
  __shared__ __align__(16) unsigned s_thr[R];
  __shared__ uint64_t s_list[SMALL ? R * 32 : 1];
  __shared__ uint64_t s_tau[SMALL ? 1 : R];                   // kk-th key held
  __shared__ int s_cnt[SMALL ? 1 : R], s_len[SMALL ? 1 : R];  // log entries, kept keys

  const int64_t G = gridDim.x;
  const int64_t t_end = scan_run_begin(blockIdx.x + 1, a.T, G);
  uint64_t* const my = a.lists + ((size_t)blockIdx.x * QM + warp * kTileQ) * a.lstride;  // this warp's rows
  int stop = 0;  // thread 0: the cancel word as of its last look

  // lane 0: row r's new limit from its kk-th key (never above what other runs of
  // the query have found).  gthr has m words, and q < m: rows past m have the limit 0,
  // which no distance is below, so they never hold a key (see the start of a piece).
  auto set_limit = [&](int r, int64_t q, uint64_t tau) {
    if (tau == KEY_NONE) return;
    const float D = key_dist(tau);
    const unsigned lim = tile_limit_bits(D, a.metric);
    const unsigned over = lim == 0xffffffffu ? lim : lim + 1;
    // this run goes up in the index, so an equal distance no longer enters here; it can
    // in another run (100 000 queries, k = 2, on 2000 x 2, each row some 50 times: 756 -> 298
    // us with both, the per-thread lists 531)
    s_thr[r] = min(s_thr[r], D == 0.0f ? 0u : a.metric == METRIC_SQEUCLIDEAN ? lim : over);
    if (a.gthr != nullptr) atomicMin(a.gthr + q, over);
  };
  // folds row j's log into its kept keys (whole warp)
  auto flush = [&](int j, int64_t q0) {
    const int r = warp * kTileQ + j;
    uint64_t* list = my + (size_t)j * a.lstride;
    const int cnt = s_cnt[r], len = s_len[r];
    const uint64_t tau = warp_select(list + a.kk, cnt, list, len, a.kk, lane);
    __syncwarp();
    if (lane == 0) {
      s_len[r] = min(a.kk, len + cnt);
      s_cnt[r] = 0;
      s_tau[r] = tau;
      set_limit(r, q0 + r, tau);
    }
    __syncwarp();
  };

  for (int64_t t = scan_run_begin(blockIdx.x, a.T, G); t < t_end;) {
    const int64_t qb = t / a.nt;
    const int64_t x_first = t - qb * a.nt;
    const int64_t x_last = min(a.nt, x_first + (t_end - t));
    const int64_t q0 = qb * QM;
    t += x_last - x_first;
    __syncthreads();  // the previous piece's tiles are no longer read
    tile_stage(qT, kTileQS, a.A, q0, QM, a.m, a.d, a.nb);
    for (int u = 0; u < a.tps && x_first + u < x_last; u++)
      tile_stage(xT + u * xtile, kTilePS, a.B, (x_first + u) * kTileP, kTileP, a.n, a.d, a.nb);
    if (lane < kTileQ) {
      const int r = warp * kTileQ + lane;
      // (rows past m: nothing is below 0, so nothing enters)
      s_thr[r] = q0 + r >= a.m ? 0u : a.gthr != nullptr ? *((volatile unsigned*)a.gthr + q0 + r) : 0xffffffffu;
      if (!SMALL) {
        s_cnt[r] = s_len[r] = 0;
        s_tau[r] = KEY_NONE;
      }
    }
    if (SMALL)
      for (int j = 0; j < kTileQ; j++) s_list[(warp * kTileQ + j) * 32 + lane] = KEY_NONE;
    __syncwarp();
    int buf = 0;
    bool stopped = false;
    for (int64_t x0 = x_first; x0 < x_last; x0 += a.tps, buf ^= 1) {
      cp_async_wait_all();
      // these tiles have landed; the other buffer is no longer read
      if (__syncthreads_or(stop)) {
        if (threadIdx.x == 0) atomicOr(a.status, DEV_CANCELLED);
        stopped = true;
        break;
      }
      // a look every 16 tiles, from the index's first ones on (an index of few tiles has no
      // 16th stage), whose answer the next barrier takes: none waits for host memory
      if (threadIdx.x == 0 && a.cancel != nullptr && ((int)x0 & 15) < a.tps) stop = *a.cancel;
      // the other runs' limits as of this stage (used from the next one on)
      unsigned seen = 0xffffffffu;
      if (a.gthr != nullptr && lane < kTileQ && q0 + warp * kTileQ + lane < a.m)
        seen = *((volatile unsigned*)a.gthr + q0 + warp * kTileQ + lane);
      for (int u = 0; u < a.tps && x0 + a.tps + u < x_last; u++)
        tile_stage(xT + (buf ^ 1) * xbuf + u * xtile, kTilePS, a.B, (x0 + a.tps + u) * kTileP, kTileP, a.n, a.d, a.nb);
      for (int u = 0; u < a.tps && x0 + u < x_last; u++) {
        float s[kTileQ][4];
        tile_dists<FMA8>(qT + warp * kTileQ, xT + buf * xbuf + u * xtile + lane, a.d, a.nb, a.nz, s);
        const uint4 th0 = *reinterpret_cast<const uint4*>(s_thr + warp * kTileQ);
        const uint4 th1 = *reinterpret_cast<const uint4*>(s_thr + warp * kTileQ + 4);
        const unsigned thr[kTileQ] = {th0.x, th0.y, th0.z, th0.w, th1.x, th1.y, th1.z, th1.w};
        unsigned hits = 0;  // rows with a distance below their limit
#pragma unroll
        for (int j = 0; j < kTileQ; j++) hits |= tile_min_bits(s[j]) < thr[j] ? 1u << j : 0u;
        hits = __reduce_or_sync(0xffffffffu, hits);
        while (hits) {
          const int j = __ffs(hits) - 1;
          hits &= hits - 1;
          const int r = warp * kTileQ + j;
          float v[4];
          auto row = [&](int jj) {
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = s[jj][i];
          };
          // (uniform branches: s stays in registers)
          if (j & 4) {
            if (j & 2) {
              if (j & 1) row(7); else row(6);
            } else {
              if (j & 1) row(5); else row(4);
            }
          } else {
            if (j & 2) {
              if (j & 1) row(3); else row(2);
            } else {
              if (j & 1) row(1); else row(0);
            }
          }
          const unsigned lim = s_thr[r];
          const int64_t p0 = (x0 + u) * kTileP;
          const int left = (int)min((int64_t)kTileP, a.n - p0) - lane;  // row lane + 32 i exists: 32 i < left
          unsigned in[4];
          int found = 0;
#pragma unroll
          for (int i = 0; i < 4; i++) {
            in[i] = __ballot_sync(0xffffffffu, __float_as_uint(v[i]) < lim && 32 * i < left);
            found += __popc(in[i]);
          }
          if (SMALL) {
            uint64_t kept = s_list[r * 32 + lane];
            uint64_t tau = shfl_u64(kept, a.kk - 1);
            if (FEW && found > 12) {
              // many candidates for few places (an index's first tiles, rows ever closer to
              // the query): the smallest keys one after the other, until one does not enter
              unsigned u[4];
#pragma unroll
              for (int i = 0; i < 4; i++) {
                const float dv = a.metric == METRIC_EUCLIDEAN ? __fsqrt_rn(v[i]) : v[i];
                u[i] = in[i] >> lane & 1 ? __float_as_uint(dv) : 0xffffffffu;
              }
              for (;;) {
                const unsigned w = __reduce_min_sync(0xffffffffu, min(min(u[0], u[1]), min(u[2], u[3])));
                if (w == 0xffffffffu || w > (uint32_t)(tau >> 32)) break;
                int at = 0;  // the lowest column that holds it
#pragma unroll
                for (int i = 3; i >= 0; i--) {
                  const unsigned b = __ballot_sync(0xffffffffu, u[i] == w);
                  if (b) at = __ffs(b) - 1 + 32 * i;
                }
                const uint64_t key = ((uint64_t)w << 32) | (uint32_t)(p0 + at);
                if (key >= tau) break;
                kept = warp_insert32(kept, key, lane);
                tau = shfl_u64(kept, a.kk - 1);
#pragma unroll
                for (int i = 0; i < 4; i++)
                  if (at == lane + 32 * i) u[i] = 0xffffffffu;
              }
              s_list[r * 32 + lane] = kept;
              if (lane == 0) set_limit(r, q0 + r, tau);
              __syncwarp();
              continue;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
              if (in[i] == 0) continue;
              if (!FEW && found > 12) {
                const float dv = a.metric == METRIC_EUCLIDEAN ? __fsqrt_rn(v[i]) : v[i];
                kept = warp_merge32(kept, in[i] >> lane & 1 ? make_key(dv, (uint32_t)(p0 + lane + 32 * i)) : KEY_NONE,
                                    lane);
                tau = shfl_u64(kept, a.kk - 1);
                continue;
              }
              do {
                const int src = __ffs(in[i]) - 1;
                in[i] &= in[i] - 1;
                float dv = __shfl_sync(0xffffffffu, v[i], src);
                if (a.metric == METRIC_EUCLIDEAN) dv = __fsqrt_rn(dv);
                const uint64_t key = make_key(dv, (uint32_t)(p0 + src + 32 * i));
                if (key < tau) {
                  kept = warp_insert32(kept, key, lane);
                  tau = shfl_u64(kept, a.kk - 1);
                }
              } while (in[i]);
            }
            s_list[r * 32 + lane] = kept;
            if (lane == 0) set_limit(r, q0 + r, tau);
            __syncwarp();
          } else {
            uint64_t* log = my + (size_t)j * a.lstride + a.kk;
            const uint64_t tau = s_tau[r];
            int cnt = s_cnt[r];
#pragma unroll
            for (int i = 0; i < 4; i++) {
              if (in[i] == 0) continue;
              const float dv = a.metric == METRIC_EUCLIDEAN ? __fsqrt_rn(v[i]) : v[i];
              const uint64_t key = in[i] >> lane & 1 ? make_key(dv, (uint32_t)(p0 + lane + 32 * i)) : KEY_NONE;
              const unsigned enter = __ballot_sync(0xffffffffu, key < tau);
              if (key < tau) log[cnt + __popc(enter & ((1u << lane) - 1u))] = key;
              cnt += __popc(enter);
            }
            __syncwarp();
            if (lane == 0) s_cnt[r] = cnt;
            __syncwarp();
            if (cnt >= kTileLogCap) flush(j, q0);
          }
        }
      }
      if (lane < kTileQ && seen < s_thr[warp * kTileQ + lane]) s_thr[warp * kTileQ + lane] = seen;
      __syncwarp();
    }
    if (stopped) break;
    const int64_t jl = blockIdx.x - scan_run_of(qb * a.nt, a.T, G);
    uint64_t* out = a.out + ((size_t)(qb * a.J + jl) * QM + warp * kTileQ) * a.kk;
    for (int j = 0; j < kTileQ; j++) {
      const int r = warp * kTileQ + j;
      if (q0 + r >= a.m) break;
      if (SMALL) {
        if (lane < a.kk) out[(size_t)j * a.kk + lane] = s_list[r * 32 + lane];
      } else {
        if (s_cnt[r] > 0) flush(j, q0);
        const int len = s_len[r];
        const uint64_t* list = my + (size_t)j * a.lstride;
        for (int o = lane; o < a.kk; o += 32) out[(size_t)j * a.kk + o] = o < len ? list[o] : KEY_NONE;
      }
    }
  }
  cp_async_wait_all();
}

// Merges the lists of each query block's runs into keys[q][0, kk), kk <= 32:
// the lists are sorted, so their r-th keys are offered rank by rank and the
// merge ends at the first rank that no list enters with.  wpq warps (1 or all
// eight of the block) share a query's lists.
__global__ void __launch_bounds__(256) merge_runs32_kernel(const uint64_t* __restrict__ in, int64_t m, int QM,
                                                           int64_t nt, int64_t T, int64_t G, int J, int kk, int wpq,
                                                           uint64_t* __restrict__ keys) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __shared__ uint64_t part[8][32];
  const int64_t q = wpq == 1 ? (int64_t)blockIdx.x * 8 + warp : (int64_t)blockIdx.x;
  if (q >= m) return;
  const int64_t qb = q / QM, row = q - qb * QM;
  const int cnt = (int)(scan_run_of((qb + 1) * nt - 1, T, G) - scan_run_of(qb * nt, T, G)) + 1;
  const uint64_t* base = in + ((size_t)qb * J * QM + row) * kk;
  const size_t lst = (size_t)QM * kk;
  uint64_t kept = KEY_NONE, tau = KEY_NONE;
  const int l0 = wpq == 1 ? 0 : warp * 32, ls = wpq * 32;
  for (int r = 0; r < kk; r++) {
    bool entered = false;
    for (int l = l0; l < cnt; l += ls) {
      const uint64_t v = l + lane < cnt ? base[(size_t)(l + lane) * lst + r] : KEY_NONE;
      if (__any_sync(0xffffffffu, v < tau)) {
        entered = true;
        kept = warp_merge32(kept, v, lane);
        tau = shfl_u64(kept, kk - 1);
      }
    }
    if (!entered) break;
  }
  if (wpq > 1) {
    part[warp][lane] = kept;
    __syncthreads();
    if (warp != 0) return;
    for (int w = 1; w < 8; w++) {
      const uint64_t v = part[w][lane];
      if (__any_sync(0xffffffffu, v < tau)) {
        kept = warp_merge32(kept, v, lane);
        tau = shfl_u64(kept, kk - 1);
      }
    }
  }
  if (lane < kk) keys[q * kk + lane] = kept;
}

}  // namespace

// The shapes the tile scan takes: a query block and two index tiles of d
// dimensions have to fit shared memory, and a row's keys one warp's selection.
bool tile_scan_supported(int d, int kk) { return d >= 1 && d <= kTileMaxD && kk >= 1 && kk <= 32 * kSel; }

int tile_scan_topk(const ExactScanParams& p, uint64_t* out_keys, int* dev_status, cudaStream_t stream) {
  const bool fma = p.order == ORDER_X86;
  const bool small = p.kk <= 32;
  const bool few = p.kk <= kFewKeys;
  auto kern = few ? (fma ? scan_tile_kernel<true, kFew> : scan_tile_kernel<false, kFew>)
              : small ? (fma ? scan_tile_kernel<true, kSorted> : scan_tile_kernel<false, kSorted>)
                      : (fma ? scan_tile_kernel<true, kLogs> : scan_tile_kernel<false, kLogs>);
  const int64_t nt = (p.n + kTileP - 1) / kTileP;
  const int lstride = p.kk + kTileLogCap + kTileP;
  // tiles per barrier: several of short rows, so that a warp with more candidates
  // than the others holds them up less often (20 000-point self-join, d = 16: 1.24
  // ms with 1, 1.15 with 2, 1.09 with 4, 1.34 with 6, where one CTA per SM is left)
  const int tps = p.d <= 16 ? 4 : p.d <= 32 ? 2 : 1;
  // queries in batches whose lists stay below 1 GiB: those of the runs, or (kk > 32,
  // a block per CTA) the kept keys with their logs
  const size_t qwords = std::max<size_t>(2 * (size_t)p.kk, small ? 0 : lstride);
  const int64_t mb_max = std::max<int64_t>(64, (int64_t)((1ull << 30) / (8 * qwords)) / 64 * 64);
  for (int64_t b0 = 0; b0 < p.m; b0 += mb_max) {
    const int64_t m = std::min<int64_t>(mb_max, p.m - b0);
    // few queries: fewer warps per CTA, so that no warp holds only padding rows
    const int warps = (int)std::min<int64_t>(kTileMaxWarps, (m + kTileQ - 1) / kTileQ);
    const int QM = kTileQ * warps;
    const size_t smem = sizeof(float) * ((size_t)p.d * kTileQS + 2 * (size_t)tps * p.d * kTilePS);
    // one limit for every shape: calls on other threads may set it at the same time
    FUELG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemMax));
    int per_sm = 1;
    FUELG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * warps, smem));
    const int64_t qblocks = (m + QM - 1) / QM;
    const int64_t T = qblocks * nt;
    const int64_t slots = 152 * (int64_t)std::max(1, per_sm);
    int64_t G = std::min(T, slots);
    // many query blocks: whole blocks, handed out by the hardware (their
    // selection cost differs); no lists to merge
    if (qblocks >= 8 * slots) G = qblocks;
    // lists per block: bounded by what a merge takes (128 for kk > 32)
    if (!small) G = std::min<int64_t>(G, std::max<int64_t>(1, qblocks * 120));
    int64_t J = 1;
    if (G != qblocks)
      J = (nt * G + T - 1) / T + 1;  // runs that one block's tiles can touch
    Scratch lists, runs, gthr;
    if (!small) FUELG_TRY(lists.alloc((size_t)G * QM * lstride * 8, stream));
    uint64_t* keys = out_keys + b0 * p.kk;
    const bool merge = J > 1;
    if (merge) {
      FUELG_TRY(runs.alloc((size_t)qblocks * J * QM * p.kk * 8, stream));
      FUELG_TRY(gthr.alloc(sizeof(unsigned) * m, stream));
      FUELG_CUDA(cudaMemsetAsync(gthr.p, 0xff, sizeof(unsigned) * m, stream));
    }
    TileScanArgs a{};
    a.A = p.A + b0 * p.d;
    a.m = m;
    a.B = p.B;
    a.n = p.n;
    a.d = p.d;
    a.nb = p.d / 8;
    a.kk = p.kk;
    a.metric = p.metric;
    a.nt = nt;
    a.T = T;
    a.lists = lists.as<uint64_t>();
    a.lstride = lstride;
    a.tps = tps;
    a.nz = kNegZero2;
    a.out = merge ? runs.as<uint64_t>() : keys;
    a.J = (int)J;
    a.gthr = merge ? gthr.as<unsigned>() : nullptr;
    a.status = dev_status;
    a.cancel = cancel_word_device();
    HotTimer* ht = hot_timer();
    if (ht) ht->begin(stream);
    kern<<<(unsigned)G, 32 * warps, smem, stream>>>(a);
    note_launch();
    if (ht) ht->end(stream);
    FUELG_CUDA(cudaGetLastError());
    if (small) {
      if (merge) {
        const int wpq = J > 64 ? 8 : 1;
        merge_runs32_kernel<<<(unsigned)(wpq == 8 ? m : (m + 7) / 8), 256, 0, stream>>>(
            runs.as<uint64_t>(), m, QM, nt, T, G, (int)J, p.kk, wpq, keys);
        note_launch();
      }
    } else {
      FUELG_TRY(sort_and_merge_runs(merge ? runs.as<uint64_t>() : keys, m, QM, nt, T, G, (int)J, p.kk, keys, stream));
    }
    FUELG_CUDA(cudaGetLastError());
  }
  return ST_OK;
}

}  // namespace fuelg
