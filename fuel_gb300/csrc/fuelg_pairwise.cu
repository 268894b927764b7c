// fuelg_pairwise.cu -- all pairwise distances of one point set, the GPU form
// of fuel.search.pairwise_distances (python/fuel/search.py:92-150 ->
// _compute_pairwise_distances[_condensed]_f32, python/mod.rs:74-124).
//
// Forms (src/api/condensed_distance_matrix.rs:16-48, square_distance_matrix.rs:11-40):
//   condensed: the lower triangle, pair (i, j) with j < i at i (i - 1) / 2 + j;
//   square:    the symmetric n x n matrix (diagonal: distance(x_i, x_i) = 0).
// Every value is fuel's SquaredEuclidean / Euclidean distance(x_i, x_j)
// (src/distance/squared_euclidean.rs:16-39 on x86 with FMA, 99-133 otherwise,
// euclidean.rs:7-9): eight lane accumulators over d & ~7, summed in lane
// order, then the tail -- the same operation sequence as the kNN scan
// (exact_dist_scalar<KIND_KNN, order>), so results are bit-identical.
// (x_i - x_j)^2 == (x_j - x_i)^2 exactly, so the mirrored half of the square
// form is the same value.
//
// Kernels: d <= 128 (pairwise_tile_kernel): blocks of 64 rows against strips of
// 128-column tiles in the register tiles of fuelg_tile.cuh; where those would leave
// places on the chip empty (pairwise_rows_kernel), 64 x 64 tiles with half the pairs per
// thread.  Larger d (pairwise_kernel): 32 x 32 tiles of the lower tile triangle,
// 64-column chunks, 2 x 2 pairs with 8 lane accumulators each.  Small d is bound by FP32
// issue and the output writes (HBM), large d by FP32 issue, few rows by latency.
#include <algorithm>
#include <cmath>

#include "../../include/fuelg.h"
#include "fuelg_common.cuh"
#include "fuelg_internal.h"
#include "fuelg_tile.cuh"

namespace fuelg {
namespace {

constexpr int PT = 32;      // tile edge (points)
constexpr int PC = 64;      // dims per staged chunk (a multiple of 8)
constexpr int PS = PC + 4;  // staged row stride (floats): 16-byte rows, rotated banks

template <int ORDER, int METRIC, int FORM>
__global__ void __launch_bounds__(256) pairwise_kernel(const float* __restrict__ X, int64_t n, int d,
                                                       int64_t ntb, float* __restrict__ out) {
  constexpr bool FMA8 = ORDER == ORDER_X86;
  __shared__ __align__(16) float sa[PT * PS];
  __shared__ __align__(16) float sb[PT * PS];
  __shared__ float st[PT][PT + 1];  // square form: the tile, for the mirrored (transposed) write
  // tile t of the lower tile triangle -> (bi, bj), bj <= bi
  const int64_t t = blockIdx.x;
  int64_t bi = (int64_t)((std::sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
  while (bi * (bi + 1) / 2 > t) bi--;
  while ((bi + 1) * (bi + 2) / 2 <= t) bi++;
  const int64_t bj = t - bi * (bi + 1) / 2;
  if (bi >= ntb) return;
  const int64_t i0 = bi * PT, j0 = bj * PT;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int r0 = 2 * ty, c0 = 2 * tx;  // this thread: rows i0 + r0 + {0,1}, cols j0 + c0 + {0,1}
  float acc[2][2][8];
#pragma unroll
  for (int a = 0; a < 2; a++)
#pragma unroll
    for (int b = 0; b < 2; b++)
#pragma unroll
      for (int l = 0; l < 8; l++) acc[a][b][l] = 0.0f;
  const int sd = d & ~7;
  for (int k0 = 0; k0 < sd; k0 += PC) {
    const int kw = min(PC, sd - k0);  // a multiple of 8
    __syncthreads();
    for (int e = threadIdx.x; e < PT * PC; e += 256) {
      const int r = e / PC, c = e - r * PC;
      const int64_t gi = i0 + r, gj = j0 + r;
      sa[r * PS + c] = (c < kw && gi < n) ? __ldg(X + gi * d + k0 + c) : 0.0f;
      sb[r * PS + c] = (c < kw && gj < n) ? __ldg(X + gj * d + k0 + c) : 0.0f;
    }
    __syncthreads();
    for (int g = 0; g < kw; g += 8) {
      float va[2][8], vb[2][8];
#pragma unroll
      for (int a = 0; a < 2; a++) {
        const float4 p = *reinterpret_cast<const float4*>(sa + (r0 + a) * PS + g);
        const float4 q = *reinterpret_cast<const float4*>(sa + (r0 + a) * PS + g + 4);
        va[a][0] = p.x, va[a][1] = p.y, va[a][2] = p.z, va[a][3] = p.w;
        va[a][4] = q.x, va[a][5] = q.y, va[a][6] = q.z, va[a][7] = q.w;
      }
#pragma unroll
      for (int b = 0; b < 2; b++) {
        const float4 p = *reinterpret_cast<const float4*>(sb + (c0 + b) * PS + g);
        const float4 q = *reinterpret_cast<const float4*>(sb + (c0 + b) * PS + g + 4);
        vb[b][0] = p.x, vb[b][1] = p.y, vb[b][2] = p.z, vb[b][3] = p.w;
        vb[b][4] = q.x, vb[b][5] = q.y, vb[b][6] = q.z, vb[b][7] = q.w;
      }
#pragma unroll
      for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 2; b++)
#pragma unroll
          for (int l = 0; l < 8; l++) {
            const float df = __fsub_rn(va[a][l], vb[b][l]);
            acc[a][b][l] = FMA8 ? __fmaf_rn(df, df, acc[a][b][l]) : __fadd_rn(sq_rn(df), acc[a][b][l]);
          }
    }
  }
  float res[2][2];
#pragma unroll
  for (int a = 0; a < 2; a++)
#pragma unroll
    for (int b = 0; b < 2; b++) {
      const int64_t gi = i0 + r0 + a, gj = j0 + c0 + b;
      float s = acc[a][b][0];
#pragma unroll
      for (int l = 1; l < 8; l++) s = __fadd_rn(s, acc[a][b][l]);
      if (gi < n && gj < n)
        for (int k = sd; k < d; k++) {
          const float df = __fsub_rn(__ldg(X + gi * d + k), __ldg(X + gj * d + k));
          s = FMA8 ? __fmaf_rn(df, df, s) : __fadd_rn(s, sq_rn(df));
        }
      res[a][b] = METRIC == METRIC_EUCLIDEAN ? __fsqrt_rn(s) : s;
    }
  if (FORM == FUELG_PAIRWISE_CONDENSED) {
#pragma unroll
    for (int a = 0; a < 2; a++) {
      const int64_t gi = i0 + r0 + a;
#pragma unroll
      for (int b = 0; b < 2; b++) {
        const int64_t gj = j0 + c0 + b;
        if (gi < n && gj < gi) out[gi * (gi - 1) / 2 + gj] = res[a][b];
      }
    }
  } else {
#pragma unroll
    for (int a = 0; a < 2; a++) {
      const int64_t gi = i0 + r0 + a;
#pragma unroll
      for (int b = 0; b < 2; b++) {
        const int64_t gj = j0 + c0 + b;
        if (gi < n && gj < n) out[gi * n + gj] = res[a][b];
        st[r0 + a][c0 + b] = res[a][b];
      }
    }
    if (bi != bj) {  // the mirrored tile (j, i), written row by row through shared memory
      __syncthreads();
      for (int e = threadIdx.x; e < PT * PT; e += 256) {
        const int rj = e / PT, ci = e - rj * PT;
        const int64_t gj = j0 + rj, gi = i0 + ci;
        if (gj < n && gi < n) out[gj * n + gi] = st[ci][rj];
      }
    }
  }
}

// Few rows: 64 x 64 tiles of the lower tile triangle, whole rows of both blocks in
// shared memory, 4 x 4 pairs per thread computed lane by lane -- lane l's sum over the
// 8-blocks is finished before it is added to the running total, which is the
// reference's order (acc_0 + acc_1 + ... + acc_7, then the tail) with 2 registers per pair
// instead of 9.  Half the serial work per thread of the tiles below, which is what a
// call takes that does not fill the chip (pairwise_launch: both sides measured).
constexpr int PR = 64;
template <int ORDER, int METRIC, int FORM>
__global__ void __launch_bounds__(256) pairwise_rows_kernel(const float* __restrict__ X, int64_t n, int d,
                                                            int64_t ntb, float* __restrict__ out) {
  constexpr bool FMA8 = ORDER == ORDER_X86;
  extern __shared__ float rs[];  // [2][PR][d + 1]: row block i, row block j
  __shared__ float st[PR][PR + 1];
  const int S = d + 1;  // odd stride: the 16 rows a half-warp reads sit in different banks
  float* sa = rs;
  float* sb = rs + PR * S;
  const int64_t t = blockIdx.x;
  int64_t bi = (int64_t)((std::sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
  while (bi * (bi + 1) / 2 > t) bi--;
  while ((bi + 1) * (bi + 2) / 2 <= t) bi++;
  const int64_t bj = t - bi * (bi + 1) / 2;
  if (bi >= ntb) return;
  const int64_t i0 = bi * PR, j0 = bj * PR;
  for (int e = threadIdx.x; e < PR * d; e += 256) {
    const int r = e / d, c = e - r * d;
    const int64_t gi = i0 + r, gj = j0 + r;
    sa[r * S + c] = gi < n ? __ldg(X + gi * d + c) : 0.0f;
    sb[r * S + c] = gj < n ? __ldg(X + gj * d + c) : 0.0f;
  }
  __syncthreads();
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;  // rows ty + 16a, cols tx + 16b
  const int sd = d & ~7;
  float sum[4][4];
#pragma unroll 1
  for (int l = 0; l < 8; l++) {
    float acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) acc[a][b] = 0.0f;
    for (int c = l; c < sd; c += 8) {
      float xa[4], yb[4];
#pragma unroll
      for (int a = 0; a < 4; a++) xa[a] = sa[(ty + 16 * a) * S + c];
#pragma unroll
      for (int b = 0; b < 4; b++) yb[b] = sb[(tx + 16 * b) * S + c];
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) {
          const float df = __fsub_rn(xa[a], yb[b]);
          acc[a][b] = FMA8 ? __fmaf_rn(df, df, acc[a][b]) : __fadd_rn(sq_rn(df), acc[a][b]);
        }
    }
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) sum[a][b] = l == 0 ? acc[a][b] : __fadd_rn(sum[a][b], acc[a][b]);
  }
  for (int c = sd; c < d; c++) {
    float xa[4], yb[4];
#pragma unroll
    for (int a = 0; a < 4; a++) xa[a] = sa[(ty + 16 * a) * S + c];
#pragma unroll
    for (int b = 0; b < 4; b++) yb[b] = sb[(tx + 16 * b) * S + c];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) {
        const float df = __fsub_rn(xa[a], yb[b]);
        sum[a][b] = FMA8 ? __fmaf_rn(df, df, sum[a][b]) : __fadd_rn(sum[a][b], sq_rn(df));
      }
  }
#pragma unroll
  for (int a = 0; a < 4; a++) {
    const int64_t gi = i0 + ty + 16 * a;
#pragma unroll
    for (int b = 0; b < 4; b++) {
      const int64_t gj = j0 + tx + 16 * b;
      const float v = METRIC == METRIC_EUCLIDEAN ? __fsqrt_rn(sum[a][b]) : sum[a][b];
      if (FORM == FUELG_PAIRWISE_CONDENSED) {
        if (gi < n && gj < gi) out[gi * (gi - 1) / 2 + gj] = v;
      } else {
        if (gi < n && gj < n) out[gi * n + gj] = v;
        st[ty + 16 * a][tx + 16 * b] = v;
      }
    }
  }
  if (FORM == FUELG_PAIRWISE_SQUARE && bi != bj) {  // the mirrored tile (j, i), row by row
    __syncthreads();
    for (int e = threadIdx.x; e < PR * PR; e += 256) {
      const int rj = e / PR, ci = e - rj * PR;
      const int64_t gj = j0 + rj, gi = i0 + ci;
      if (gj < n && gi < n) out[gj * n + gi] = st[ci][rj];
    }
  }
}

constexpr int kRows = kTileQ * kTileMaxWarps;  // 64 rows of a block
constexpr int kTileMaxD = 128;
constexpr int kMaxStrip = 8;                    // most 128-column tiles that one CTA works through
constexpr int kTwoPerSm = 2 * 152;              // places on the chip with two CTAs per SM
constexpr int kTwoCtas = 113 * 1024;            // shared memory with which two CTAs fit an SM
constexpr int kMirror = kTileP * (kRows + 1);   // floats of the square form's transposed tile

// Rows of up to 128 dimensions: a block of 64 rows against `strip` tiles of 128
// columns (tile_dists: 32 pairs per thread, 32 consecutive columns per warp and
// store).  BUFS 2 stages the next tile while one is computed.  Only tiles that reach
// below the diagonal are computed; the square form's mirrored half goes through
// shared memory (BUFS 1: over the tile just used) so that its rows are written as
// runs too.  Bound by FP32 issue (20000 rows of 16 dimensions: 247 us of packed
// lane steps, 119 us of writes).  Whole calls against 64 x 64 tiles with 4 x 4
// pairs per thread, condensed: 20000 x 16 722 -> 413 us (Euclidean 798 -> 494),
// 20000 x 3 382 -> 206, 20000 x 128 3482 -> 2942; square 20000 x 16 873 -> 649,
// 5000 x 64 175 -> 144.
template <bool FMA8, int METRIC, int FORM, int BUFS>
__global__ void __launch_bounds__(256, 2) pairwise_tile_kernel(const float* __restrict__ X, int64_t n, int d, int nb,
                                                               int strip, f32x2 nz, float* __restrict__ out) {
  extern __shared__ __align__(16) float psm[];
  float* qT = psm;                               // [d][kTileQS]
  float* xT = qT + (size_t)d * kTileQS;          // [BUFS][d][kTilePS]
  const size_t xbuf = (size_t)d * kTilePS;
  float* st = BUFS == 2 ? xT + 2 * xbuf : xT;    // square form: [kTileP][kRows + 1]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // row blocks from the last one down, which has the longest strips
  const int64_t i0 = ((int64_t)gridDim.x - 1 - blockIdx.x) * kRows;
  const int64_t i1 = min(n, i0 + kRows);
  const int64_t jt_end = min((i1 + kTileP - 1) / kTileP, ((int64_t)blockIdx.y + 1) * strip);
  int64_t jt = (int64_t)blockIdx.y * strip;
  if (jt >= jt_end) return;
  tile_stage(qT, kTileQS, X, i0, kRows, n, d, nb);
  tile_stage(xT, kTilePS, X, jt * kTileP, kTileP, n, d, nb);
  for (int buf = 0; jt < jt_end; jt++) {
    cp_async_wait_all();
    __syncthreads();  // this tile has landed; BUFS 2: the other buffer and st are no longer read
    if (BUFS == 2 && jt + 1 < jt_end)
      tile_stage(xT + (buf ^ 1) * xbuf, kTilePS, X, (jt + 1) * kTileP, kTileP, n, d, nb);
    float s[kTileQ][4];
    tile_dists<FMA8>(qT + warp * kTileQ, xT + buf * xbuf + lane, d, nb, nz, s);
    const int64_t j0 = jt * kTileP;
    if (METRIC == METRIC_EUCLIDEAN) {
#pragma unroll
      for (int j = 0; j < kTileQ; j++)
#pragma unroll
        for (int i = 0; i < 4; i++) s[j][i] = __fsqrt_rn(s[j][i]);
    }
    const int64_t gw = i0 + warp * kTileQ;
    if (j0 + kTileP <= gw && gw + kTileQ <= n) {  // the warp's rows take the whole tile
#pragma unroll
      for (int j = 0; j < kTileQ; j++) {
        const int64_t gi = gw + j;
        float* row = out + (FORM == FUELG_PAIRWISE_CONDENSED ? gi * (gi - 1) / 2 : gi * n) + j0 + lane;
#pragma unroll
        for (int i = 0; i < 4; i++) row[32 * i] = s[j][i];
      }
    } else {
#pragma unroll
      for (int j = 0; j < kTileQ; j++) {
        const int64_t gi = gw + j;
        // below the diagonal; the square form's lower half has the diagonal too
        const int64_t end = gi < n ? (FORM == FUELG_PAIRWISE_CONDENSED ? gi : gi + 1) : 0;
        float* row = out + (FORM == FUELG_PAIRWISE_CONDENSED ? gi * (gi - 1) / 2 : gi * n) + j0;
#pragma unroll
        for (int i = 0; i < 4; i++)
          if (j0 + lane + 32 * i < end) row[lane + 32 * i] = s[j][i];
      }
    }
    if (FORM == FUELG_PAIRWISE_SQUARE) {  // mirrored: row j0 + c, columns i0 .. above the diagonal
      if (BUFS == 1) __syncthreads();     // the tile has been read by all
#pragma unroll
      for (int j = 0; j < kTileQ; j++)
#pragma unroll
        for (int i = 0; i < 4; i++) st[(lane + 32 * i) * (kRows + 1) + warp * kTileQ + j] = s[j][i];
      __syncthreads();
      for (int c = warp; c < kTileP; c += kTileMaxWarps) {
        const int64_t gj = j0 + c;
        if (gj >= n) break;
        for (int r = lane; r < kRows; r += 32)
          if (i0 + r < n && i0 + r > gj) out[gj * n + i0 + r] = st[c * (kRows + 1) + r];
      }
    }
    if (BUFS == 2) {
      buf ^= 1;
    } else if (jt + 1 < jt_end) {
      __syncthreads();
      tile_stage(xT, kTilePS, X, (jt + 1) * kTileP, kTileP, n, d, nb);
    }
  }
}

}  // namespace

int pairwise_launch(const float* X, int64_t n, int d, int metric, int order, int form, float* out,
                    cudaStream_t stream) {
  if (n < 2 && form == FUELG_PAIRWISE_CONDENSED) return ST_OK;
  if (n < 1) return ST_OK;
  const bool wide = d > kTileMaxD;
  const int64_t ntb = (n + (wide ? PT : PR) - 1) / (wide ? PT : PR);
  const int64_t tiles = ntb * (ntb + 1) / 2;
  if (tiles > 0x7fffffffll) {
    set_error("pairwise: %lld points need more tiles than one launch holds", (long long)n);
    return ST_ENOTSUP;
  }
  HotTimer* ht = hot_timer();
  if (ht) ht->begin(stream);
  const bool square = form == FUELG_PAIRWISE_SQUARE;
  const size_t smem2 = sizeof(float) * ((size_t)d * (kTileQS + 2 * kTilePS) + (square ? kMirror : 0));
  const size_t smem1 = sizeof(float) * ((size_t)d * kTileQS + std::max(d * kTilePS, square ? kMirror : 0));
  // two buffers only while two CTAs still fit an SM: one buffer and two CTAs beat
  // two buffers and one CTA (20000 x 100 condensed: 2285 against 2857 us)
  const bool two = smem2 <= kTwoCtas;
  const int64_t rb = (n + kRows - 1) / kRows, cb = (n + kTileP - 1) / kTileP;
  // strips (which stage the 64 rows once) only as long as leaves four CTAs for each
  // place on the chip: strips of eight at any n took 253 us at 5000 x 64 (144), 54
  // at 1000 x 16 (34)
  const int strip = (int)std::clamp<int64_t>(rb * cb / 2 / (kTwoPerSm * 4), 1, kMaxStrip);
  // 64 x 64 tiles while all of them are resident at once, up to 1536 rows.  Kernel, us, 64 x
  // 64 / 64 x 128: n = 300, d = 64 13.8 / 17.9, d = 128 19.8 / 28.5; n = 1500, d = 8 10.1 / 10.0,
  // d = 64 20.0 / 26.0, d = 128 30.1 / 43.2; n = 1700, d = 8 12.3 / 10.3, d = 64 25.9 / 25.9,
  // n = 1900, d = 128 52.8 / 43.2.
  const bool few = tiles <= kTwoPerSm;
  auto launch = [&](auto kr, auto k1, auto k2, auto kc) -> int {
    if (!wide && few) {
      const size_t rsm = sizeof(float) * 2 * PR * (d + 1);
      FUELG_CUDA(cudaFuncSetAttribute(kr, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rsm));
      kr<<<(unsigned)tiles, 256, rsm, stream>>>(X, n, d, ntb, out);
    } else if (!wide) {
      auto kt = two ? k2 : k1;
      FUELG_CUDA(cudaFuncSetAttribute(kt, cudaFuncAttributeMaxDynamicSharedMemorySize, kTwoCtas));
      kt<<<dim3((unsigned)rb, (unsigned)((cb + strip - 1) / strip)), 256, two ? smem2 : smem1, stream>>>(
          X, n, d, d / 8, strip, kNegZero2, out);
    } else {
      kc<<<(unsigned)tiles, 256, 0, stream>>>(X, n, d, ntb, out);
    }
    return ST_OK;
  };
#define FUELG_PW(O, M, F)                                                                        \
  FUELG_TRY(launch(pairwise_rows_kernel<O, M, F>, pairwise_tile_kernel<O == ORDER_X86, M, F, 1>, \
                   pairwise_tile_kernel<O == ORDER_X86, M, F, 2>, pairwise_kernel<O, M, F>))
  const bool x86 = order == ORDER_X86, eu = metric == METRIC_EUCLIDEAN, cond = form == FUELG_PAIRWISE_CONDENSED;
  if (x86 && eu && cond) FUELG_PW(ORDER_X86, METRIC_EUCLIDEAN, FUELG_PAIRWISE_CONDENSED);
  else if (x86 && eu) FUELG_PW(ORDER_X86, METRIC_EUCLIDEAN, FUELG_PAIRWISE_SQUARE);
  else if (x86 && cond) FUELG_PW(ORDER_X86, METRIC_SQEUCLIDEAN, FUELG_PAIRWISE_CONDENSED);
  else if (x86) FUELG_PW(ORDER_X86, METRIC_SQEUCLIDEAN, FUELG_PAIRWISE_SQUARE);
  else if (eu && cond) FUELG_PW(ORDER_ARM, METRIC_EUCLIDEAN, FUELG_PAIRWISE_CONDENSED);
  else if (eu) FUELG_PW(ORDER_ARM, METRIC_EUCLIDEAN, FUELG_PAIRWISE_SQUARE);
  else if (cond) FUELG_PW(ORDER_ARM, METRIC_SQEUCLIDEAN, FUELG_PAIRWISE_CONDENSED);
  else FUELG_PW(ORDER_ARM, METRIC_SQEUCLIDEAN, FUELG_PAIRWISE_SQUARE);
#undef FUELG_PW
  ::fuelg::note_launch();
  if (ht) ht->end(stream);
  FUELG_CUDA(cudaGetLastError());
  return ST_OK;
}

}  // namespace fuelg
