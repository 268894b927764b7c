// fuelg_tile.cuh -- register-tiled exact f32 distances of a 64 x 128 block of
// (row a, row b) pairs, the core of the kNN scan, the range search and the
// pairwise matrices.
//
// Each warp owns 8 a-rows; lane l holds the b-rows l, l + 32, l + 64, l + 96:
// 32 pairs per thread.  Both operands sit in shared memory dimension-major,
// so one dimension costs two broadcast 16-byte loads (the 8 a-values, the same
// for the whole warp) and four conflict-free 4-byte loads for 96 arithmetic
// instructions.  fuel's order (src/distance/squared_euclidean.rs:16-39 with
// FMA, :99-133 without) sums lane l's terms over the 8-blocks first and then
// the lanes left to right, so the dimensions are stored lane by lane
// (tile_pos) and a pair needs two registers -- the lane sum and the running
// total -- instead of nine.  A sum that starts at +0 is the first term itself
// (squares are >= +0 or NaN), so results are bit-identical.
#pragma once
#include "fuelg_common.cuh"

namespace fuelg {

constexpr int kTileQ = 8;             // a-rows per warp
constexpr int kTileP = 128;           // b-rows per tile
constexpr int kTilePS = kTileP + 1;   // b tile stride (floats): staged rows spread over the banks
constexpr int kTileMaxWarps = 8;

constexpr int kTileQS = kTileQ * kTileMaxWarps + 4;  // a tile stride: 16-byte aligned

// Storage position of dimension c: the d & ~7 leading dimensions lane by lane.
__device__ __forceinline__ int tile_pos(int c, int nb) { return c < 8 * nb ? (c & 7) * nb + (c >> 3) : c; }

__device__ __forceinline__ void cp_async4(uint32_t smem, const void* gmem, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem), "l"(gmem), "r"(bytes) : "memory");
}

// Stages rows [row0, row0 + rows) of src [total, d] dimension-major into dst
// (element (r, c) at tile_pos(c) * stride + r) with 4-byte asynchronous copies;
// rows past total are zero-filled.  The caller waits for the copies.  A thread
// keeps its column, so a copy costs two increments.
__device__ __forceinline__ void tile_stage(float* __restrict__ dst, int stride, const float* __restrict__ src,
                                           int64_t row0, int rows, int64_t total, int d, int nb) {
  const int T = blockDim.x;
  const int left = (int)min((int64_t)rows, total - row0);  // rows that exist (may be <= 0)
  const float* g0 = left > 0 ? src + row0 * d : src;
  if (d <= T) {
    const int rs = T / d;
    if ((int)threadIdx.x < rs * d) {
      const int r0 = threadIdx.x / d, c = threadIdx.x - r0 * d;
      uint32_t s = (uint32_t)__cvta_generic_to_shared(dst + tile_pos(c, nb) * stride + r0);
      const float* g = g0 + (int64_t)r0 * d + c;
      const int step = rs * d;
      if (left == rows) {
#pragma unroll 4
        for (int r = r0; r < rows; r += rs, g += step, s += 4 * rs) cp_async4(s, g, 4);
      } else {
        for (int r = r0; r < rows; r += rs, g += step, s += 4 * rs) cp_async4(s, r < left ? g : src, r < left ? 4 : 0);
      }
    }
  } else {
    for (int c = threadIdx.x; c < d; c += T) {
      const float* g = g0 + c;
      uint32_t s = (uint32_t)__cvta_generic_to_shared(dst + tile_pos(c, nb) * stride);
      for (int r = 0; r < rows; r++, g += d, s += 4) cp_async4(s, r < left ? g : src, r < left ? 4 : 0);
    }
  }
}

// Pairs of floats in one 64-bit register: half the issue slots.  Each half is
// the scalar operation's result: a difference as fma(b, -1, a) and a square as
// fma(x, x, -0) round once, as the subtraction and the product do (a square is
// never -0).  The -0 pair is a kernel argument (nz): ptxas turns a paired product,
// or an fma whose -0 it can see, into one fma with the add that follows, which
// rounds once where the reference rounds twice (seen as differing results).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
constexpr f32x2 kNegOne2 = 0xbf800000bf800000ull, kNegZero2 = 0x8000000080000000ull;  // kNegZero2: for nz

// One pair's next term: its square (FIRST), or s plus it.
template <bool FMA8, bool FIRST>
__device__ __forceinline__ f32x2 tile_term(f32x2 a, f32x2 b, f32x2 nz, f32x2 s) {
  const f32x2 df = fma2(b, kNegOne2, a);
  if (FIRST) return fma2(df, df, nz);
  return FMA8 ? fma2(df, df, s) : add2(fma2(df, df, nz), s);
}
__device__ __forceinline__ void tile_load_a(const float* __restrict__ q, f32x2 (&a)[4]) {
  const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(q), a1 = *reinterpret_cast<const ulonglong2*>(q + 4);
  a[0] = a0.x, a[1] = a0.y, a[2] = a1.x, a[3] = a1.y;
}

// The 8 x 4 pairs' sums with NB = d / 8 known: the NB terms of one SIMD lane of
// fuel's kernel go into a short-lived lane sum and then into the total, so a
// pair holds one register while the next lane's values are loaded.
template <bool FMA8, int NB>
__device__ __forceinline__ void tile_lanes(const float* __restrict__ q, const float* __restrict__ x, f32x2 nz,
                                           f32x2 (&s)[kTileQ / 2][4]) {
#pragma unroll 1
  for (int l = 0; l < 8; l++, q += NB * kTileQS, x += NB * kTilePS) {
    f32x2 a[NB][4];
#pragma unroll
    for (int k = 0; k < NB; k++) tile_load_a(q + k * kTileQS, a[k]);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      f32x2 b[NB];
#pragma unroll
      for (int k = 0; k < NB; k++) {
        const float xv = x[k * kTilePS + 32 * i];
        b[k] = pack2(xv, xv);
      }
#pragma unroll
      for (int j = 0; j < 4; j++) {
        f32x2 t = tile_term<FMA8, true>(a[0][j], b[0], nz, 0);
#pragma unroll
        for (int k = 1; k < NB; k++) t = tile_term<FMA8, false>(a[k][j], b[k], nz, t);
        s[j][i] = add2(s[j][i], t);  // (+0 + the first lane's sum is that sum)
      }
    }
  }
}

// The same for any nb: two b-rows at a time, lane sums held over the nb terms.
template <bool FMA8>
__device__ __forceinline__ void tile_lanes_any(const float* __restrict__ q0, const float* __restrict__ x0, int nb,
                                               f32x2 nz, f32x2 (&s)[kTileQ / 2][4]) {
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const float *q = q0, *x = x0 + 64 * h;
#pragma unroll 1
    for (int l = 0; l < 8; l++) {
      f32x2 acc[kTileQ / 2][2];
#pragma unroll 1
      for (int k = 0; k < nb; k++, q += kTileQS, x += kTilePS) {
        f32x2 a[4];
        tile_load_a(q, a);
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const f32x2 b = pack2(x[32 * i], x[32 * i]);
#pragma unroll
          for (int j = 0; j < 4; j++)
            acc[j][i] = k == 0 ? tile_term<FMA8, true>(a[j], b, nz, 0) : tile_term<FMA8, false>(a[j], b, nz, acc[j][i]);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int i = 0; i < 2; i++) s[j][2 * h + i] = add2(s[j][2 * h + i], acc[j][i]);
    }
  }
}

// out[j][i] = squared distance of a-row q[j] and b-row x[32 i]: q points at the
// warp's first a-row of the dimension-major a tile (stride kTileQS), x at the
// lane's first b-row (stride kTilePS).
template <bool FMA8>
__device__ __forceinline__ void tile_dists(const float* __restrict__ q, const float* __restrict__ x, int d, int nb,
                                           f32x2 nz, float (&out)[kTileQ][4]) {
  f32x2 s[kTileQ / 2][4];
#pragma unroll
  for (int j = 0; j < kTileQ / 2; j++)
#pragma unroll
    for (int i = 0; i < 4; i++) s[j][i] = 0;
  switch (nb) {  // rows of up to 32 dimensions with a lane's terms unrolled
    case 0: break;
    case 1: tile_lanes<FMA8, 1>(q, x, nz, s); break;
    case 2: tile_lanes<FMA8, 2>(q, x, nz, s); break;
    case 3: tile_lanes<FMA8, 3>(q, x, nz, s); break;
    default: tile_lanes_any<FMA8>(q, x, nb, nz, s); break;
  }
#pragma unroll 1
  for (int c = 8 * nb; c < d; c++) {  // the tail, one term after the other
    f32x2 a[4];
    tile_load_a(q + c * kTileQS, a);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float xv = x[c * kTilePS + 32 * i];
      const f32x2 b = pack2(xv, xv);
#pragma unroll
      for (int j = 0; j < 4; j++) s[j][i] = tile_term<FMA8, false>(a[j], b, nz, s[j][i]);
    }
  }
#pragma unroll
  for (int j = 0; j < kTileQ / 2; j++)
#pragma unroll
    for (int i = 0; i < 4; i++) unpack2(s[j][i], out[2 * j][i], out[2 * j + 1][i]);
}

// Smallest bit pattern of the warp-lane's four distances to a-row j.  Squared
// distances are >= +0 or the canonical NaN, so integer order is DistPair order
// with NaN last (a float minimum would drop the NaN).
__device__ __forceinline__ unsigned tile_min_bits(const float (&v)[4]) {
  return min(min(__float_as_uint(v[0]), __float_as_uint(v[1])), min(__float_as_uint(v[2]), __float_as_uint(v[3])));
}

// Largest squared-distance bit pattern whose key distance can be <= D: D
// itself, or for Euclidean keys a bound on D^2 rounded up far enough that every s
// with sqrt(s) <= D is below it; everything passes when D is NaN.
__device__ __forceinline__ unsigned tile_limit_bits(float D, int metric) {
  if (D != D) return 0xffffffffu;
  if (metric == METRIC_SQEUCLIDEAN) return __float_as_uint(D);
  return __float_as_uint(__fadd_ru(__fmul_ru(__fmul_ru(D, D), 1.000001f), 3e-45f));
}

}  // namespace fuelg
