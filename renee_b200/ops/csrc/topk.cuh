// Shared by the fused top-k GEMM (gemm.cu, epilogue TOPK) and the row selection (topk.cu).
#pragma once
#include "common.cuh"

namespace rb {

constexpr int TOPK_GROUPS = 4;      // epilogue groups per CTA: each takes max(32, BN / 4) columns of a tile
constexpr int TOPK_LIST = 8;        // entries a thread keeps

// Tile number -> (M tile, N tile): M tiles in pairs, the two of a pair interleaved; a last single one in order.
__host__ __device__ __forceinline__ void topk_tile(int tile, int n_m, int n_n, int& mt, int& nt) {
  const int q = tile / (2 * n_n), l = tile - q * 2 * n_n;
  if (2 * q + 1 < n_m) { mt = 2 * q + (l & 1); nt = l >> 1; }
  else { mt = 2 * q; nt = l; }
}

// First tile number and step between the tiles of M tile mt.
__host__ __device__ __forceinline__ void topk_range(int mt, int n_m, int n_n, int& first, int& step) {
  const int q = mt >> 1;
  if (2 * q + 1 < n_m) { first = q * 2 * n_n + (mt & 1); step = 2; }
  else { first = q * 2 * n_n; step = 1; }
}

// The first tile of M tile mt that `unit` of `units` works on, or -1.  Its further ones follow in steps of `units` (a
// unit with several tiles keeps one M tile: the number of units is even then).
__host__ __device__ __forceinline__ int topk_unit_first(int unit, int units, int first, int step, int n_n) {
  int o = (unit - first) % units;
  if (o < 0) o += units;
  if (o % step != 0 || o / step >= n_n) return -1;
  return first + o;
}

__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
// A NaN logit ranks above all others, +inf included, as in torch.topk.  In the lists, where values are compared as floats, a
// NaN travels as +inf and +inf as the largest finite float, which no product of 16-bit operands reaches; the result has them
// back.
__device__ __forceinline__ float topk_store_value(float x) {
  return x != x ? INFINITY : fminf(x, 3.402823466e38f);
}
__device__ __forceinline__ float topk_load_value(float x) {
  return x == INFINITY ? __int_as_float(0x7fffffff) : (x == 3.402823466e38f ? INFINITY : x);
}

// fp32 -> unsigned with the same order; 0 is smaller than the key of every stored value
__device__ __forceinline__ uint32_t order_key(float x) {
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

}  // namespace rb
