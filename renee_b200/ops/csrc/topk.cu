// Row selection behind the fused top-k GEMM (gemm.cu, epilogue TOPK): the k best of a row's candidates, in order, with
// the labels of lists that may have dropped one of them recomputed.
//
// The GEMM leaves, per row, one list of the 8 best for every (unit, column group) that met the row.  Let t be the k-th
// best of all candidates.  An entry above t can only be missing from a list whose own 8th entry is above t, and fewer
// than k candidates are above t, so at most (k - 1) / 8 lists of a row are in doubt -- none for k <= 8, and for k = 100
// over a million labels one row in some thousands when the labels are in no particular order.  The logits of such a
// list's labels are formed again here, directly, in place of the list.  Rows with fewer than k
// candidates in all (few labels, or logits of -inf) have t = nothing and every list in doubt, which is the same path.
// So the result is exact for any order of the labels, with a bounded worst case.
//
// One CTA per row.  The selection is a binary search for the k-th largest key: each step is one sweep over the keys and
// one block-wide count, where the radix select it replaces serialised on the
// few histogram bins that logits of similar size share (256 rows x 2368 candidates, k = 5: 36 us and 35 us more of
// library sort and gather launches -> 26 us, 9 with the keys in registers).  The whole call: 512 rows x 1.3 M labels,
// k = 100, 9.40 -> 1.07 ms (before: fp32 logits written chunk by chunk and a selection over each chunk); 256 x 131 K, k = 5,
// 187 -> 88 us.
#include "topk.cuh"

namespace rb {
namespace tk {

constexpr int THREADS = 256;
constexpr int MAX_K = 256;          // winners are sorted by one thread each
constexpr int EXTRA = 1024;         // recomputed entries that fit beside the candidates before a selection makes room
constexpr int TILE_COLS = 64;       // most columns a list has in one tile

struct Args {
  const float* cand_val; const int* cand_idx; int per_row;      // candidates
  int ncta, bn, units, n_n, n_m;                                // how the GEMM spread the tiles
  int B, Ls, D, ldx, ldw, k;
  float* out_val; long long* out_idx;
};

// The kk-th largest key of key[0 .. n) (0 if fewer than kk keys are non-zero); the same value in every thread.
__device__ uint32_t kth_key(const uint32_t* key, int n, int kk, int* s_count) {
  uint32_t t = 0u;
  for (int bit = 31; bit >= 0; --bit) {
    const uint32_t trial = t | (1u << bit);
    int c = 0;
    for (int i = threadIdx.x; i < n; i += THREADS) c += key[i] >= trial ? 1 : 0;
    c = __reduce_add_sync(0xffffffffu, c);
    int* cnt = s_count + (bit & 1) * (THREADS / 32);            // two sets: one barrier per step
    if ((threadIdx.x & 31) == 0) cnt[threadIdx.x >> 5] = c;
    __syncthreads();
    int total = 0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) total += cnt[w];
    if (total >= kk) t = trial;
  }
  __syncthreads();
  return t;
}

// The same for the candidates alone, with each thread's share of the keys in registers and two bits per step: 16 steps of
// three counts (13 bits each fit two words), 1 us where 32 sweeps of shared memory took 15 of the kernel's 26 us.
template <int NPT>
__device__ uint32_t kth_key_reg(const uint32_t* key, int n, int kk, int* s_count) {
  uint32_t k[NPT];
#pragma unroll
  for (int u = 0; u < NPT; ++u) { const int i = threadIdx.x + u * THREADS; k[u] = i < n ? key[i] : 0u; }
  uint32_t t = 0u;
#pragma unroll 1
  for (int sh = 30; sh >= 0; sh -= 2) {
    const uint32_t t1 = t | (1u << sh), t2 = t | (2u << sh), t3 = t | (3u << sh);
    uint32_t c12 = 0u, c3 = 0u;
#pragma unroll
    for (int u = 0; u < NPT; ++u) {
      c12 += (k[u] >= t1 ? 1u : 0u) + (k[u] >= t2 ? 0x10000u : 0u);
      c3 += k[u] >= t3 ? 1u : 0u;
    }
    c12 = __reduce_add_sync(0xffffffffu, c12);
    c3 = __reduce_add_sync(0xffffffffu, c3);
    uint2* cnt = reinterpret_cast<uint2*>(s_count) + ((sh >> 1) & 1) * (THREADS / 32);
    if ((threadIdx.x & 31) == 0) cnt[threadIdx.x >> 5] = make_uint2(c12, c3);
    __syncthreads();
    uint32_t s12 = 0u, s3 = 0u;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) { const uint2 c = cnt[w]; s12 += c.x; s3 += c.y; }
    if ((int)s3 >= kk) t = t3;
    else if ((int)(s12 >> 16) >= kk) t = t2;
    else if ((int)(s12 & 0xffffu) >= kk) t = t1;
  }
  __syncthreads();
  return t;
}

// Writes the kk largest entries of the pool to win[0 .. kk), in any order, and 0 behind them.
__device__ void gather_best(const uint32_t* key, const int* idx, int n, int kk, uint32_t t, unsigned long long* win, int* s_slots) {
  for (int i = threadIdx.x; i < MAX_K; i += THREADS) win[i] = 0ull;
  if (threadIdx.x < 2) s_slots[threadIdx.x] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += THREADS)
    if (key[i] > t) {
      const int s = atomicAdd(s_slots, 1);                      // fewer than kk of them
      if (s < kk) win[s] = ((unsigned long long)key[i] << 32) | (0xffffffffu - (uint32_t)idx[i]);
    }
  __syncthreads();
  const int above = min(s_slots[0], kk);
  for (int i = threadIdx.x; i < n; i += THREADS)
    if (key[i] == t && t != 0u) {
      const int s = above + atomicAdd(s_slots + 1, 1);
      if (s < kk) win[s] = ((unsigned long long)key[i] << 32) | (0xffffffffu - (uint32_t)idx[i]);
    }
  __syncthreads();
}

template <typename T>
__global__ void __launch_bounds__(THREADS) topk_select_kernel(const Args a, const T* __restrict__ X, const T* __restrict__ W) {
  extern __shared__ __align__(16) uint8_t sm[];
  const int cap = a.per_row + EXTRA;
  unsigned long long* win = reinterpret_cast<unsigned long long*>(sm);            // [MAX_K]
  uint32_t* key = reinterpret_cast<uint32_t*>(win + MAX_K);                       // [cap]
  int* idx = reinterpret_cast<int*>(key + cap);                                   // [cap]
  uint8_t* doubt = reinterpret_cast<uint8_t*>(idx + cap);                         // [per_row / 8] lists to recompute
  __shared__ __align__(8) int s_count[4 * (THREADS / 32)];
  __shared__ int s_slots[2];
  __shared__ int s_extra, s_any;
  const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int mt = row / (128 * a.ncta);
  int first, step;
  topk_range(mt, a.n_m, a.n_n, first, step);
  const int ucols = max(32, a.bn / TOPK_GROUPS);
  const int n_lists = a.per_row / TOPK_LIST;
  const float* cv = a.cand_val + (size_t)row * a.per_row;
  const int* ci = a.cand_idx + (size_t)row * a.per_row;
  if (tid == 0) { s_extra = 0; s_any = 0; }
  for (int i = tid; i < cap; i += THREADS) {
    uint32_t kx = 0u;
    int id = 0;
    if (i < a.per_row) {
      const int list = i / TOPK_LIST;
      // lists of units that never met this row, and of groups without columns, were not written
      if ((list % TOPK_GROUPS) * ucols < a.bn && topk_unit_first(list / TOPK_GROUPS, a.units, first, step, a.n_n) >= 0) {
        id = ci[i];
        if (id >= 0) kx = order_key(cv[i]);
      }
    }
    key[i] = kx;
    idx[i] = id;
  }
  __syncthreads();
  uint32_t t;
  if (a.per_row <= 10 * THREADS) t = kth_key_reg<10>(key, a.per_row, a.k, s_count);
  else if (a.per_row <= 20 * THREADS) t = kth_key_reg<20>(key, a.per_row, a.k, s_count);
  else t = kth_key(key, a.per_row, a.k, s_count);
  for (int l = tid; l < n_lists; l += THREADS) {
    const bool met = (l % TOPK_GROUPS) * ucols < a.bn && topk_unit_first(l / TOPK_GROUPS, a.units, first, step, a.n_n) >= 0;
    const bool in_doubt = met && (t == 0u || key[l * TOPK_LIST + TOPK_LIST - 1] > t);
    doubt[l] = in_doubt ? 1 : 0;
    if (in_doubt) s_any = 1;
  }
  __syncthreads();
  int n = a.per_row;
  if (s_any) {
    for (int i = tid; i < a.per_row; i += THREADS)               // their entries come back with the recomputed ones
      if (doubt[i / TOPK_LIST]) key[i] = 0u;
    n = cap;
    __syncthreads();
    // what is left bounds the result from below; the t above does not, since sums formed here round differently
    t = kth_key(key, a.per_row, a.k, s_count);
    const T* x = X + (size_t)row * a.ldx;
    for (int l = 0; l < n_lists; ++l) {
      if (!doubt[l]) continue;
      const int c_lo = (l % TOPK_GROUPS) * ucols, c_hi = min(a.bn, c_lo + ucols);
      for (int tile = topk_unit_first(l / TOPK_GROUPS, a.units, first, step, a.n_n); tile < first + step * a.n_n; tile += a.units) {
        // every thread reads the count between two barriers, so all take the branch (which has barriers of its own) or
        // none: without the second one a fast warp's first append of this tile could still change what a slow warp reads
        const bool full = s_extra + TILE_COLS > EXTRA;
        __syncthreads();
        if (full) {                                              // make room: keep the k best so far
          t = kth_key(key, cap, a.k, s_count);
          gather_best(key, idx, cap, a.k, t, win, s_slots);
          for (int i = tid; i < cap; i += THREADS) {
            key[i] = i < a.k ? (uint32_t)(win[i] >> 32) : 0u;
            idx[i] = i < a.k ? (int)(0xffffffffu - (uint32_t)win[i]) : 0;
          }
          if (tid == 0) s_extra = max(0, a.k - a.per_row);
          __syncthreads();
        }
        const int n0 = (tile - first) / step * a.bn;
        for (int c = c_lo + warp; c < c_hi; c += THREADS / 32) {
          const int label = n0 + c;
          if (label >= a.Ls) break;
          const T* w = W + (size_t)label * a.ldw;
          float s = 0.f;
          for (int d = lane; d < a.D; d += 32) s = fmaf(to_f(x[d]), to_f(w[d]), s);
          s = warp_sum(s);
          if (lane == 0) {
            const uint32_t kx = order_key(topk_store_value(s));
            if (kx >= t) {
              const int e = a.per_row + atomicAdd(&s_extra, 1);
              key[e] = kx;
              idx[e] = label;
            }
          }
        }
        __syncthreads();
      }
    }
    t = kth_key(key, cap, a.k, s_count);
  }
  gather_best(key, idx, n, a.k, t, win, s_slots);
  // bitonic sort, descending: by value, then by the lower label (the low word holds its complement)
  int size = 32;
  while (size < a.k) size <<= 1;
  for (int len = 2; len <= size; len <<= 1)
    for (int j = len >> 1; j > 0; j >>= 1) {
      const int o = tid ^ j;
      if (tid < size && o > tid) {
        const unsigned long long p = win[tid], q = win[o];
        if (((tid & len) == 0) == (p < q)) { win[tid] = q; win[o] = p; }
      }
      __syncthreads();
    }
  if (tid < a.k) {
    const unsigned long long p = win[tid];
    a.out_val[(size_t)row * a.k + tid] = topk_load_value(key_value((uint32_t)(p >> 32)));
    a.out_idx[(size_t)row * a.k + tid] = (long long)(0xffffffffu - (uint32_t)p);
  }
}

template <typename T>
static int launch(const Args& a, const void* X, const void* W, cudaStream_t st) {
  const size_t smem = MAX_K * 8 + (size_t)(a.per_row + EXTRA) * 8 + a.per_row / TOPK_LIST;
  auto k = topk_select_kernel<T>;
  if (smem > 48 * 1024 && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -5;
  k<<<a.B, THREADS, smem, st>>>(a, (const T*)X, (const T*)W);
  return 0;
}

}  // namespace tk
}  // namespace rb

using namespace rb;

RB_API int rb_topk_max_k(void) { return tk::MAX_K; }

// The k (<= rb_topk_max_k(), <= Ls) largest logits of every row of X [B, ldx >= D] against W [Ls, ldw >= D], descending,
// with their labels, from the candidates that rb_xfc_topk_candidates left; plan = rb_xfc_topk_plan's output for the shape.
RB_API int rb_topk_select(int dtype, const float* cand_val, const int* cand_idx, const int* plan, const void* X, const void* W,
                          int B, int Ls, int D, int ldx, int ldw, int k, float* out_val, long long* out_idx, cudaStream_t st) {
  if (dtype != RB_BF16 && dtype != RB_F16) return -1;
  if (B < 1 || k < 1 || k > tk::MAX_K || k > Ls) return -3;
  tk::Args a{};
  a.cand_val = cand_val; a.cand_idx = cand_idx; a.per_row = plan[5];
  a.ncta = plan[0]; a.bn = plan[1]; a.units = plan[2]; a.n_n = plan[3]; a.n_m = plan[4];
  a.B = B; a.Ls = Ls; a.D = D; a.ldx = ldx; a.ldw = ldw; a.k = k; a.out_val = out_val; a.out_idx = out_idx;
  const int rc = dtype == RB_BF16 ? tk::launch<__nv_bfloat16>(a, X, W, st) : tk::launch<__half>(a, X, W, st);
  if (rc) return rc;
  RB_LAUNCH_CHECK();
  return 0;
}
