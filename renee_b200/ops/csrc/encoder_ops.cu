// Fused encoder kernels (memory-bound, one pass over the activations each):
//   embed_ln_fwd / embed_ln_bwd            word+position gather, LayerNorm, dropout (+ scatter of gradients)
//   bias_dropout_add_ln_fwd / _bwd         y = LN(resid + dropout(x + bias))
//   bias_gelu_fwd / _bwd                   exact-erf GELU with the bias add and the bias gradient fused
//   pool_fwd / pool_bwd                    mask-weighted mean or CLS pooling
//   dropout_cast_fwd / dropout_bwd         classifier-input dropout
//   colsum                                 column sums (bias gradients)
// They stand in for the ATen/Inductor kernels behind the HF encoder the reference runs
// (dl_base.py:121-141 and the DistilBERT blocks it wraps).  Rows are handled one warp each with
// 16-byte accesses; column reductions (dgamma, dbeta, dbias) are accumulated in registers across the
// rows of a warp, combined per block in shared memory, added to an fp32 accumulator in global memory
// and converted by the last block to finish, which also re-zeroes the accumulator for the next call.
#include <cstdio>
#include "common.cuh"
#include "token_map.cuh"

namespace rb {


template <typename T> __device__ __forceinline__ void atomic_add8(T* p, const float (&v)[8]);
template <> __device__ __forceinline__ void atomic_add8<float>(float* p, const float (&v)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) atomicAdd(p + i, v[i]);
}
// 16 bytes per reduction instead of 4 (p is 16-byte aligned: rows and columns are multiples of 8 elements)
template <> __device__ __forceinline__ void atomic_add8<__nv_bfloat16>(__nv_bfloat16* p, const float (&v)[8]) {
  const uint4 r = pack16x8<__nv_bfloat16>(v);
  asm volatile("red.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(r.x), "r"(r.y), "r"(r.z), "r"(r.w) : "memory");
}
template <> __device__ __forceinline__ void atomic_add8<__half>(__half* p, const float (&v)[8]) {
  const uint4 r = pack16x8<__half>(v);
  asm volatile("red.global.add.noftz.v4.f16x2 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(r.x), "r"(r.y), "r"(r.z), "r"(r.w) : "memory");
}

// Last-block-done column reduction epilogue.  Every block has already added its partial sums to one of
// kCopies replicas of acc[n_vec][H] (fp32, global; replica = block index mod kCopies, which divides the
// same-address atomic traffic by kCopies).  The last block sums the replicas, converts to the outputs
// and clears the accumulator.
constexpr int kCopies = 8;

__device__ __forceinline__ float* acc_replica(float* acc, int n_vec, int H) {
  const unsigned blk = blockIdx.y * gridDim.x + blockIdx.x;
  return acc + (size_t)(blk % kCopies) * n_vec * H;
}

template <typename T>
__device__ void finalize_columns(float* acc, unsigned* counter, int n_vec, int H, T* o0, T* o1, T* o2) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned done = atomicAdd(counter, 1u);
    last = (done == gridDim.x * gridDim.y - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int tot = n_vec * H;
  // four column groups per round so that 32 independent loads are in flight per thread
  for (int base = 0; base < tot; base += 4 * blockDim.x) {
    float v[4][kCopies];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = base + u * blockDim.x + threadIdx.x;
#pragma unroll
      for (int k = 0; k < kCopies; ++k) v[u][k] = (i < tot) ? __ldcg(acc + (size_t)k * tot + i) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = base + u * blockDim.x + threadIdx.x;
      if (i < tot) {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < kCopies; ++k) { s += v[u][k]; acc[(size_t)k * tot + i] = 0.f; }
        const int which = i / H;
        T* o = which == 0 ? o0 : (which == 1 ? o1 : o2);
        if (o != nullptr) o[i - which * H] = from_f<T>(s);
      }
    }
  }
  if (threadIdx.x == 0) *counter = 0u;
}

// Deferred variant: kernels called with counter == nullptr only accumulate into their own replica block;
// one launch of this kernel at the end of the backward pass then converts ALL pending column sums
// (LayerNorm gammas/betas, every bias gradient) and clears the accumulators — one serial tail per step
// instead of one per kernel.  Row r of the table: {acc base, out pointer, tot, v_off, len}.
struct ColumnJob { const float* acc; void* out; int tot; int v_off; int len; int pad; };

template <typename T>
__global__ void __launch_bounds__(256) finalize_jobs_kernel(const ColumnJob* __restrict__ jobs) {
  const ColumnJob j = jobs[blockIdx.x];
  float* acc = const_cast<float*>(j.acc);
  T* out = reinterpret_cast<T*>(j.out);
  for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < j.len; c += gridDim.y * blockDim.x) {
    float v[kCopies];
#pragma unroll
    for (int k = 0; k < kCopies; ++k) v[k] = __ldcg(acc + (size_t)k * j.tot + j.v_off + c);
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < kCopies; ++k) { s += v[k]; acc[(size_t)k * j.tot + j.v_off + c] = 0.f; }
    out[c] = from_f<T>(s);
  }
}

// ------------------------------------------------------------------------------------ LN forward
template <typename T, int NV>
__global__ void __launch_bounds__(128) bias_dropout_add_ln_fwd_kernel(
    const T* __restrict__ x, const T* __restrict__ bias, const T* __restrict__ resid,
    const T* __restrict__ gamma, const T* __restrict__ beta, T* __restrict__ y, T* __restrict__ pre,
    float* __restrict__ mean, float* __restrict__ rstd, int rows, int H, float eps, float p,
    const int* __restrict__ seed_ptr, uint32_t stream) {
  const int lane = threadIdx.x & 31;
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (row >= rows) return;
  const uint32_t seed = p > 0.f ? (uint32_t)(*seed_ptr) : 0u;
  const float inv_keep = p > 0.f ? 1.f / (1.f - p) : 1.f;
  float v[NV][8];
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = (lane + 32 * i) * 8;
    if (col < H) {
      float a[8], b[8], r[8];
      load8(x + (size_t)row * H + col, a);
      load8(bias + col, b);
      load8(resid + (size_t)row * H + col, r);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float t = a[j] + b[j];
        if (p > 0.f) t = keep(seed, stream, (uint32_t)(row * H + col + j), p) ? t * inv_keep : 0.f;
        v[i][j] = round_through<T>(r[j] + t);
        sum += v[i][j];
      }
      store8(pre + (size_t)row * H + col, v[i]);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] = 0.f;
    }
  }
  const float mu = warp_sum(sum) / H;
  float sq = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = (lane + 32 * i) * 8;
    if (col < H) {
#pragma unroll
      for (int j = 0; j < 8; ++j) { float d = v[i][j] - mu; sq += d * d; }
    }
  }
  const float rs = rsqrtf(warp_sum(sq) / H + eps);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = (lane + 32 * i) * 8;
    if (col < H) {
      float g[8], b[8], o[8];
      load8(gamma + col, g);
      load8(beta + col, b);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = (v[i][j] - mu) * rs * g[j] + b[j];
      store8(y + (size_t)row * H + col, o);
    }
  }
  if (lane == 0) { mean[row] = mu; rstd[row] = rs; }
}

// Per-sequence counts of the token map and their prefix sum.  A group of G = min(32, S rounded up to a power of two)
// lanes reads one mask row, 32 / G rows per warp; the last CTA to finish scans the B counts (one contiguous run per
// thread).  Latency-bound: a few dependent loads and two block scans, whatever the batch.
__global__ void __launch_bounds__(1024) token_map_kernel(const int* __restrict__ mask, int B, int S, int G,
                                                         int* __restrict__ off, int* __restrict__ len,
                                                         int* __restrict__ cnt, int* __restrict__ meta) {
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int per_warp = 32 / G, lig = lane % G, grp = lane / G;
  const unsigned gmask = (G == 32 ? 0xffffffffu : (1u << G) - 1u);
  for (int b0 = (blockIdx.x * 32 + wib) * per_warp; b0 < B; b0 += gridDim.x * 32 * per_warp) {
    const int b = b0 + grp;
    int n = 0, last = -1, first = 0;
    for (int s0 = 0; s0 < S; s0 += G) {                       // the same trip count in every lane
      const int s = s0 + lig;
      const bool on = b < B && s < S && mask[(size_t)b * S + s] != 0;
      const unsigned bits = (__ballot_sync(0xffffffffu, on) >> (grp * G)) & gmask;
      n += __popc(bits);
      if (bits) last = s0 + 31 - __clz(bits);
      if (s0 == 0) first = bits & 1u;
    }
    if (lig == 0 && b < B) {
      off[b] = n == 0 ? S : n + (first ? 0 : 1);
      len[b] = n == 0 ? S : max(last + 1, 1);
      cnt[b] = n;
    }
  }
  __shared__ int s_last;
  __shared__ int s_part[32];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(meta + TOK_COUNTER, 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const int per = (B + 1023) / 1024, lo = min(B, (int)threadIdx.x * per), hi = min(B, lo + per);
  int sum = 0;
  for (int b = lo; b < hi; ++b) sum += __ldcg(off + b);
  int inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += v; }
  if (lane == 31) s_part[wib] = inc;
  __syncthreads();
  if (wib == 0) {
    int v = s_part[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += u; }
    s_part[lane] = v;
  }
  __syncthreads();
  int run = inc - sum + (wib > 0 ? s_part[wib - 1] : 0);
  for (int b = lo; b < hi; ++b) { const int c = __ldcg(off + b); off[b] = run; run += c; }
  if (threadIdx.x == 0) {
    const int total = s_part[31];
    meta[TOK_VALID] = total;
    meta[TOK_ROWS] = min(B * S, (total + TOK_ALIGN - 1) / TOK_ALIGN * TOK_ALIGN);
    meta[TOK_COUNTER] = 0;
  }
}

// With a token map (meta != nullptr): the warp of padded token `row` works out its packed row from the sequence's offset
// and mask row, records the pair in tok / slot, and writes there; warps of dropped tokens only record -1, and up to
// TOK_ALIGN - 1 warps past the last token fill the zero rows.
template <typename T, int NV>
__global__ void __launch_bounds__(128) embed_ln_fwd_kernel(
    const int* __restrict__ ids, const T* __restrict__ word, const T* __restrict__ pos,
    const T* __restrict__ gamma, const T* __restrict__ beta, T* __restrict__ y,
    float* __restrict__ mean, float* __restrict__ rstd, int rows, int H, int S, float eps, float p,
    const int* __restrict__ seed_ptr, uint32_t stream, const int* __restrict__ mask, const int* __restrict__ meta,
    const int* __restrict__ off, const int* __restrict__ cnt, int* __restrict__ tok, int* __restrict__ slot) {
  grid_dep_launch();
  const int lane = threadIdx.x & 31;
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int out = row;                                              // row of y, mean and rstd
  if (meta != nullptr) {
    if (row >= rows) {
      out = meta[TOK_VALID] + (row - rows);
      if (out >= meta[TOK_ROWS]) return;
      const float zero[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int col = lane * 8; col < H; col += 256) store8(y + (size_t)out * H + col, zero);
      if (lane == 0) { mean[out] = 0.f; rstd[out] = 0.f; tok[out] = -1; }
      return;
    }
    const int b = row / S, s = row - b * S;
    const bool all = cnt[b] == 0;
    int before = 0;
    for (int s0 = 0; s0 <= s; s0 += 32) {                     // kept tokens of the row up to and including s
      const int q = s0 + lane;
      before += __popc(__ballot_sync(0xffffffffu, q <= s && (q == 0 || all || mask[(size_t)b * S + q] != 0)));
    }
    const bool kept = s == 0 || all || mask[row] != 0;
    out = kept ? off[b] + before - 1 : -1;
    if (lane == 0) { slot[row] = out; if (kept) tok[out] = row; }
    if (!kept) return;
  }
  if (row >= rows) return;
  const uint32_t seed = p > 0.f ? (uint32_t)(*seed_ptr) : 0u;
  const float inv_keep = p > 0.f ? 1.f / (1.f - p) : 1.f;
  const int id = ids[row];
  const int s = row % S;
  float v[NV][8];
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = (lane + 32 * i) * 8;
    if (col < H) {
      float a[8], b[8];
      load8(word + (size_t)id * H + col, a);
      load8(pos + (size_t)s * H + col, b);
#pragma unroll
      for (int j = 0; j < 8; ++j) { v[i][j] = a[j] + b[j]; sum += v[i][j]; }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] = 0.f;
    }
  }
  const float mu = warp_sum(sum) / H;
  float sq = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = (lane + 32 * i) * 8;
    if (col < H) {
#pragma unroll
      for (int j = 0; j < 8; ++j) { float d = v[i][j] - mu; sq += d * d; }
    }
  }
  const float rs = rsqrtf(warp_sum(sq) / H + eps);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = (lane + 32 * i) * 8;
    if (col < H) {
      float g[8], b[8], o[8];
      load8(gamma + col, g);
      load8(beta + col, b);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float t = (v[i][j] - mu) * rs * g[j] + b[j];
        if (p > 0.f) t = keep(seed, stream, (uint32_t)(row * H + col + j), p) ? t * inv_keep : 0.f;
        o[j] = t;
      }
      store8(y + (size_t)out * H + col, o);
    }
  }
  if (lane == 0) { mean[out] = mu; rstd[out] = rs; }
}

// ------------------------------------------------------------------------------------ LN backward
// EMBED = false: inputs dy, pre;   outputs d_pre, d_branch (if p > 0), dgamma, dbeta, dbias.
// EMBED = true : inputs dy (dropout re-applied to it), ids/word/pos to rebuild the LN input; outputs
//                dgamma, dbeta and gradients scattered into dword (atomic, pad id skipped) and dpos.
//                The launch makes the total warp count a multiple of S so a warp sees one position.
// Column sums are accumulated per warp in shared memory (a lane only touches its own columns, so no
// atomics are needed there), which keeps the register count low enough for 4+ CTAs per SM.
__device__ __forceinline__ void smem_add8(float* p, const float (&v)[8]) {
  float4 a = *reinterpret_cast<float4*>(p), b = *reinterpret_cast<float4*>(p + 4);
  a.x += v[0]; a.y += v[1]; a.z += v[2]; a.w += v[3];
  b.x += v[4]; b.y += v[5]; b.z += v[6]; b.w += v[7];
  *reinterpret_cast<float4*>(p) = a;
  *reinterpret_cast<float4*>(p + 4) = b;
}

template <typename T, int NV, bool EMBED, int WARPS = 4>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 4 ? (EMBED ? 5 : 6) : (WARPS == 8 ? 2 : 1)) ln_bwd_kernel(
    const T* __restrict__ dy, const T* __restrict__ pre, const int* __restrict__ ids,
    const T* __restrict__ word, const T* __restrict__ pos, const T* __restrict__ gamma,
    const float* __restrict__ mean, const float* __restrict__ rstd,
    T* __restrict__ d_pre, T* __restrict__ d_branch, T* __restrict__ dword, T* __restrict__ dpos,
    float* __restrict__ acc, unsigned* __restrict__ counter, T* __restrict__ dgamma, T* __restrict__ dbeta,
    T* __restrict__ dbias, int rows, int H, int S, int pad_id, float p, const int* __restrict__ seed_ptr,
    uint32_t stream, const int* __restrict__ tok_meta, const int* __restrict__ tok) {
  // packed tokens (token_map.cuh): EMBED walks the padded layout and tok is its slot array (dropped tokens are skipped);
  // otherwise the rows are the packed ones and tok numbers their dropout counters
  grid_dep_wait();            // launched with launch_pdl: nothing above touches global memory
  grid_dep_launch();
  if (!EMBED && tok_meta != nullptr) rows = __ldcg(tok_meta + TOK_ROWS);
  extern __shared__ __align__(16) float sm[];  // [warps][3][H]
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int wpb = blockDim.x >> 5;
  const int warp = blockIdx.x * wpb + wib;
  const int total_warps = gridDim.x * wpb;
  const uint32_t seed = p > 0.f ? (uint32_t)(*seed_ptr) : 0u;
  const float inv_keep = p > 0.f ? 1.f / (1.f - p) : 1.f;
  for (int i = threadIdx.x; i < wpb * 3 * H; i += blockDim.x) sm[i] = 0.f;
  __syncthreads();
  float* s_dg = sm + (size_t)wib * 3 * H;
  float* s_db = s_dg + H;
  float* s_x = s_db + H;    // dbias (resid mode) or position-embedding gradient (embed mode)

  Raw8<T> gam[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = (lane + 32 * i) * 8;
    if (col < H) gam[i] = load_raw8<T>(gamma + col);
  }
  // EMBED: the next token's packed row and id are on their way while this one is worked on (every load of a token hangs
  // on them), and a dropout decision is hashed once: 128 x 128 tokens 61 -> 43 us
  int next_row = -1, next_id = 0;
  if (EMBED && warp < rows) {
    next_row = tok != nullptr ? __ldcg(tok + warp) : warp;
    next_id = ids[warp];
  }
  for (int row0 = warp; row0 < rows; row0 += total_warps) {
    const int row = EMBED ? next_row : row0;                                   // row of the stored activations
    const int id = EMBED ? next_id : 0;
    if (EMBED && row0 + total_warps < rows) {
      next_row = tok != nullptr ? __ldcg(tok + row0 + total_warps) : row0 + total_warps;
      next_id = ids[row0 + total_warps];
    }
    if (EMBED && row < 0) continue;
    uint32_t kept[EMBED ? (NV + 3) / 4 : 1] = {};                              // dropout decisions, bit 8 (i % 4) + j
    const int crow = !EMBED && tok != nullptr && p > 0.f ? __ldcg(tok + row0) : row0;   // row of the dropout counters
    const float mu = mean[row], rs = rstd[row];
    // dy and the LN input stay packed across the two warp reductions
    Raw8<T> rd[NV], rx[NV], rb[NV];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (lane + 32 * i) * 8;
      if (col < H) {
        rd[i] = load_raw8<T>(dy + (size_t)row * H + col);
        if (EMBED) {
          rx[i] = load_raw8<T>(word + (size_t)id * H + col);
          rb[i] = load_raw8<T>(pos + (size_t)(row0 % S) * H + col);
        } else {
          rx[i] = load_raw8<T>(pre + (size_t)row * H + col);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (lane + 32 * i) * 8;
      if (col < H) {
        float d[8], x[8], gm[8], dgv[8];
        unpack8<T>(rd[i], d);
        unpack8<T>(rx[i], x);
        unpack8<T>(gam[i], gm);
        if (EMBED) {
          float b[8];
          unpack8<T>(rb[i], b);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            x[j] += b[j];
            if (p > 0.f) {
              const bool on = keep(seed, stream, (uint32_t)(crow * H + col + j), p);
              if (on) kept[EMBED ? i / 4 : 0] |= 1u << (8 * (i % 4) + j);
              d[j] = on ? d[j] * inv_keep : 0.f;
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = (x[j] - mu) * rs;
          const float g = d[j] * gm[j];
          s1 += g;
          s2 += g * xh;
          dgv[j] = d[j] * xh;
        }
        smem_add8(s_dg + col, dgv);
        smem_add8(s_db + col, d);
      }
    }
    s1 = warp_sum(s1) / H;
    s2 = warp_sum(s2) / H;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (lane + 32 * i) * 8;
      if (col < H) {
        float d[8], x[8], gm[8], dx[8];
        unpack8<T>(rd[i], d);
        unpack8<T>(rx[i], x);
        unpack8<T>(gam[i], gm);
        if (EMBED) {
          float b[8];
          unpack8<T>(rb[i], b);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            x[j] += b[j];
            if (p > 0.f) d[j] = (kept[EMBED ? i / 4 : 0] >> (8 * (i % 4) + j)) & 1u ? d[j] * inv_keep : 0.f;
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = (x[j] - mu) * rs;
          dx[j] = (d[j] * gm[j] - s1 - xh * s2) * rs;
        }
        if (EMBED) {
          if (id != pad_id) atomic_add8(dword + (size_t)id * H + col, dx);
          smem_add8(s_x + col, dx);
        } else {
          store8(d_pre + (size_t)row * H + col, dx);
          float db[8];
          if (p > 0.f) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              db[j] = round_through<T>(keep(seed, stream, (uint32_t)(crow * H + col + j), p) ? dx[j] * inv_keep : 0.f);
            store8(d_branch + (size_t)row * H + col, db);
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) db[j] = round_through<T>(dx[j]);
          }
          smem_add8(s_x + col, db);
        }
      }
    }
  }
  __syncwarp();
  if (EMBED && warp < rows) {
    const int s = warp % S;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (lane + 32 * i) * 8;
      if (col < H) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = s_x[col + j];
        atomic_add8(dpos + (size_t)s * H + col, v);
      }
    }
  }
  __syncthreads();
  const int nvec = EMBED ? 2 : 3;
  float* my_acc = acc_replica(acc, nvec, H);
  for (int i = threadIdx.x * 4; i < nvec * H; i += blockDim.x * 4) {
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int w = 0; w < wpb; ++w) {
      const float4 v = *reinterpret_cast<const float4*>(sm + (size_t)w * 3 * H + i);
      t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
    }
    red_add_f32x4(my_acc + i, t.x, t.y, t.z, t.w);
  }
  if (counter != nullptr) finalize_columns<T>(acc, counter, nvec, H, dgamma, dbeta, EMBED ? nullptr : dbias);
}

// LayerNorm backward of the blocks (EMBED = false above) for 16-bit activations and H <= 1024: the three column sums live in
// registers (24 NV per lane) instead of a shared-memory row per warp, so a row costs neither the read-modify-write of
// 12 H bytes of shared memory nor, per CTA, a pass over 12 H floats to clear and to flush them; one CTA of 8 warps per SM
// walks the rows with the next row's loads in flight, and its flush is one reduction over the warps and
// H / 4 x 3 vector reductions per SM.  Arithmetic in pairs (F2).  8192 x 768 padded rows took 34.9 us alone in the kernel
// above; 4900 packed rows take 9.5 us here.  Steps: 256 x 32 2.85 -> 2.77 ms, 64 x 256 7.31 -> 7.05 ms.
template <typename T, int NV>
__global__ void __launch_bounds__(256, 1) ln_bwd_reg_kernel(
    const T* __restrict__ dy, const T* __restrict__ pre, const T* __restrict__ gamma, const float* __restrict__ mean,
    const float* __restrict__ rstd, T* __restrict__ d_pre, T* __restrict__ d_branch, float* __restrict__ acc,
    unsigned* __restrict__ counter, T* __restrict__ dgamma, T* __restrict__ dbeta, T* __restrict__ dbias, int rows, int H,
    float p, const int* __restrict__ seed_ptr, uint32_t stream, const int* __restrict__ tok_meta, const int* __restrict__ tok) {
  grid_dep_wait();            // launched with launch_pdl: nothing above touches global memory
  grid_dep_launch();
  if (tok_meta != nullptr) rows = __ldcg(tok_meta + TOK_ROWS);
  extern __shared__ __align__(16) float sm[];      // [warps][3][H]
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const int total_warps = gridDim.x * wpb;
  const uint32_t seed = p > 0.f ? (uint32_t)(*seed_ptr) : 0u;
  const float inv_keep = p > 0.f ? 1.f / (1.f - p) : 1.f;
  const float inv_h = 1.f / H;
  Raw8<T> gam[NV], nd[NV], nx[NV];
  F2 dg[NV][4], db[NV][4], dr[NV][4];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = (lane + 32 * i) * 8;
    gam[i].v = make_uint4(0u, 0u, 0u, 0u);
    nd[i].v = nx[i].v = gam[i].v;
    if (col < H) gam[i] = load_raw8<T>(gamma + col);
#pragma unroll
    for (int j = 0; j < 4; ++j) dg[i][j] = db[i][j] = dr[i][j] = f2(0.f);
  }
  int row = blockIdx.x + gridDim.x * wib;          // neighbouring rows go to different SMs: a short tail is spread
  float mu = 0.f, rs = 0.f;
  int crow = 0;
  const auto fetch = [&](int r) {
    if (r >= rows) return;
    mu = mean[r];
    rs = rstd[r];
    crow = tok != nullptr && p > 0.f ? __ldcg(tok + r) : r;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (lane + 32 * i) * 8;
      if (col < H) {
        nd[i] = load_raw8<T>(dy + (size_t)r * H + col);
        nx[i] = load_raw8<T>(pre + (size_t)r * H + col);
      }
    }
  };
  fetch(row);
  for (; row < rows; row += total_warps) {
    Raw8<T> rd[NV], rx[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) { rd[i] = nd[i]; rx[i] = nx[i]; }
    const F2 nmu = f2(-mu), rs2 = f2(rs);
    const int drow = crow;
    fetch(row + total_warps);
    F2 s1 = f2(0.f), s2 = f2(0.f);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float d[8], x[8], gm[8];
      unpack8<T>(rd[i], d);
      unpack8<T>(rx[i], x);
      unpack8<T>(gam[i], gm);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const F2 d2 = f2(d[2 * j], d[2 * j + 1]);
        const F2 xh = (f2(x[2 * j], x[2 * j + 1]) + nmu) * rs2;
        const F2 g = d2 * f2(gm[2 * j], gm[2 * j + 1]);
        s1 = s1 + g;
        s2 = f2_fma(g, xh, s2);
        dg[i][j] = f2_fma(d2, xh, dg[i][j]);
        db[i][j] = db[i][j] + d2;
      }
    }
    float a0, a1, b0, b1;
    f2_get(s1, a0, a1);
    f2_get(s2, b0, b1);
    const F2 m1 = f2(-warp_sum(a0 + a1) * inv_h), m2 = f2(-warp_sum(b0 + b1) * inv_h);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (lane + 32 * i) * 8;
      if (col < H) {
        float d[8], x[8], gm[8], dx[8];
        unpack8<T>(rd[i], d);
        unpack8<T>(rx[i], x);
        unpack8<T>(gam[i], gm);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const F2 xh = (f2(x[2 * j], x[2 * j + 1]) + nmu) * rs2;
          const F2 g = f2_fma(f2(d[2 * j], d[2 * j + 1]), f2(gm[2 * j], gm[2 * j + 1]), m1);
          f2_get(f2_fma(xh, m2, g) * rs2, dx[2 * j], dx[2 * j + 1]);
        }
        Raw8<T> o;
        o.v = pack16x8<T>(dx);
        *reinterpret_cast<uint4*>(d_pre + (size_t)row * H + col) = o.v;
        if (p > 0.f) {
#pragma unroll
          for (int j = 0; j < 8; ++j) dx[j] = keep(seed, stream, (uint32_t)(drow * H + col + j), p) ? dx[j] * inv_keep : 0.f;
          o.v = pack16x8<T>(dx);
          *reinterpret_cast<uint4*>(d_branch + (size_t)row * H + col) = o.v;
        }
        unpack8<T>(o, dx);                         // the bias gradient sums the rounded values
#pragma unroll
        for (int j = 0; j < 4; ++j) dr[i][j] = dr[i][j] + f2(dx[2 * j], dx[2 * j + 1]);
      }
    }
  }
  float* mine = sm + (size_t)wib * 3 * H;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = (lane + 32 * i) * 8;
    if (col < H) {
#pragma unroll
      for (int v = 0; v < 3; ++v) {
        const F2* a = v == 0 ? dg[i] : (v == 1 ? db[i] : dr[i]);
        float o[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) f2_get(a[j], o[2 * j], o[2 * j + 1]);
        store8<float>(mine + v * H + col, o);
      }
    }
  }
  __syncthreads();
  float* my_acc = acc_replica(acc, 3, H);
  for (int i = threadIdx.x * 4; i < 3 * H; i += blockDim.x * 4) {
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int w = 0; w < wpb; ++w) {
      const float4 v = *reinterpret_cast<const float4*>(sm + (size_t)w * 3 * H + i);
      t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
    }
    red_add_f32x4(my_acc + i, t.x, t.y, t.z, t.w);
  }
  if (counter != nullptr) finalize_columns<T>(acc, counter, 3, H, dgamma, dbeta, dbias);
}

// ------------------------------------------------------------------------------------ GELU

// grid = (ceil(F/8/128), row_chunks): a thread owns 8 columns (its bias stays in registers) and walks rows
template <typename T>
__global__ void __launch_bounds__(128) bias_gelu_fwd_kernel(const T* __restrict__ x, const T* __restrict__ bias,
                                                            T* __restrict__ out, int rows, int F) {
  const int col = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (col >= F) return;
  float b[8];
  load8(bias + col, b);
  for (int r = blockIdx.y; r < rows; r += 4 * gridDim.y) {
    float a[4][8];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (r + u * gridDim.y < rows) load8(x + (size_t)(r + u * gridDim.y) * F + col, a[u]);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (r + u * gridDim.y < rows) {
#pragma unroll
        for (int j = 0; j < 8; j += 2) f2_get(gelu2(f2(a[u][j], a[u][j + 1]) + f2(b[j], b[j + 1])), a[u][j], a[u][j + 1]);
        store8(out + (size_t)(r + u * gridDim.y) * F + col, a[u]);
      }
  }
}

// grid = (ceil(F/8/128), row_chunks); a thread owns 8 columns and walks the rows of its chunk
template <typename T>
__global__ void __launch_bounds__(128) bias_gelu_bwd_kernel(const T* __restrict__ da, const T* __restrict__ x,
                                                            const T* __restrict__ bias, T* __restrict__ dx,
                                                            float* __restrict__ acc, unsigned* __restrict__ counter,
                                                            T* __restrict__ dbias, int rows, int F) {
  const int col = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (col < F) {
    float b[8];
    F2 s[4];
    load8(bias + col, b);
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] = f2(0.f);
    for (int r = blockIdx.y; r < rows; r += 2 * gridDim.y) {
      Raw8<T> a[2], g[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int rr = r + u * gridDim.y;
        if (rr < rows) { a[u] = load_raw8<T>(x + (size_t)rr * F + col); g[u] = load_raw8<T>(da + (size_t)rr * F + col); }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int rr = r + u * gridDim.y;
        if (rr < rows) {
          float z[8], o[8];
          unpack8<T>(a[u], z);
          unpack8<T>(g[u], o);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            f2_get(f2(o[2 * j], o[2 * j + 1]) * gelu_grad2(f2(z[2 * j], z[2 * j + 1]) + f2(b[2 * j], b[2 * j + 1])), o[2 * j], o[2 * j + 1]);
          store8(dx + (size_t)rr * F + col, o);
#pragma unroll
          for (int j = 0; j < 4; ++j) s[j] = s[j] + f2(round_through<T>(o[2 * j]), round_through<T>(o[2 * j + 1]));
        }
      }
    }
    float* my_acc = acc_replica(acc, 1, F);
    float t[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) f2_get(s[j], t[2 * j], t[2 * j + 1]);
    red_add_f32x4(my_acc + col, t[0], t[1], t[2], t[3]);
    red_add_f32x4(my_acc + col + 4, t[4], t[5], t[6], t[7]);
  }
  if (counter != nullptr) finalize_columns<T>(acc, counter, 1, F, dbias, nullptr, nullptr);
}

template <typename T>
__global__ void __launch_bounds__(128) colsum_kernel(const T* __restrict__ x, float* __restrict__ acc,
                                                     unsigned* __restrict__ counter, T* __restrict__ out,
                                                     int rows, int N) {
  const int col = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (col < N) {
    float s[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] = 0.f;
    for (int r = blockIdx.y; r < rows; r += 4 * gridDim.y) {
      float a[4][8];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (r + u * gridDim.y < rows) load8(x + (size_t)(r + u * gridDim.y) * N + col, a[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (r + u * gridDim.y < rows) {
#pragma unroll
          for (int j = 0; j < 8; ++j) s[j] += a[u][j];
        }
    }
    float* my_acc = acc_replica(acc, 1, N);
    red_add_f32x4(my_acc + col, s[0], s[1], s[2], s[3]);
    red_add_f32x4(my_acc + col + 4, s[4], s[5], s[6], s[7]);
  }
  if (counter != nullptr) finalize_columns<T>(acc, counter, 1, N, out, nullptr, nullptr);
}

// ------------------------------------------------------------------------------------ pooling
// grid = b.  The block's threads are `slices` sets of H/8 column vectors; for the mean each set walks every slices-th token
// (one set alone waited for 256 loads one after the other at S = 256: 72 us) and shared memory joins them.  Packed tokens:
// slot gives the row of a token (CLS and attended ones are kept).
constexpr int POOL_THREADS = 512;
template <typename T>
__global__ void __launch_bounds__(POOL_THREADS) pool_fwd_kernel(const T* __restrict__ h, const int* __restrict__ mask,
                                                                float* __restrict__ out, int S, int H, int cls,
                                                                const int* __restrict__ slot) {
  extern __shared__ __align__(16) float s_acc[];   // [slices][H]
  __shared__ int s_cnt;
  const int b = blockIdx.x, nv = H / 8;
  if (cls) {
    for (int col = threadIdx.x * 8; col < H; col += blockDim.x * 8) {
      float acc[8];
      load8(h + (size_t)(slot != nullptr ? slot[b * S] : b * S) * H + col, acc);
      store8(out + (size_t)b * H + col, acc);
    }
    return;
  }
  const int slices = max(1, (int)blockDim.x / nv);
  if (threadIdx.x == 0) s_cnt = 0;
  __syncthreads();
  int n = 0;
  for (int s = threadIdx.x; s < S; s += blockDim.x) n += mask[b * S + s] != 0 ? 1 : 0;
  if (n > 0) atomicAdd(&s_cnt, n);
  __syncthreads();
  const float inv = 1.f / fmaxf((float)s_cnt, 1e-9f);
  const int slice = nv <= (int)blockDim.x ? (int)threadIdx.x / nv : 0;
  for (int v = nv <= (int)blockDim.x ? (int)threadIdx.x % nv : (int)threadIdx.x; v < nv && slice < slices; v += blockDim.x) {
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
#pragma unroll 4
    for (int s = slice; s < S; s += slices) {
      if (mask[b * S + s] != 0) {
        float a[8];
        load8(h + (size_t)(slot != nullptr ? slot[b * S + s] : b * S + s) * H + v * 8, a);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += a[j];
      }
    }
    if (slices == 1) {
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] *= inv;
      store8(out + (size_t)b * H + v * 8, acc);
    } else {
      store8(s_acc + (size_t)slice * H + v * 8, acc);
    }
  }
  if (slices == 1) return;
  __syncthreads();
  for (int c = threadIdx.x; c < H; c += blockDim.x) {
    float t = 0.f;
    for (int q = 0; q < slices; ++q) t += s_acc[(size_t)q * H + c];
    out[(size_t)b * H + c] = t * inv;
  }
}

// grid = b*S rows.  Packed tokens: rows past the packed ones do nothing, the zero rows (tok < 0) get zeros.
template <typename T>
__global__ void pool_bwd_kernel(const float* __restrict__ de, const int* __restrict__ mask, T* __restrict__ dh,
                                int S, int H, int cls, const int* __restrict__ tok_meta, const int* __restrict__ tok,
                                const int* __restrict__ tok_cnt) {
  const int row = blockIdx.x;
  if (tok_meta != nullptr && row >= tok_meta[TOK_ROWS]) return;
  const int src = tok_meta != nullptr ? tok[row] : row;
  const int b = src < 0 ? 0 : src / S, s = src - b * S;
  float w;
  if (src < 0) {
    w = 0.f;
  } else if (cls) {
    w = (s == 0) ? 1.f : 0.f;
  } else {
    float cnt = 0.f;
    if (tok_cnt != nullptr) cnt = (float)tok_cnt[b];
    else
      for (int t = 0; t < S; ++t) cnt += mask[b * S + t] != 0 ? 1.f : 0.f;
    w = mask[src] != 0 ? 1.f / fmaxf(cnt, 1e-9f) : 0.f;
  }
  for (int col = threadIdx.x * 8; col < H; col += blockDim.x * 8) {
    float a[8];
    load8(de + (size_t)b * H + col, a);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = w == 0.f ? 0.f : a[j] * w;
    store8(dh + (size_t)row * H + col, a);
  }
}

// ------------------------------------------------------------------------------------ dropout on [n] elements
template <typename TI, typename TO>
__global__ void dropout_kernel(const TI* __restrict__ x, TO* __restrict__ out, size_t n, float p,
                               const int* __restrict__ seed_ptr, uint32_t stream) {
  const uint32_t seed = p > 0.f ? (uint32_t)(*seed_ptr) : 0u;
  const float inv_keep = p > 0.f ? 1.f / (1.f - p) : 1.f;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    float v = to_f(x[i]);
    if (p > 0.f) v = keep(seed, stream, (uint32_t)i, p) ? v * inv_keep : 0.f;
    out[i] = from_f<TO>(v);
  }
}

}  // namespace rb

using namespace rb;

#define DISPATCH_T(dtype, ...)                                                     \
  switch (dtype) {                                                                 \
    case RB_F32: { using T = float; __VA_ARGS__; break; }                          \
    case RB_BF16: { using T = __nv_bfloat16; __VA_ARGS__; break; }                 \
    case RB_F16: { using T = __half; __VA_ARGS__; break; }                         \
    default: return -1;                                                            \
  }

#define DISPATCH_NV(H, ...)                                                        \
  {                                                                                \
    const int nv_ = ((H) + 255) / 256;                                             \
    if (nv_ <= 1) { constexpr int NV = 1; __VA_ARGS__; }                           \
    else if (nv_ <= 2) { constexpr int NV = 2; __VA_ARGS__; }                      \
    else if (nv_ <= 3) { constexpr int NV = 3; __VA_ARGS__; }                      \
    else if (nv_ <= 4) { constexpr int NV = 4; __VA_ARGS__; }                      \
    else if (nv_ <= 8) { constexpr int NV = 8; __VA_ARGS__; }                      \
    else return -2;                                                                \
  }

RB_API int rb_bias_dropout_add_ln_fwd(int dtype, const void* x, const void* bias, const void* resid, const void* gamma,
                                      const void* beta, void* y, void* pre, float* mean, float* rstd, int rows, int H,
                                      float eps, float p, const int* seed, unsigned stream_id, cudaStream_t st) {
  if (H % 8) return -3;
  const int blocks = (rows + 3) / 4;
  DISPATCH_T(dtype, DISPATCH_NV(H, (bias_dropout_add_ln_fwd_kernel<T, NV><<<blocks, 128, 0, st>>>(
      (const T*)x, (const T*)bias, (const T*)resid, (const T*)gamma, (const T*)beta, (T*)y, (T*)pre, mean, rstd,
      rows, H, eps, p, seed, stream_id))));
  RB_LAUNCH_CHECK();
  return 0;
}

RB_API int rb_embed_ln_fwd(int dtype, const int* ids, const void* word, const void* pos, const void* gamma,
                           const void* beta, void* y, float* mean, float* rstd, int rows, int H, int S, float eps,
                           float p, const int* seed, unsigned stream_id, const int* mask, const int* tok_meta,
                           const int* tok_off, const int* tok_cnt, int* tok, int* tok_slot, cudaStream_t st) {
  if (H % 8) return -3;
  const int blocks = (rows + (tok_meta != nullptr ? TOK_ALIGN : 0) + 3) / 4;
  DISPATCH_T(dtype, DISPATCH_NV(H, (embed_ln_fwd_kernel<T, NV><<<blocks, 128, 0, st>>>(
      ids, (const T*)word, (const T*)pos, (const T*)gamma, (const T*)beta, (T*)y, mean, rstd, rows, H, S, eps, p,
      seed, stream_id, mask, tok_meta, tok_off, tok_cnt, tok, tok_slot))));
  RB_LAUNCH_CHECK();
  return 0;
}

// Counts, lengths and packed offsets of the B sequences of a [B, S] mask (token_map.cuh); tok and slot are filled by
// rb_embed_ln_fwd.  meta's counter word must be 0 on entry and is left 0.
RB_API int rb_token_map(const int* mask, int B, int S, int* off, int* len, int* cnt, int* meta, cudaStream_t st) {
  if (B < 1 || S < 1 || (long long)B * S > (1LL << 30)) return -3;
  int G = 1;
  while (G < 32 && G < S) G <<= 1;
  int blocks = (B + 32 * (32 / G) - 1) / (32 * (32 / G));
  if (blocks > sm_count()) blocks = sm_count();
  token_map_kernel<<<blocks, 1024, 0, st>>>(mask, B, S, G, off, len, cnt, meta);
  RB_LAUNCH_CHECK();
  return 0;
}

static int ln_bwd_blocks(int rows, int S, bool embed, int warps = 4) {
  int blocks = (rows + warps - 1) / warps;
  const int per_sm = warps == 4 ? 5 : (warps == 8 ? 2 : 1);
  if (blocks > sm_count() * per_sm) blocks = sm_count() * per_sm;
  if (embed) {  // total warps (4 per block) must be a multiple of S: round blocks to a multiple of S
    blocks = (blocks / S) * S;
    if (blocks == 0) blocks = S;
  }
  return blocks;
}

// Warps per CTA of the general LayerNorm backward kernel (fp32, or H > 1024).  Every CTA ends with a flush of its 3 H column sums into the fp32
// replicas (L2 reductions); fewer, larger CTAs flush less often per row.
static int g_ln_bwd_warps = 4;
RB_API void rb_set_ln_bwd_warps(int w) { g_ln_bwd_warps = (w == 8 || w == 16) ? w : 4; }

template <int WARPS>
static int launch_ln_bwd(int dtype, const void* dy, const void* pre, const void* gamma, const float* mean,
                         const float* rstd, void* d_pre, void* d_branch, float* acc, unsigned* counter, void* dgamma,
                         void* dbeta, void* dbias, int rows, int H, float p, const int* seed, unsigned stream_id,
                         const int* tok_meta, const int* tok, cudaStream_t st) {
  const int blocks = ln_bwd_blocks(rows, 1, false, WARPS);
  const size_t smem = (size_t)WARPS * 3 * (size_t)H * sizeof(float);
  DISPATCH_T(dtype, DISPATCH_NV(H, (cudaFuncSetAttribute(ln_bwd_kernel<T, NV, false, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                                    launch_pdl(ln_bwd_kernel<T, NV, false, WARPS>, dim3(blocks), dim3(WARPS * 32), smem, st,
      (const T*)dy, (const T*)pre, (const int*)nullptr, (const T*)nullptr, (const T*)nullptr, (const T*)gamma, mean, rstd,
      (T*)d_pre, (T*)d_branch, (T*)nullptr, (T*)nullptr, acc, counter, (T*)dgamma, (T*)dbeta, (T*)dbias, rows, H, 1, 0, p,
      seed, stream_id, tok_meta, tok))));
  RB_LAUNCH_CHECK();
  return 0;
}

template <typename T, int NV>
static int launch_ln_bwd_reg(const void* dy, const void* pre, const void* gamma, const float* mean, const float* rstd, void* d_pre,
                             void* d_branch, float* acc, unsigned* counter, void* dgamma, void* dbeta, void* dbias, int rows,
                             int H, float p, const int* seed, unsigned stream_id, const int* tok_meta, const int* tok,
                             cudaStream_t st) {
  constexpr int warps = 8;
  const int want = (rows + warps - 1) / warps;
  const int blocks = want < sm_count() ? want : sm_count();
  const size_t smem = (size_t)warps * 3 * H * sizeof(float);
  if (cudaFuncSetAttribute(ln_bwd_reg_kernel<T, NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -5;
  launch_pdl(ln_bwd_reg_kernel<T, NV>, dim3(blocks), dim3(warps * 32), smem, st, (const T*)dy, (const T*)pre, (const T*)gamma,
             mean, rstd, (T*)d_pre, (T*)d_branch, acc, counter, (T*)dgamma, (T*)dbeta, (T*)dbias, rows, H, p, seed, stream_id,
             tok_meta, tok);
  return 0;
}

RB_API int rb_bias_dropout_add_ln_bwd(int dtype, const void* dy, const void* pre, const void* gamma, const float* mean,
                                      const float* rstd, void* d_pre, void* d_branch, float* acc, unsigned* counter,
                                      void* dgamma, void* dbeta, void* dbias, int rows, int H, float p, const int* seed,
                                      unsigned stream_id, const int* tok_meta, const int* tok, cudaStream_t st) {
  if (H % 8) return -3;
  if (dtype != RB_F32 && H <= 1024) {
#define RB_LN_REG(T, NV) launch_ln_bwd_reg<T, NV>(dy, pre, gamma, mean, rstd, d_pre, d_branch, acc, counter, dgamma, dbeta, dbias, rows, H, p, seed, stream_id, tok_meta, tok, st)
    const int nv = (H + 255) / 256;
    int rc = -1;
    if (dtype == RB_BF16) rc = nv <= 1 ? RB_LN_REG(__nv_bfloat16, 1) : nv == 2 ? RB_LN_REG(__nv_bfloat16, 2) : nv == 3 ? RB_LN_REG(__nv_bfloat16, 3) : RB_LN_REG(__nv_bfloat16, 4);
    else if (dtype == RB_F16) rc = nv <= 1 ? RB_LN_REG(__half, 1) : nv == 2 ? RB_LN_REG(__half, 2) : nv == 3 ? RB_LN_REG(__half, 3) : RB_LN_REG(__half, 4);
#undef RB_LN_REG
    if (rc) return rc;
    RB_LAUNCH_CHECK();
    return 0;
  }
  int w = g_ln_bwd_warps;
  while (w > 4 && (size_t)w * 3 * H * sizeof(float) > 200 * 1024) w >>= 1;     // the per-warp column sums must fit
  if (w == 16) return launch_ln_bwd<16>(dtype, dy, pre, gamma, mean, rstd, d_pre, d_branch, acc, counter, dgamma, dbeta, dbias, rows, H, p, seed, stream_id, tok_meta, tok, st);
  if (w == 8) return launch_ln_bwd<8>(dtype, dy, pre, gamma, mean, rstd, d_pre, d_branch, acc, counter, dgamma, dbeta, dbias, rows, H, p, seed, stream_id, tok_meta, tok, st);
  return launch_ln_bwd<4>(dtype, dy, pre, gamma, mean, rstd, d_pre, d_branch, acc, counter, dgamma, dbeta, dbias, rows, H, p, seed, stream_id, tok_meta, tok, st);
}

RB_API int rb_embed_ln_bwd(int dtype, const void* dy, const int* ids, const void* word, const void* pos,
                           const void* gamma, const float* mean, const float* rstd, void* dword, void* dpos,
                           float* acc, unsigned* counter, void* dgamma, void* dbeta, int rows, int H, int S, int pad_id,
                           float p, const int* seed, unsigned stream_id, const int* tok_slot, cudaStream_t st) {
  if (H % 8) return -3;
  const int blocks = ln_bwd_blocks(rows, S, true);
  const size_t smem = 4 * 3 * (size_t)H * sizeof(float);
  DISPATCH_T(dtype, DISPATCH_NV(H, (cudaFuncSetAttribute(ln_bwd_kernel<T, NV, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                                    launch_pdl(ln_bwd_kernel<T, NV, true>, dim3(blocks), dim3(128), smem, st,
      (const T*)dy, (const T*)nullptr, ids, (const T*)word, (const T*)pos, (const T*)gamma, mean, rstd, (T*)nullptr,
      (T*)nullptr, (T*)dword, (T*)dpos, acc, counter, (T*)dgamma, (T*)dbeta, (T*)nullptr, rows, H, S, pad_id, p, seed,
      stream_id, (const int*)nullptr, tok_slot))));
  RB_LAUNCH_CHECK();
  return 0;
}

RB_API int rb_bias_gelu_fwd(int dtype, const void* x, const void* bias, void* out, int rows, int F, cudaStream_t st) {
  if (F % 8) return -3;
  const int cb = (F / 8 + 127) / 128;
  int rc = sm_count() * 8 / cb;   // 8 CTAs per SM measured best (5, 10: 15 % slower)
  if (rc > (rows + 3) / 4) rc = (rows + 3) / 4;
  if (rc < 1) rc = 1;
  dim3 grid(cb, rc);
  DISPATCH_T(dtype, (bias_gelu_fwd_kernel<T><<<grid, 128, 0, st>>>((const T*)x, (const T*)bias, (T*)out, rows, F)));
  RB_LAUNCH_CHECK();
  return 0;
}

RB_API int rb_bias_gelu_bwd(int dtype, const void* da, const void* x, const void* bias, void* dx, float* acc,
                            unsigned* counter, void* dbias, int rows, int F, cudaStream_t st) {
  if (F % 8) return -3;
  const int cb = (F / 8 + 127) / 128;
  int rc = sm_count() * 8 / cb;
  if (rc > (rows + 3) / 4) rc = (rows + 3) / 4;
  if (rc < 1) rc = 1;
  dim3 grid(cb, rc);
  DISPATCH_T(dtype, (bias_gelu_bwd_kernel<T><<<grid, 128, 0, st>>>((const T*)da, (const T*)x, (const T*)bias, (T*)dx,
                                                                    acc, counter, (T*)dbias, rows, F)));
  RB_LAUNCH_CHECK();
  return 0;
}

RB_API int rb_colsum(int dtype, const void* x, float* acc, unsigned* counter, void* out, int rows, int N,
                     cudaStream_t st) {
  if (N % 8) return -3;
  const int cb = (N / 8 + 127) / 128;
  int rc = sm_count() * 5 / cb;
  if (rc > (rows + 3) / 4) rc = (rows + 3) / 4;
  if (rc < 1) rc = 1;
  dim3 grid(cb, rc);
  DISPATCH_T(dtype, (colsum_kernel<T><<<grid, 128, 0, st>>>((const T*)x, acc, counter, (T*)out, rows, N)));
  RB_LAUNCH_CHECK();
  return 0;
}

RB_API int rb_pool_fwd(int dtype, const void* h, const int* mask, float* out, int b, int S, int H, int cls,
                       const int* tok_slot, cudaStream_t st) {
  if (H % 8) return -3;
  const int nv = H / 8, slices = nv < POOL_THREADS ? POOL_THREADS / nv : 1;
  const size_t smem = cls || slices == 1 ? 0 : (size_t)slices * H * sizeof(float);     // at most 16 KB
  DISPATCH_T(dtype, (pool_fwd_kernel<T><<<b, POOL_THREADS, smem, st>>>((const T*)h, mask, out, S, H, cls, tok_slot)));
  RB_LAUNCH_CHECK();
  return 0;
}

RB_API int rb_pool_bwd(int dtype, const float* de, const int* mask, void* dh, int b, int S, int H, int cls,
                       const int* tok_meta, const int* tok, const int* tok_cnt, cudaStream_t st) {
  if (H % 8) return -3;
  DISPATCH_T(dtype, (pool_bwd_kernel<T><<<b * S, 128, 0, st>>>(de, mask, (T*)dh, S, H, cls, tok_meta, tok, tok_cnt)));
  RB_LAUNCH_CHECK();
  return 0;
}

// fp32 in → out dtype (fp32 / fp16 / bf16): classifier-input dropout + cast
RB_API int rb_dropout_cast_fwd(int out_dtype, const float* x, void* out, long long n, float p, const int* seed,
                               unsigned stream_id, cudaStream_t st) {
  int blocks = (int)((n + 255) / 256);
  if (blocks > sm_count() * 8) blocks = sm_count() * 8;
  DISPATCH_T(out_dtype, (dropout_kernel<float, T><<<blocks, 256, 0, st>>>(x, (T*)out, (size_t)n, p, seed, stream_id)));
  RB_LAUNCH_CHECK();
  return 0;
}

// ------------------------------------------------------------------------------------ allocation-free column sum
// rb_colsum_noalloc: the column sum above for callers that must not allocate device memory (declared
// and documented in renee_b200_noalloc.h).  Its fp32 accumulator replicas and its block counter live in
// the two file-scope device arrays below instead of in a caller-provided workspace.  In host code these
// names are only host-side handles of the symbols, so their device addresses are looked up once per
// device with cudaGetSymbolAddress and those addresses are what the kernel receives.
constexpr int kNoAllocMaxCols = 8192;
static __device__ __align__(256) float g_colsum_scratch[rb::kCopies * kNoAllocMaxCols];
static __device__ __align__(256) unsigned g_colsum_counter[64];

namespace {
struct NoAllocSlot { bool ready; float* scratch; unsigned* counter; };
NoAllocSlot g_noalloc_slots[64];
}  // namespace

RB_API int rb_colsum_noalloc_max_cols(void) { return kNoAllocMaxCols; }

RB_API int rb_colsum_noalloc(int dtype, const void* x, void* out, int rows, int N, cudaStream_t st) {
  if (dtype != RB_F32 && dtype != RB_BF16 && dtype != RB_F16) {
    fprintf(stderr, "rb_colsum_noalloc: unknown dtype code %d (0 = fp32, 1 = bf16, 2 = fp16)\n", dtype);
    return -1;     // checked before anything is queued on the stream
  }
  if (rows < 1 || N < 8 || N % 8) {
    fprintf(stderr, "rb_colsum_noalloc: rows must be >= 1 and N a positive multiple of 8 (got rows=%d, N=%d)\n", rows, N);
    return -3;
  }
  if (N > kNoAllocMaxCols) {
    fprintf(stderr, "rb_colsum_noalloc: N=%d exceeds the built-in scratch (at most %d columns)\n", N, kNoAllocMaxCols);
    return -10;
  }
  int device = -1;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return -11;
  NoAllocSlot& slot = g_noalloc_slots[device];
  if (!slot.ready) {
    // first call on this device (keep it outside any stream capture): resolve the device addresses
    void* s = nullptr;
    void* c = nullptr;
    if (cudaGetSymbolAddress(&s, g_colsum_scratch) != cudaSuccess) return -12;
    if (cudaGetSymbolAddress(&c, g_colsum_counter) != cudaSuccess) return -12;
    slot.scratch = static_cast<float*>(s);
    slot.counter = static_cast<unsigned*>(c);
    slot.ready = true;
  }
  // the arrays keep whatever the previous call (or an interrupted one) left: start from zero
  if (cudaMemsetAsync(slot.scratch, 0, sizeof(float) * rb::kCopies * (size_t)N, st) != cudaSuccess) return -13;
  if (cudaMemsetAsync(slot.counter, 0, sizeof(unsigned), st) != cudaSuccess) return -13;
  const int cb = (N / 8 + 127) / 128;
  int rc = sm_count() * 5 / cb;
  if (rc > (rows + 3) / 4) rc = (rows + 3) / 4;
  if (rc < 1) rc = 1;
  dim3 grid(cb, rc);
  DISPATCH_T(dtype, (colsum_kernel<T><<<grid, 128, 0, st>>>((const T*)x, slot.scratch, slot.counter, (T*)out, rows, N)));
  RB_LAUNCH_CHECK();
  return 0;
}


RB_API int rb_finalize_columns(int dtype, const void* jobs, int n_jobs, int max_len, cudaStream_t st) {
  if (n_jobs < 1) return 0;
  dim3 grid(n_jobs, (max_len + 255) / 256);
  DISPATCH_T(dtype, (finalize_jobs_kernel<T><<<grid, 256, 0, st>>>((const ColumnJob*)jobs)));
  RB_LAUNCH_CHECK();
  return 0;
}
