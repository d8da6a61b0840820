// Register-resident self-attention forward/backward for 16-bit activations, head dim 64 (S <= 512) or 32 (S <= 128):
// one CTA per (batch, head) up to 256 tokens, with score rows in registers up to 64 (forward: 128) and key blocks beyond;
// streaming kernels, further down, for 257..512.
// Same fusion and interface as attention_tc.cu (bias add, scale, key-padding mask, softmax, counter-based
// attention dropout, head split/merge addressing, q/k/v bias gradients), organised so that the score
// matrix never touches shared memory:
//   * one CTA per (batch, head); the padded sequence SP is 16 to 64 (forward: to 128) and the CTA has SP/16 warps;
//   * a warp owns 16 query rows.  S = Q K^T (forward) or dP = dO V^T (backward) for those rows is
//     accumulated in registers by m16n8k16 MMAs fed with ldmatrix, the softmax / softmax-gradient runs on
//     the accumulator fragments (a row lives in one quad: two shuffles per reduction), and the fragments
//     are re-packed in place as the A operand of the next product (O = P~ V, dQ = dS K);
//   * only dK = dS^T Q and dV = P~^T dO need other warps' rows: dS and P~ go through shared memory once
//     and each warp then owns 16 key rows.
// Shared memory per CTA: 3 (forward) or 4 (backward) [SP][72] operand tiles, plus two [SP][SP+8] tiles in
// the backward: 14 KB / 24 KB at SP = 32, so many CTAs share an SM at short sequences; 28 KB / 56 KB at SP = 64, 55 KB in the
// forward at SP = 128.  At S = 32 a head is a quarter of the 128-row tcgen05 tile, so the warp-level MMA is the
// shape that fits this op; the classifier GEMMs, where the FLOPs are, use tcgen05.
// First-token variant (template parameter CLS): where only the first token of a sequence is read behind a layer (CLS pooling
// behind the last one), it is the only query.  Its row goes through the same fragments and the same sums as above -- the other
// 15 rows of its tile are dropped or zero -- so it comes out bit for bit; ctx and dctx then have one row per sequence, the
// forward also copies the first token's layer input there (the residual of the output projection), and the backward spreads
// the gradient of that residual over the packed rows (zeros behind the first), where the next GEMM adds it.
// Reference behaviour: the attention of the HF DistilBERT layers that main.py:225-262 wraps.
#include <type_traits>
#include "common.cuh"
#include "token_map.cuh"

namespace rb {
namespace amma {

constexpr int HD = 64;
constexpr int RP = HD + 8;   // operand row pitch (elements): 144 B keeps the 8 rows of an ldmatrix on distinct banks

// Where the tokens of a sequence live: packed rows (token_map.cuh) or, with slot == nullptr, the padded [b, S] layout.
// Dropped tokens are masked keys that no kept query can see and queries nobody reads: they are neither loaded nor
// written, and tiles of 8 keys or 16 queries behind a sequence's last kept token are skipped.
struct Tok {
  const int* slot;   // [b * S] row of a token or -1
  const int* len;    // [b] last kept position + 1
  const int* meta;   // row counts
};
// First-token variant: forward src = layer input, packed rows of H columns, dst = its first tokens [b, H]; backward src = [b, H]
// gradient of the residual, dst = packed rows.
template <typename T> struct FirstTok { const T* src; T* dst; };
__device__ __forceinline__ int seq_len(const Tok& tk, int b, int S) { return tk.slot != nullptr ? __ldcg(tk.len + b) : S; }
__device__ __forceinline__ int seq_row(const Tok& tk, int b, int S, int s) {
  return tk.slot != nullptr ? __ldcg(tk.slot + (size_t)b * S + s) : b * S + s;
}
// The zero rows behind the last packed token (rows of no sequence): columns [c0, c0 + HD) of each, by the CTAs of the
// last sequence.
template <typename T>
__device__ __forceinline__ void clear_zero_rows(const Tok& tk, T* out, int ld, int c0, int width) {
  const int lo = __ldcg(tk.meta + TOK_VALID), hi = __ldcg(tk.meta + TOK_ROWS);
  const int per = width / 8;
  for (int i = threadIdx.x; i < (hi - lo) * per; i += blockDim.x)
    *reinterpret_cast<uint4*>(out + (size_t)(lo + i / per) * ld + c0 + (i % per) * 8) = make_uint4(0u, 0u, 0u, 0u);
}

template <typename T> struct Pack;
template <> struct Pack<__nv_bfloat16> {
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t u) {
    return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u));
  }
};
template <> struct Pack<__half> {
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t u) {
    return __half22float2(*reinterpret_cast<__half2*>(&u));
  }
};

template <typename T>
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  } else {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
}

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const void* smem_row) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem_row);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], const void* smem_row) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem_row);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

__device__ __forceinline__ float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v;
}
__device__ __forceinline__ float quad_max(float v) {
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
  return v;
}

// acc[j] (j = 8-wide tile of columns) += A(16 rows r0.. of `a`, all HD columns) * B^T, B = SP rows of `bsm`:
// the shape of Q K^T and of dO V^T.  Both operands are [row][RP] tiles; only the first `lim` rows of B exist (in all
// of these routines lim is a multiple of 16 and the same in every lane).
template <typename T, int SP, int HD = amma::HD>
__device__ __forceinline__ void rows_times_transposed(float (&acc)[SP / 8][4], const T* a, const T* bsm, int r0, int lane, int lim) {
  constexpr int RP = HD + 8;
  uint32_t af[HD / 16][4];
#pragma unroll
  for (int kk = 0; kk < HD / 16; ++kk)
    ldsm4(af[kk], a + (r0 + (lane & 7) + ((lane >> 3) & 1) * 8) * RP + kk * 16 + (lane >> 4) * 8);
#pragma unroll
  for (int j = 0; j < SP / 8; ++j) {
    if (8 * j >= lim) continue;
#pragma unroll
    for (int kk = 0; kk < HD / 16; kk += 2) {
      uint32_t bf[4];   // {b0, b1} of k-step kk, {b0, b1} of k-step kk + 1
      ldsm4(bf, bsm + (8 * j + (lane & 7)) * RP + kk * 16 + (lane >> 3) * 8);
      mma16816<T>(acc[j], af[kk], bf[0], bf[1]);
      mma16816<T>(acc[j], af[kk + 1], bf[2], bf[3]);
    }
  }
}

// out[jd] (jd = 8-wide tile of the HD columns) += A * B for a 16 x SP A held as packed fragments
// (afr[kq] = the 16 x 16 block of columns 16 kq..) and B = the SP rows of the [row][RP] tile `bsm`.
template <typename T, int SP, int HD = amma::HD>
__device__ __forceinline__ void frag_times_rows(float (&out)[HD / 8][4], const uint32_t (&afr)[SP / 16][4], const T* bsm, int lane, int lim) {
  constexpr int RP = HD + 8;
#pragma unroll
  for (int kq = 0; kq < SP / 16; ++kq) {
    if (16 * kq >= lim) continue;
#pragma unroll
    for (int jd = 0; jd < HD / 8; jd += 2) {
      uint32_t bf[4];   // {b0, b1} of column tile jd, {b0, b1} of column tile jd + 1
      ldsm4_t(bf, bsm + (16 * kq + (lane & 7) + ((lane >> 3) & 1) * 8) * RP + 8 * jd + (lane >> 4) * 8);
      mma16816<T>(out[jd], afr[kq], bf[0], bf[1]);
      mma16816<T>(out[jd + 1], afr[kq], bf[2], bf[3]);
    }
  }
}

// out[jd] += A^T * B where A is the [SP][PP] tile `asm_` (rows = reduction index) restricted to its 16 columns
// c0.., and B = the SP rows of the [row][RP] tile `bsm` (its first 8 NJ columns): the shape of dS^T Q and of P~^T dO.
template <typename T, int SP, int HD = amma::HD, int NJ = HD / 8>
__device__ __forceinline__ void transposed_times_rows(float (&out)[NJ][4], const T* asm_, int PP, int c0, const T* bsm, int lane, int lim) {
  constexpr int RP = HD + 8;
#pragma unroll
  for (int kq = 0; kq < SP / 16; ++kq) {
    if (16 * kq >= lim) continue;
    uint32_t af[4];
    const int mi = lane >> 3;
    ldsm4_t(af, asm_ + (16 * kq + (lane & 7) + (mi >> 1) * 8) * PP + c0 + (mi & 1) * 8);
#pragma unroll
    for (int jd = 0; jd < NJ; jd += 2) {
      uint32_t bf[4];
      ldsm4_t(bf, bsm + (16 * kq + (lane & 7) + ((lane >> 3) & 1) * 8) * RP + 8 * jd + (lane >> 4) * 8);
      mma16816<T>(out[jd], af, bf[0], bf[1]);
      mma16816<T>(out[jd + 1], af, bf[2], bf[3]);
    }
  }
}

// Writes the warp's 16 x 8 NJ accumulator tile to the global rows row_lo / row_hi (this lane's two rows; negative: none)
// of stride ld and,
// when col_sums != nullptr, adds the column sums of the rounded values to col_sums[0..8 NJ) in shared memory.
template <typename T, int NJ>
__device__ __forceinline__ void write_rows(const float (&out)[NJ][4], T* dst, int ld, int row_lo, int row_hi, int lane,
                                           float* col_sums) {
  const int t = lane & 3;
  const bool v0 = row_lo >= 0, v1 = row_hi >= 0;
  float cs[2 * NJ];                                // this lane's columns 8 jd + 2 t + e over its two rows
#pragma unroll
  for (int jd = 0; jd < NJ; ++jd) {
    const uint32_t lo = Pack<T>::pack(out[jd][0], out[jd][1]);
    const uint32_t hi = Pack<T>::pack(out[jd][2], out[jd][3]);
    if (v0) *reinterpret_cast<uint32_t*>(dst + (size_t)row_lo * ld + 8 * jd + 2 * t) = lo;
    if (v1) *reinterpret_cast<uint32_t*>(dst + (size_t)row_hi * ld + 8 * jd + 2 * t) = hi;
    const float2 a = Pack<T>::unpack(lo), b = Pack<T>::unpack(hi);
    cs[2 * jd] = (v0 ? a.x : 0.f) + (v1 ? b.x : 0.f);
    cs[2 * jd + 1] = (v0 ? a.y : 0.f) + (v1 ? b.y : 0.f);
  }
  if (col_sums == nullptr) return;
  // over the eight lanes of equal t: each step hands half of the columns to the partner lane, 14 shuffles and 2 shared-memory
  // additions per lane at NJ = 8 instead of 48 and 16
  int at = 0;
#pragma unroll
  for (int o = 16, n = NJ; o >= 4; o >>= 1, n >>= 1) {
    const bool upper = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float send = upper ? cs[i] : cs[i + n], mine = upper ? cs[i + n] : cs[i];
      cs[i] = mine + __shfl_xor_sync(0xffffffffu, send, o);
    }
    at += upper ? n : 0;
  }
#pragma unroll
  for (int i = 0; i < NJ / 4; ++i) atomicAdd(col_sums + 8 * ((at + i) >> 1) + 2 * t + ((at + i) & 1), cs[i]);
}

// Elements idx, idx + 1 of a [.., S] row as one packed word, ok0 / ok1 saying which exist (0 for the others); `pair` =
// 4-byte access allowed.  Issued well before the use: the backward kernels spent most of their time waiting for the stored
// probabilities one tile after another.
template <typename T>
__device__ __forceinline__ uint32_t load_pair_raw(const T* __restrict__ base, size_t idx, bool ok0, bool ok1, bool pair) {
  uint32_t r = 0u;
  if (ok0) {
    if (pair) r = *reinterpret_cast<const uint32_t*>(base + idx);
    else {
      r = *reinterpret_cast<const uint16_t*>(base + idx);
      if (ok1) r |= (uint32_t)*reinterpret_cast<const uint16_t*>(base + idx + 1) << 16;
    }
  }
  return r;
}

// Sums of 8 pairs, two per instruction, rounded once
template <typename T> __device__ __forceinline__ uint4 add16x8(const uint4& a, const uint4& b) {
  using T2 = typename std::conditional<std::is_same<T, __half>::value, __half2, __nv_bfloat162>::type;
  uint4 r;
  const T2 *x = reinterpret_cast<const T2*>(&a), *y = reinterpret_cast<const T2*>(&b);
  T2* o = reinterpret_cast<T2*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) o[i] = __hadd2(x[i], y[i]);
  return r;
}

// Stages (q + bq, k + bk, v + bv [, dO]) of one (batch, head) as [SP][RP] tiles; rows of tokens that do not
// exist are zero, rows >= lim are left alone.
// The CTA has SP * 2 threads and the tiles SP * HD / 8 segments of 8 columns, so a thread owns the same 8 columns of
// HD / 16 rows: all of its global loads are issued before the first one is used.
// CLS: dO has one row per sequence (that of token 0), and only the first 16 queries are staged.
// The rows of a thread's tokens come from stage_rows.  Up to 32 tokens its loads go out together with that of the sequence's
// length: one after the other these two and the loads that hang on them were three round trips before the first product
// (256 x 32 packed, forward / backward with what follows: 15.3 / 40.1 -> 12.7 / 24.8 us).  Longer tiles have the length first,
// which leaves out the rows behind it.  The bias is added two values per instruction, rounded once as before; the longer
// forward tiles are the exception, where that came out slower (128 x 128: 66.9 us against 63.0).
template <int SP, int HD>
__device__ __forceinline__ void stage_rows(int (&row)[HD / 16], const Tok& tk, int b, int S, int n) {
  constexpr int SEGS = HD / 8, ROWS_PER_PASS = SP * 2 / SEGS;
#pragma unroll
  for (int it = 0; it < HD / 16; ++it) {
    const int s = (int)threadIdx.x / SEGS + it * ROWS_PER_PASS;
    row[it] = s < n ? seq_row(tk, b, S, s) : -1;           // of a packed token behind the last kept one: -1 too
  }
}
template <typename T, int SP, int HD, bool WITH_DO, bool CLS = false>
__device__ __forceinline__ void stage_operands(const T* __restrict__ qkv, const T* __restrict__ bqkv, const T* __restrict__ dctx,
                                               T* sQ, T* sK, T* sV, T* sDO, const int (&row)[HD / 16], int b, int h, int H,
                                               int lim) {
  constexpr int RP = HD + 8, SEGS = HD / 8, ROWS_PER_PASS = SP * 2 / SEGS, NIT = HD / 16;
  const int d = (threadIdx.x % SEGS) * 8, s0 = threadIdx.x / SEGS;
  Raw8<T> rq[NIT], rk[NIT], rv[NIT], rg[NIT];
#pragma unroll
  for (int it = 0; it < NIT; ++it) {
    if (row[it] >= 0) {
      const size_t base = (size_t)row[it] * 3 * H + h * HD + d;
      if (!CLS || s0 + it * ROWS_PER_PASS < 16) rq[it] = load_raw8(qkv + base);
      rk[it] = load_raw8(qkv + base + H); rv[it] = load_raw8(qkv + base + 2 * H);
      if constexpr (WITH_DO) {
        if (!CLS) rg[it] = load_raw8(dctx + (size_t)row[it] * H + h * HD + d);
        else if (s0 + it * ROWS_PER_PASS == 0) rg[it] = load_raw8(dctx + (size_t)b * H + h * HD + d);
        else rg[it].v = make_uint4(0u, 0u, 0u, 0u);
      }
    }
  }
  constexpr bool PAIRS = WITH_DO || SP < 64;
  const Raw8<T> bq = load_raw8(bqkv + h * HD + d), bk = load_raw8(bqkv + H + h * HD + d), bv = load_raw8(bqkv + 2 * H + h * HD + d);
  const auto sum = [](const Raw8<T>& x, const Raw8<T>& bias) -> uint4 {
    if constexpr (PAIRS) return add16x8<T>(x.v, bias.v);
    float a[8], c[8];
    unpack8(x, a);
    unpack8(bias, c);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] += c[j];
    return pack16x8<T>(a);
  };
#pragma unroll
  for (int it = 0; it < NIT; ++it) {
    const int s = s0 + it * ROWS_PER_PASS;
    if (s >= lim) continue;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    const bool on = row[it] >= 0;
    if (!CLS || s < 16) *reinterpret_cast<uint4*>(sQ + s * RP + d) = on ? sum(rq[it], bq) : zero;
    *reinterpret_cast<uint4*>(sK + s * RP + d) = on ? sum(rk[it], bk) : zero;
    *reinterpret_cast<uint4*>(sV + s * RP + d) = on ? sum(rv[it], bv) : zero;
    if constexpr (WITH_DO) { if (!CLS || s < 16) *reinterpret_cast<uint4*>(sDO + s * RP + d) = on ? rg[it].v : zero; }
  }
}

// First-token variant, backward: dst rows of the sequence = src row b for token 0, zeros for the others, columns of head h.
template <typename T, int HD>
__device__ __forceinline__ void spread_first(const FirstTok<T>& ft, const int* sRow, int len, int b, int h, int H) {
  constexpr int SEGS = HD / 8;
  for (int i = threadIdx.x; i < len * SEGS; i += blockDim.x) {
    const int s = i / SEGS, c = h * HD + (i % SEGS) * 8, row = sRow[s];
    if (row < 0) continue;
    *reinterpret_cast<uint4*>(ft.dst + (size_t)row * H + c) =
        s == 0 ? *reinterpret_cast<const uint4*>(ft.src + (size_t)b * H + c) : make_uint4(0u, 0u, 0u, 0u);
  }
}
// ... and the zero gradient of the queries behind the 16 of the first tile (dst already at the head's first column).
template <typename T, int HD>
__device__ __forceinline__ void zero_rest(T* dst, const int* sRow, int len, int ld) {
  constexpr int SEGS = HD / 8;
  for (int i = 16 * SEGS + threadIdx.x; i < len * SEGS; i += blockDim.x) {
    const int row = sRow[i / SEGS];
    if (row >= 0) *reinterpret_cast<uint4*>(dst + (size_t)row * ld + (i % SEGS) * 8) = make_uint4(0u, 0u, 0u, 0u);
  }
}

template <typename T, int SP, int HD, bool CLS>
__global__ void __launch_bounds__(SP * 2, SP == 128 ? 2 : SP == 64 ? 4 : SP == 32 ? 9 : 16) attention_fwd_mma_kernel(
    const T* __restrict__ qkv, const T* __restrict__ bqkv, const int* __restrict__ mask, T* __restrict__ ctx,
    T* __restrict__ probs, int S, int H, int nh, float p, const int* __restrict__ seed_ptr, uint32_t stream, const Tok tk, int len_lo,
    const FirstTok<T> ft) {
  rb::grid_dep_wait();        // launched with launch_pdl: nothing above touches global memory
  rb::grid_dep_launch();      // the kernel that follows may start its set-up; it waits for this grid before reading
  extern __shared__ __align__(128) uint8_t sm_raw[];
  constexpr int RP = HD + 8;
  T* sQ = reinterpret_cast<T*>(sm_raw);
  T* sK = sQ + SP * RP;
  T* sV = sK + SP * RP;
  int* sRow = reinterpret_cast<int*>(sV + SP * RP);            // row of each token, -1 = none
  uint8_t* sCode = reinterpret_cast<uint8_t*>(sRow + SP);      // per key: 0 = no such token, 1 = attend, 2 = masked
  const int h = blockIdx.x, b = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const uint32_t seed = p > 0.f ? (uint32_t)(*seed_ptr) : 0u;
  const float inv_keep = p > 0.f ? 1.f / (1.f - p) : 1.f;
  const float scale = rsqrtf((float)HD);
  if (!CLS && tk.slot != nullptr && b == (int)gridDim.y - 1) clear_zero_rows<T>(tk, ctx, H, h * HD, HD);
  int srow[HD / 16];
  if constexpr (SP < 64) stage_rows<SP, HD>(srow, tk, b, S, S);
  const int trow = threadIdx.x < SP && (int)threadIdx.x < S ? seq_row(tk, b, S, threadIdx.x) : -1;    // of token threadIdx.x
  const int tmask = threadIdx.x < SP && (int)threadIdx.x < S ? mask[b * S + threadIdx.x] : 0;
  const int len = seq_len(tk, b, S), lim = (len + 15) & ~15;
  if (len > SP || len <= len_lo) return;       // another launch serves this length
  if constexpr (SP >= 64) stage_rows<SP, HD>(srow, tk, b, S, len);
  if (threadIdx.x < SP) {
    sRow[threadIdx.x] = trow;
    sCode[threadIdx.x] = trow >= 0 ? (tmask != 0 ? 1 : 2) : 0;
  }
  stage_operands<T, SP, HD, false, CLS>(qkv, bqkv, nullptr, sQ, sK, sV, nullptr, srow, b, h, H, lim);
  __syncthreads();
  const int r0 = warp * 16;
  if (r0 >= (CLS ? 16 : lim)) return;
  if (CLS && lane < HD / 8)
    *reinterpret_cast<uint4*>(ft.dst + (size_t)b * H + h * HD + 8 * lane) =
        *reinterpret_cast<const uint4*>(ft.src + (size_t)sRow[0] * H + h * HD + 8 * lane);
  float acc[SP / 8][4];
#pragma unroll
  for (int j = 0; j < SP / 8; ++j) { acc[j][0] = 0.f; acc[j][1] = 0.f; acc[j][2] = 0.f; acc[j][3] = 0.f; }
  rows_times_transposed<T, SP, HD>(acc, sQ, sK, r0, lane, lim);
  // softmax of rows r0 + g (elements 0, 1 of each tile) and r0 + g + 8 (elements 2, 3)
  float mx0 = -1e30f, mx1 = -1e30f;
#pragma unroll
  for (int j = 0; j < SP / 8; ++j) {
    if (8 * j >= lim) continue;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const bool on = sCode[8 * j + 2 * t + e] == 1;
      acc[j][e] = on ? acc[j][e] * scale : -1e30f;
      acc[j][2 + e] = on ? acc[j][2 + e] * scale : -1e30f;
      mx0 = fmaxf(mx0, acc[j][e]);
      mx1 = fmaxf(mx1, acc[j][2 + e]);
    }
  }
  mx0 = quad_max(mx0); mx1 = quad_max(mx1);
  float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
  for (int j = 0; j < SP / 8; ++j) {
    if (8 * j >= lim) continue;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const bool in_range = sCode[8 * j + 2 * t + e] != 0;
      acc[j][e] = in_range ? __expf(acc[j][e] - mx0) : 0.f;
      acc[j][2 + e] = in_range ? __expf(acc[j][2 + e] - mx1) : 0.f;
      sum0 += acc[j][e];
      sum1 += acc[j][2 + e];
    }
  }
  sum0 = quad_sum(sum0); sum1 = quad_sum(sum1);
  const int i0 = r0 + g, i1 = r0 + g + 8;
  const int row0 = !CLS ? sRow[i0] : (i0 == 0 ? b : -1), row1 = CLS ? -1 : sRow[i1];     // rows of ctx
  const float inv0 = row0 >= 0 ? 1.f / sum0 : 0.f, inv1 = row1 >= 0 ? 1.f / sum1 : 0.f;
  const size_t prow0 = ((size_t)(b * nh + h) * S + i0) * S, prow1 = prow0 + 8 * S;
  const bool pair_store = (S & 1) == 0;   // then every (row, even column) element is 4-byte aligned
  uint32_t pf[SP / 16][4];                // P~ as the A operand of O = P~ V
#pragma unroll
  for (int j = 0; j < SP / 8; ++j) {
    if (8 * j >= lim) continue;
    const int c = 8 * j + 2 * t;
    // the stored probabilities are the rounded ones, as in the unfused op
    const uint32_t u0 = Pack<T>::pack(acc[j][0] * inv0, acc[j][1] * inv0);
    const uint32_t u1 = Pack<T>::pack(acc[j][2] * inv1, acc[j][3] * inv1);
    if (row0 >= 0) {
      if (pair_store) { if (c < S) *reinterpret_cast<uint32_t*>(probs + prow0 + c) = u0; }
      else {
        const T* e = reinterpret_cast<const T*>(&u0);
        if (c < S) probs[prow0 + c] = e[0];
        if (c + 1 < S) probs[prow0 + c + 1] = e[1];
      }
    }
    if (row1 >= 0) {
      if (pair_store) { if (c < S) *reinterpret_cast<uint32_t*>(probs + prow1 + c) = u1; }
      else {
        const T* e = reinterpret_cast<const T*>(&u1);
        if (c < S) probs[prow1 + c] = e[0];
        if (c + 1 < S) probs[prow1 + c + 1] = e[1];
      }
    }
    float2 q0 = Pack<T>::unpack(u0), q1 = Pack<T>::unpack(u1);
    if (p > 0.f) {
      q0.x = keep(seed, stream, (uint32_t)(prow0 + c), p) ? q0.x * inv_keep : 0.f;
      q0.y = keep(seed, stream, (uint32_t)(prow0 + c + 1), p) ? q0.y * inv_keep : 0.f;
      q1.x = keep(seed, stream, (uint32_t)(prow1 + c), p) ? q1.x * inv_keep : 0.f;
      q1.y = keep(seed, stream, (uint32_t)(prow1 + c + 1), p) ? q1.y * inv_keep : 0.f;
    }
    // tiles 2 kq and 2 kq + 1 are the left and right halves of the 16-wide A block kq
    pf[j >> 1][(j & 1) * 2 + 0] = Pack<T>::pack(q0.x, q0.y);
    pf[j >> 1][(j & 1) * 2 + 1] = Pack<T>::pack(q1.x, q1.y);
  }
  float out[HD / 8][4];
#pragma unroll
  for (int jd = 0; jd < HD / 8; ++jd) { out[jd][0] = 0.f; out[jd][1] = 0.f; out[jd][2] = 0.f; out[jd][3] = 0.f; }
  frag_times_rows<T, SP, HD>(out, pf, sV, lane, lim);
  write_rows<T>(out, ctx + h * HD, H, row0, row1, lane, nullptr);
}

template <typename T, int SP, int HD, bool CLS>
__global__ void __launch_bounds__(SP * 2, SP == 64 ? 4 : SP == 32 ? 8 : 16) attention_bwd_mma_kernel(
    const T* __restrict__ dctx, const T* __restrict__ qkv, const T* __restrict__ bqkv, const T* __restrict__ probs,
    T* __restrict__ dqkv, int S, int H, int nh, float p, const int* __restrict__ seed_ptr, uint32_t stream,
    float* __restrict__ bias_acc, const Tok tk, int len_lo, const FirstTok<T> ft) {
  rb::grid_dep_wait();
  rb::grid_dep_launch();
  extern __shared__ __align__(128) uint8_t sm_raw[];
  constexpr int RP = HD + 8;
  constexpr int PP = SP + 8;   // 4-byte fragment stores of a quad group land on distinct banks
  T* sQ = reinterpret_cast<T*>(sm_raw);
  T* sK = sQ + SP * RP;
  T* sV = sK + SP * RP;
  T* sDO = sV + SP * RP;
  T* sDS = sDO + SP * RP;      // [query][key] dS
  T* sW = sDS + SP * PP;       // [query][key] dropped-out probabilities P~
  float* sBias = reinterpret_cast<float*>(sW + SP * PP);   // [3][HD] column sums of dQ, dK, dV
  int* sRow = reinterpret_cast<int*>(sBias + 3 * HD);      // row of each token, -1 = none
  const int h = blockIdx.x, b = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const uint32_t seed = p > 0.f ? (uint32_t)(*seed_ptr) : 0u;
  const float inv_keep = p > 0.f ? 1.f / (1.f - p) : 1.f;
  const float scale = rsqrtf((float)HD);
  if (bias_acc != nullptr)
    for (int i = threadIdx.x; i < 3 * HD; i += blockDim.x) sBias[i] = 0.f;
  if (tk.slot != nullptr && b == (int)gridDim.y - 1)
    for (int w = 0; w < (CLS ? 4 : 3); ++w)
      clear_zero_rows<T>(tk, w < 3 ? dqkv : ft.dst, w < 3 ? 3 * H : H, (w < 3 ? w * H : 0) + h * HD, HD);
  int srow[HD / 16];
  if constexpr (SP < 64) stage_rows<SP, HD>(srow, tk, b, S, S);
  const int trow = threadIdx.x < SP && (int)threadIdx.x < S ? seq_row(tk, b, S, threadIdx.x) : -1;    // of token threadIdx.x
  const int len = seq_len(tk, b, S), lim = (len + 15) & ~15;
  if (len > SP || len <= len_lo) return;       // another launch serves this length
  if constexpr (SP >= 64) stage_rows<SP, HD>(srow, tk, b, S, len);
  if (threadIdx.x < SP) sRow[threadIdx.x] = trow;
  const int r0 = warp * 16;
  const int i0 = r0 + g, i1 = r0 + g + 8;
  const size_t prow0 = ((size_t)(b * nh + h) * S + i0) * S, prow1 = ((size_t)(b * nh + h) * S + i1) * S;
  const bool pair_load = (S & 1) == 0;
  uint32_t wf[SP / 8][2];     // the probabilities of rows i0 / i1 (of rows that are no kept token: anything)
#pragma unroll
  for (int j = 0; j < SP / 8; ++j) {
    const int c = 8 * j + 2 * t;
    wf[j][0] = load_pair_raw<T>(probs, prow0 + c, r0 < lim && 8 * j < lim && i0 < (CLS ? 1 : S) && c < S, c + 1 < S, pair_load);
    wf[j][1] = load_pair_raw<T>(probs, prow1 + c, r0 < lim && 8 * j < lim && i1 < (CLS ? 1 : S) && c < S, c + 1 < S, pair_load);
  }
  stage_operands<T, SP, HD, true, CLS>(qkv, bqkv, dctx, sQ, sK, sV, sDO, srow, b, h, H, lim);
  __syncthreads();
  const int row0 = sRow[r0 + g], row1 = sRow[r0 + g + 8];
  const int qlim = CLS ? 16 : lim;             // queries that have a gradient (CLS: the rows behind the first are zeros)
  if (CLS) {
    spread_first<T, HD>(ft, sRow, len, b, h, H);
    zero_rest<T, HD>(dqkv + h * HD, sRow, len, 3 * H);
  }
  if (r0 < qlim) {
    // dP for this warp's 16 query rows, then dS and P~ in registers
    float acc[SP / 8][4];
#pragma unroll
    for (int j = 0; j < SP / 8; ++j) { acc[j][0] = 0.f; acc[j][1] = 0.f; acc[j][2] = 0.f; acc[j][3] = 0.f; }
    rows_times_transposed<T, SP, HD>(acc, sDO, sV, r0, lane, lim);
    float dot0 = 0.f, dot1 = 0.f;
#pragma unroll
    for (int j = 0; j < SP / 8; ++j) {
      if (8 * j >= lim) continue;
      const int c = 8 * j + 2 * t;
      if (row0 < 0) wf[j][0] = 0u;
      if (row1 < 0) wf[j][1] = 0u;
      const float2 pr0 = Pack<T>::unpack(wf[j][0]), pr1 = Pack<T>::unpack(wf[j][1]);
      float m00 = 1.f, m01 = 1.f, m10 = 1.f, m11 = 1.f;
      if (p > 0.f) {
        m00 = keep(seed, stream, (uint32_t)(prow0 + c), p) ? inv_keep : 0.f;
        m01 = keep(seed, stream, (uint32_t)(prow0 + c + 1), p) ? inv_keep : 0.f;
        m10 = keep(seed, stream, (uint32_t)(prow1 + c), p) ? inv_keep : 0.f;
        m11 = keep(seed, stream, (uint32_t)(prow1 + c + 1), p) ? inv_keep : 0.f;
      }
      // dP~ -> dP through the dropout mask; acc keeps dP, the probabilities move to wf as P (plain) for now
      acc[j][0] *= m00; acc[j][1] *= m01; acc[j][2] *= m10; acc[j][3] *= m11;
      dot0 += acc[j][0] * pr0.x + acc[j][1] * pr0.y;
      dot1 += acc[j][2] * pr1.x + acc[j][3] * pr1.y;
      // dS needs the row's dot product first: park P * dP and P, finish below
      const uint32_t w0 = Pack<T>::pack(pr0.x * m00, pr0.y * m01), w1 = Pack<T>::pack(pr1.x * m10, pr1.y * m11);
      *reinterpret_cast<uint32_t*>(sW + i0 * PP + c) = w0;
      *reinterpret_cast<uint32_t*>(sW + i1 * PP + c) = w1;
    }
    dot0 = quad_sum(dot0); dot1 = quad_sum(dot1);
    uint32_t dsf[SP / 16][4];   // dS as the A operand of dQ = dS K
#pragma unroll
    for (int j = 0; j < SP / 8; ++j) {
      if (8 * j >= lim) continue;
      const int c = 8 * j + 2 * t;
      const float2 pr0 = Pack<T>::unpack(wf[j][0]), pr1 = Pack<T>::unpack(wf[j][1]);
      const uint32_t d0 = Pack<T>::pack(pr0.x * (acc[j][0] - dot0) * scale, pr0.y * (acc[j][1] - dot0) * scale);
      const uint32_t d1 = Pack<T>::pack(pr1.x * (acc[j][2] - dot1) * scale, pr1.y * (acc[j][3] - dot1) * scale);
      *reinterpret_cast<uint32_t*>(sDS + i0 * PP + c) = d0;
      *reinterpret_cast<uint32_t*>(sDS + i1 * PP + c) = d1;
      dsf[j >> 1][(j & 1) * 2 + 0] = d0;
      dsf[j >> 1][(j & 1) * 2 + 1] = d1;
    }
    float out[HD / 8][4];
#pragma unroll
    for (int jd = 0; jd < HD / 8; ++jd) { out[jd][0] = 0.f; out[jd][1] = 0.f; out[jd][2] = 0.f; out[jd][3] = 0.f; }
    frag_times_rows<T, SP, HD>(out, dsf, sK, lane, lim);
    write_rows<T>(out, dqkv + h * HD, 3 * H, row0, row1, lane,
                  bias_acc != nullptr ? sBias : nullptr);
  }
  __syncthreads();
  // this warp's 16 key rows of dK = dS^T Q and dV = P~^T dO
  if (r0 < lim) {
    float out[HD / 8][4];
#pragma unroll
    for (int jd = 0; jd < HD / 8; ++jd) { out[jd][0] = 0.f; out[jd][1] = 0.f; out[jd][2] = 0.f; out[jd][3] = 0.f; }
    transposed_times_rows<T, SP, HD>(out, sDS, PP, r0, sQ, lane, qlim);
    write_rows<T>(out, dqkv + H + h * HD, 3 * H, row0, row1, lane,
                  bias_acc != nullptr ? sBias + HD : nullptr);
#pragma unroll
    for (int jd = 0; jd < HD / 8; ++jd) { out[jd][0] = 0.f; out[jd][1] = 0.f; out[jd][2] = 0.f; out[jd][3] = 0.f; }
    transposed_times_rows<T, SP, HD>(out, sW, PP, r0, sDO, lane, qlim);
    write_rows<T>(out, dqkv + 2 * H + h * HD, 3 * H, row0, row1, lane,
                  bias_acc != nullptr ? sBias + 2 * HD : nullptr);
  }
  if (bias_acc != nullptr) {
    // the bias gradient of the packed projection is the column sum of dqkv: add this (batch, head)'s part to
    // one of the 8 replicas of the step-wide accumulator (converted later by the deferred finalize kernel)
    __syncthreads();
    float* my_acc = bias_acc + (size_t)((blockIdx.y * gridDim.x + blockIdx.x) % 8) * 3 * H;
    for (int i = threadIdx.x; i < 3 * HD; i += blockDim.x)
      atomicAdd(my_acc + (i / HD) * H + h * HD + (i % HD), sBias[i]);
  }
}


// two consecutive elements idx, idx + 1 of a [.., S] row; ok0 / ok1 say which exist; `pair` = 4-byte access allowed
template <typename T>
__device__ __forceinline__ float2 load_pair(const T* __restrict__ base, size_t idx, bool ok0, bool ok1, bool pair) {
  float2 r = make_float2(0.f, 0.f);
  if (ok0) {
    if (pair) r = Pack<T>::unpack(*reinterpret_cast<const uint32_t*>(base + idx));
    else { r.x = to_f(base[idx]); if (ok1) r.y = to_f(base[idx + 1]); }
  }
  return r;
}
template <typename T>
__device__ __forceinline__ void store_pair(T* __restrict__ base, size_t idx, uint32_t u, bool ok0, bool ok1, bool pair) {
  if (ok0) {
    if (pair) *reinterpret_cast<uint32_t*>(base + idx) = u;
    else {
      const T* e = reinterpret_cast<const T*>(&u);
      base[idx] = e[0];
      if (ok1) base[idx + 1] = e[1];
    }
  }
}

// ------------------------------------------------------------------------------------ sequences of 65..256 tokens
// The backward of 65..256 tokens and the forward of 129..256 (up to 128 its score rows still fit in registers): one CTA of
// SP / 16 warps per (batch, head), SP = 128 or 256, operands staged once.  What keeps the scores in
// registers at 32..64 tokens does not scale: a warp's 16 x SP score rows and, in the backward, two [SP][SP] tiles in
// shared memory allowed one CTA of 8 warps per SM at 128 tokens and forced two streaming kernels beyond.  So both passes
// walk the keys in blocks of KB = 64 over the resident operands: 128 registers per thread, and the dS and P~ tiles shrink
// to [SP][KB] (112 KB per CTA at SP = 128: two per SM; 218 KB at SP = 256).
// Measured inside the 64 x 256 training step (12 heads, lengths 64..256): streaming kernels 520 (forward) + 842 (dQ) +
// 304 us (dK, dV) per layer padded; packed, on these, 120 and 210 us (both tiles).  Step 11.36 (packed, streaming kernels) ->
// 7.50 ms when they went in.
//   forward   pass 1: running row maximum and sum; pass 2: probabilities (stored for the backward), dropout, O += P~ V
//   backward  pass 1: row sums of dP * P, keeping the dropout decisions as one bit each; pass 2, per key block: dS and P~
//             to shared memory, dQ += dS K, then the block's dK = dS^T Q and dV = P~^T dO, spread over all warps.
constexpr int KB = 64;

template <typename T, int SP, int HD, bool CLS>
__global__ void __launch_bounds__(SP * 2, SP == 128 ? 2 : 1) attention_fwd_blk_kernel(
    const T* __restrict__ qkv, const T* __restrict__ bqkv, const int* __restrict__ mask, T* __restrict__ ctx,
    T* __restrict__ probs, int S, int H, int nh, float p, const int* __restrict__ seed_ptr, uint32_t stream, const Tok tk,
    int len_lo, const FirstTok<T> ft) {
  rb::grid_dep_wait();
  rb::grid_dep_launch();
  extern __shared__ __align__(128) uint8_t sm_raw[];
  constexpr int RP = HD + 8;
  T* sQ = reinterpret_cast<T*>(sm_raw);
  T* sK = sQ + SP * RP;
  T* sV = sK + SP * RP;
  int* sRow = reinterpret_cast<int*>(sV + SP * RP);
  uint8_t* sCode = reinterpret_cast<uint8_t*>(sRow + SP);      // per key: 0 = no such token, 1 = attend, 2 = masked
  const int h = blockIdx.x, b = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const uint32_t seed = p > 0.f ? (uint32_t)(*seed_ptr) : 0u;
  const float inv_keep = p > 0.f ? 1.f / (1.f - p) : 1.f;
  const float scale = rsqrtf((float)HD);
  if (!CLS && tk.slot != nullptr && b == (int)gridDim.y - 1) clear_zero_rows<T>(tk, ctx, H, h * HD, HD);
  int srow[HD / 16];
  const int trow = threadIdx.x < SP && (int)threadIdx.x < S ? seq_row(tk, b, S, threadIdx.x) : -1;    // of token threadIdx.x
  const int tmask = threadIdx.x < SP && (int)threadIdx.x < S ? mask[b * S + threadIdx.x] : 0;
  const int len = seq_len(tk, b, S), lim = (len + 15) & ~15;
  if (len > SP || len <= len_lo) return;
  stage_rows<SP, HD>(srow, tk, b, S, len);
  if (threadIdx.x < SP) {
    sRow[threadIdx.x] = trow;
    sCode[threadIdx.x] = trow >= 0 ? (tmask != 0 ? 1 : 2) : 0;
  }
  stage_operands<T, SP, HD, false, CLS>(qkv, bqkv, nullptr, sQ, sK, sV, nullptr, srow, b, h, H, lim);
  __syncthreads();
  const int r0 = warp * 16;
  if (r0 >= (CLS ? 16 : lim)) return;
  if (CLS && lane < HD / 8)
    *reinterpret_cast<uint4*>(ft.dst + (size_t)b * H + h * HD + 8 * lane) =
        *reinterpret_cast<const uint4*>(ft.src + (size_t)sRow[0] * H + h * HD + 8 * lane);
  float m0 = -1e30f, m1 = -1e30f, l0 = 0.f, l1 = 0.f;
#pragma unroll 1
  for (int k0 = 0; k0 < lim; k0 += KB) {
    float acc[KB / 8][4];
#pragma unroll
    for (int j = 0; j < KB / 8; ++j) { acc[j][0] = 0.f; acc[j][1] = 0.f; acc[j][2] = 0.f; acc[j][3] = 0.f; }
    rows_times_transposed<T, KB, HD>(acc, sQ, sK + k0 * RP, r0, lane, lim - k0);
    float b0 = -1e30f, b1 = -1e30f;
#pragma unroll
    for (int j = 0; j < KB / 8; ++j) {
      if (k0 + 8 * j >= lim) continue;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const bool on = sCode[k0 + 8 * j + 2 * t + e] == 1;
        acc[j][e] = on ? acc[j][e] * scale : -1e30f;
        acc[j][2 + e] = on ? acc[j][2 + e] * scale : -1e30f;
        b0 = fmaxf(b0, acc[j][e]);
        b1 = fmaxf(b1, acc[j][2 + e]);
      }
    }
    const float n0 = fmaxf(m0, quad_max(b0)), n1 = fmaxf(m1, quad_max(b1));
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int j = 0; j < KB / 8; ++j) {
      if (k0 + 8 * j >= lim) continue;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (sCode[k0 + 8 * j + 2 * t + e] != 0) { s0 += __expf(acc[j][e] - n0); s1 += __expf(acc[j][2 + e] - n1); }
      }
    }
    l0 = l0 * __expf(m0 - n0) + s0;
    l1 = l1 * __expf(m1 - n1) + s1;
    m0 = n0; m1 = n1;
  }
  l0 = quad_sum(l0); l1 = quad_sum(l1);
  const int i0 = r0 + g, i1 = r0 + g + 8;
  const int row0 = !CLS ? sRow[i0] : (i0 == 0 ? b : -1), row1 = CLS ? -1 : sRow[i1];     // rows of ctx
  const float inv0 = row0 >= 0 ? 1.f / l0 : 0.f, inv1 = row1 >= 0 ? 1.f / l1 : 0.f;
  const size_t prow0 = ((size_t)(b * nh + h) * S + i0) * S, prow1 = ((size_t)(b * nh + h) * S + i1) * S;
  const bool pair = (S & 1) == 0;          // then every (row, even column) element is 4-byte aligned
  float out[HD / 8][4];
#pragma unroll
  for (int jd = 0; jd < HD / 8; ++jd) { out[jd][0] = 0.f; out[jd][1] = 0.f; out[jd][2] = 0.f; out[jd][3] = 0.f; }
#pragma unroll 1
  for (int k0 = 0; k0 < lim; k0 += KB) {
    float acc[KB / 8][4];
#pragma unroll
    for (int j = 0; j < KB / 8; ++j) { acc[j][0] = 0.f; acc[j][1] = 0.f; acc[j][2] = 0.f; acc[j][3] = 0.f; }
    rows_times_transposed<T, KB, HD>(acc, sQ, sK + k0 * RP, r0, lane, lim - k0);
    uint32_t pf[KB / 16][4];
#pragma unroll
    for (int j = 0; j < KB / 8; ++j) {
      if (k0 + 8 * j >= lim) continue;
      const int key = k0 + 8 * j + 2 * t;
      const int c0 = sCode[key], c1 = sCode[key + 1];
      const float e00 = c0 != 0 ? __expf((c0 == 1 ? acc[j][0] * scale : -1e30f) - m0) * inv0 : 0.f;
      const float e01 = c1 != 0 ? __expf((c1 == 1 ? acc[j][1] * scale : -1e30f) - m0) * inv0 : 0.f;
      const float e10 = c0 != 0 ? __expf((c0 == 1 ? acc[j][2] * scale : -1e30f) - m1) * inv1 : 0.f;
      const float e11 = c1 != 0 ? __expf((c1 == 1 ? acc[j][3] * scale : -1e30f) - m1) * inv1 : 0.f;
      // the stored probabilities are the rounded ones, as in the unfused op
      const uint32_t u0 = Pack<T>::pack(e00, e01), u1 = Pack<T>::pack(e10, e11);
      store_pair<T>(probs, prow0 + key, u0, row0 >= 0 && key < S, key + 1 < S, pair);
      store_pair<T>(probs, prow1 + key, u1, row1 >= 0 && key < S, key + 1 < S, pair);
      float2 q0 = Pack<T>::unpack(u0), q1 = Pack<T>::unpack(u1);
      if (p > 0.f) {
        q0.x = keep(seed, stream, (uint32_t)(prow0 + key), p) ? q0.x * inv_keep : 0.f;
        q0.y = keep(seed, stream, (uint32_t)(prow0 + key + 1), p) ? q0.y * inv_keep : 0.f;
        q1.x = keep(seed, stream, (uint32_t)(prow1 + key), p) ? q1.x * inv_keep : 0.f;
        q1.y = keep(seed, stream, (uint32_t)(prow1 + key + 1), p) ? q1.y * inv_keep : 0.f;
      }
      pf[j >> 1][(j & 1) * 2 + 0] = Pack<T>::pack(q0.x, q0.y);
      pf[j >> 1][(j & 1) * 2 + 1] = Pack<T>::pack(q1.x, q1.y);
    }
    frag_times_rows<T, KB, HD>(out, pf, sV + k0 * RP, lane, lim - k0);
  }
  write_rows<T>(out, ctx + h * HD, H, row0, row1, lane, nullptr);
}

template <typename T, int SP, int HD, bool CLS>
__global__ void __launch_bounds__(SP * 2, SP == 128 ? 2 : 1) attention_bwd_blk_kernel(
    const T* __restrict__ dctx, const T* __restrict__ qkv, const T* __restrict__ bqkv, const T* __restrict__ probs,
    T* __restrict__ dqkv, int S, int H, int nh, float p, const int* __restrict__ seed_ptr, uint32_t stream,
    float* __restrict__ bias_acc, const Tok tk, int len_lo, const FirstTok<T> ft) {
  rb::grid_dep_wait();
  rb::grid_dep_launch();
  extern __shared__ __align__(128) uint8_t sm_raw[];
  constexpr int RP = HD + 8, PB = KB + 8;
  constexpr int NW = SP / 16;                      // warps
  constexpr int SLICES = NW / 8;                   // column slices of a dK / dV tile: 4 key tiles x 2 x SLICES = NW tasks
  constexpr int NJ = HD / 8 / SLICES;
  T* sQ = reinterpret_cast<T*>(sm_raw);
  T* sK = sQ + SP * RP;
  T* sV = sK + SP * RP;
  T* sDO = sV + SP * RP;
  T* sDS = sDO + SP * RP;                          // [query][key of the block] dS
  T* sW = sDS + SP * PB;                           // [query][key of the block] dropped-out probabilities P~
  float* sBias = reinterpret_cast<float*>(sW + SP * PB);   // [3][HD] column sums of dQ, dK, dV
  int* sRow = reinterpret_cast<int*>(sBias + 3 * HD);
  const int h = blockIdx.x, b = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const uint32_t seed = p > 0.f ? (uint32_t)(*seed_ptr) : 0u;
  const float inv_keep = p > 0.f ? 1.f / (1.f - p) : 1.f;
  const float scale = rsqrtf((float)HD);
  if (tk.slot != nullptr && b == (int)gridDim.y - 1)
    for (int w = 0; w < (CLS ? 4 : 3); ++w)
      clear_zero_rows<T>(tk, w < 3 ? dqkv : ft.dst, w < 3 ? 3 * H : H, (w < 3 ? w * H : 0) + h * HD, HD);
  int srow[HD / 16];
  const int trow = threadIdx.x < SP && (int)threadIdx.x < S ? seq_row(tk, b, S, threadIdx.x) : -1;    // of token threadIdx.x
  const int len = seq_len(tk, b, S), lim = (len + 15) & ~15;
  if (len > SP || len <= len_lo) return;
  stage_rows<SP, HD>(srow, tk, b, S, len);
  if (bias_acc != nullptr)
    for (int i = threadIdx.x; i < 3 * HD; i += blockDim.x) sBias[i] = 0.f;
  if (threadIdx.x < SP) sRow[threadIdx.x] = trow;
  stage_operands<T, SP, HD, true, CLS>(qkv, bqkv, dctx, sQ, sK, sV, sDO, srow, b, h, H, lim);
  __syncthreads();
  const int r0 = warp * 16, i0 = r0 + g, i1 = r0 + g + 8;
  const int qlim = CLS ? 16 : lim;                 // queries that have a gradient (CLS: the rows behind the first are zeros)
  const bool active = r0 < qlim;                   // this warp's 16 query rows exist
  const int row0 = sRow[i0], row1 = sRow[i1];
  if (CLS) {
    spread_first<T, HD>(ft, sRow, len, b, h, H);
    zero_rest<T, HD>(dqkv + h * HD, sRow, len, 3 * H);
  }
  const size_t prow0 = ((size_t)(b * nh + h) * S + i0) * S, prow1 = ((size_t)(b * nh + h) * S + i1) * S;
  const bool pair = (S & 1) == 0;
  uint32_t kept[SP / KB];                          // dropout decisions: bit 4 j + e of block k is element e of tile j
  float dot0 = 0.f, dot1 = 0.f;
  if (active) {
#pragma unroll
    for (int kb = 0; kb < SP / KB; ++kb) {
      const int k0 = kb * KB;
      kept[kb] = 0xffffffffu;
      if (k0 >= lim) continue;
      uint32_t w0[KB / 8], w1[KB / 8];             // the block's probabilities, on their way during the products
#pragma unroll
      for (int j = 0; j < KB / 8; ++j) {
        const int key = k0 + 8 * j + 2 * t;
        w0[j] = load_pair_raw<T>(probs, prow0 + key, row0 >= 0 && (!CLS || i0 == 0) && k0 + 8 * j < lim && key < S, key + 1 < S, pair);
        w1[j] = load_pair_raw<T>(probs, prow1 + key, row1 >= 0 && (!CLS || i1 == 0) && k0 + 8 * j < lim && key < S, key + 1 < S, pair);
      }
      float acc[KB / 8][4];
#pragma unroll
      for (int j = 0; j < KB / 8; ++j) { acc[j][0] = 0.f; acc[j][1] = 0.f; acc[j][2] = 0.f; acc[j][3] = 0.f; }
      rows_times_transposed<T, KB, HD>(acc, sDO, sV + k0 * RP, r0, lane, lim - k0);
      uint32_t bits = 0u;
#pragma unroll
      for (int j = 0; j < KB / 8; ++j) {
        if (k0 + 8 * j >= lim) continue;
        const int key = k0 + 8 * j + 2 * t;
        const float2 pr0 = Pack<T>::unpack(w0[j]), pr1 = Pack<T>::unpack(w1[j]);
        float m00 = 1.f, m01 = 1.f, m10 = 1.f, m11 = 1.f;
        if (p > 0.f) {
          const bool a = keep(seed, stream, (uint32_t)(prow0 + key), p), c = keep(seed, stream, (uint32_t)(prow0 + key + 1), p);
          const bool d = keep(seed, stream, (uint32_t)(prow1 + key), p), f = keep(seed, stream, (uint32_t)(prow1 + key + 1), p);
          bits |= ((a ? 1u : 0u) | (c ? 2u : 0u) | (d ? 4u : 0u) | (f ? 8u : 0u)) << (4 * j);
          m00 = a ? inv_keep : 0.f; m01 = c ? inv_keep : 0.f; m10 = d ? inv_keep : 0.f; m11 = f ? inv_keep : 0.f;
        }
        dot0 += acc[j][0] * m00 * pr0.x + acc[j][1] * m01 * pr0.y;
        dot1 += acc[j][2] * m10 * pr1.x + acc[j][3] * m11 * pr1.y;
      }
      if (p > 0.f) kept[kb] = bits;
    }
    dot0 = quad_sum(dot0); dot1 = quad_sum(dot1);
  }
  float dq[HD / 8][4];
#pragma unroll
  for (int jd = 0; jd < HD / 8; ++jd) { dq[jd][0] = 0.f; dq[jd][1] = 0.f; dq[jd][2] = 0.f; dq[jd][3] = 0.f; }
#pragma unroll
  for (int kb = 0; kb < SP / KB; ++kb) {
    const int k0 = kb * KB;
    if (k0 >= lim) break;                          // the same answer in every thread
    if (active) {
      uint32_t w0[KB / 8], w1[KB / 8];             // the block's probabilities, on their way during the products
#pragma unroll
      for (int j = 0; j < KB / 8; ++j) {
        const int key = k0 + 8 * j + 2 * t;
        w0[j] = load_pair_raw<T>(probs, prow0 + key, row0 >= 0 && (!CLS || i0 == 0) && k0 + 8 * j < lim && key < S, key + 1 < S, pair);
        w1[j] = load_pair_raw<T>(probs, prow1 + key, row1 >= 0 && (!CLS || i1 == 0) && k0 + 8 * j < lim && key < S, key + 1 < S, pair);
      }
      float acc[KB / 8][4];
#pragma unroll
      for (int j = 0; j < KB / 8; ++j) { acc[j][0] = 0.f; acc[j][1] = 0.f; acc[j][2] = 0.f; acc[j][3] = 0.f; }
      rows_times_transposed<T, KB, HD>(acc, sDO, sV + k0 * RP, r0, lane, lim - k0);
      uint32_t dsf[KB / 16][4];                    // dS as the A operand of dQ += dS K
#pragma unroll
      for (int j = 0; j < KB / 8; ++j) {
        if (k0 + 8 * j >= lim) continue;
        const float2 pr0 = Pack<T>::unpack(w0[j]), pr1 = Pack<T>::unpack(w1[j]);
        const uint32_t bits = kept[kb] >> (4 * j);
        const float m00 = (bits & 1u) ? inv_keep : 0.f, m01 = (bits & 2u) ? inv_keep : 0.f;
        const float m10 = (bits & 4u) ? inv_keep : 0.f, m11 = (bits & 8u) ? inv_keep : 0.f;
        const uint32_t d0 = Pack<T>::pack(pr0.x * (acc[j][0] * m00 - dot0) * scale, pr0.y * (acc[j][1] * m01 - dot0) * scale);
        const uint32_t d1 = Pack<T>::pack(pr1.x * (acc[j][2] * m10 - dot1) * scale, pr1.y * (acc[j][3] * m11 - dot1) * scale);
        const int c = 8 * j + 2 * t;
        *reinterpret_cast<uint32_t*>(sDS + i0 * PB + c) = d0;
        *reinterpret_cast<uint32_t*>(sDS + i1 * PB + c) = d1;
        *reinterpret_cast<uint32_t*>(sW + i0 * PB + c) = Pack<T>::pack(pr0.x * m00, pr0.y * m01);
        *reinterpret_cast<uint32_t*>(sW + i1 * PB + c) = Pack<T>::pack(pr1.x * m10, pr1.y * m11);
        dsf[j >> 1][(j & 1) * 2 + 0] = d0;
        dsf[j >> 1][(j & 1) * 2 + 1] = d1;
      }
      frag_times_rows<T, KB, HD>(dq, dsf, sK + k0 * RP, lane, lim - k0);
    }
    __syncthreads();
    {
      // one 16-key tile of dK (even tasks) or dV (odd ones), or a column slice of it
      const int kt = (warp >> 1) & 3, which = warp & 1, slice = warp >> 3;
      const int key0 = k0 + 16 * kt;
      if (key0 < lim) {
        float out[NJ][4];
#pragma unroll
        for (int jd = 0; jd < NJ; ++jd) { out[jd][0] = 0.f; out[jd][1] = 0.f; out[jd][2] = 0.f; out[jd][3] = 0.f; }
        const int c0 = slice * NJ * 8;
        transposed_times_rows<T, SP, HD, NJ>(out, which == 0 ? sDS : sW, PB, 16 * kt, (which == 0 ? sQ : sDO) + c0, lane, qlim);
        write_rows<T>(out, dqkv + (1 + which) * H + h * HD + c0, 3 * H, sRow[key0 + g], sRow[key0 + g + 8], lane,
                      bias_acc != nullptr ? sBias + (1 + which) * HD + c0 : nullptr);
      }
    }
    __syncthreads();
  }
  if (active) write_rows<T>(dq, dqkv + h * HD, 3 * H, row0, row1, lane, bias_acc != nullptr ? sBias : nullptr);
  if (bias_acc != nullptr) {
    __syncthreads();
    float* my_acc = bias_acc + (size_t)((blockIdx.y * gridDim.x + blockIdx.x) % 8) * 3 * H;
    for (int i = threadIdx.x; i < 3 * HD; i += blockDim.x)
      atomicAdd(my_acc + (i / HD) * H + h * HD + (i % HD), sBias[i]);
  }
}

template <int SP, int HD> constexpr size_t fwd_smem(size_t esz) { return (size_t)3 * SP * (HD + 8) * esz + SP * sizeof(int) + SP; }
template <int SP, int HD> constexpr size_t bwd_smem(size_t esz) {
  return (size_t)4 * SP * (HD + 8) * esz + (size_t)2 * SP * ((SP > 64 ? KB : SP) + 8) * esz + 3 * HD * sizeof(float) + SP * sizeof(int);
}

// One launch of the kernels for sequences of len_lo + 1 .. SP tokens (a CTA whose sequence has another length exits).
template <typename T, int SP, int HD>
static int launch_fwd(const void* qkv, const void* bqkv, const int* mask, void* ctx, void* probs, int b, int S, int H,
                      int nh, float p, const int* seed, unsigned stream_id, const Tok& tk, const void* first_src, void* first_dst, int len_lo,
                      cudaStream_t st) {
  constexpr size_t smem = fwd_smem<SP, HD>(sizeof(T));
  const auto go = [&](auto k) -> int {
    if (smem > 48 * 1024 && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -5;
    rb::launch_pdl(k, dim3(nh, b), dim3(SP * 2), smem, st, (const T*)qkv, (const T*)bqkv, mask, (T*)ctx, (T*)probs, S, H, nh, p, seed, stream_id, tk, len_lo,
                   FirstTok<T>{(const T*)first_src, (T*)first_dst});
    return 0;
  };
  if constexpr (SP > 128) return first_dst ? go(attention_fwd_blk_kernel<T, SP, HD, true>) : go(attention_fwd_blk_kernel<T, SP, HD, false>);
  else return first_dst ? go(attention_fwd_mma_kernel<T, SP, HD, true>) : go(attention_fwd_mma_kernel<T, SP, HD, false>);
}

template <typename T, int SP, int HD>
static int launch_bwd(const void* dctx, const void* qkv, const void* bqkv, const void* probs, void* dqkv, int b, int S,
                      int H, int nh, float p, const int* seed, unsigned stream_id, float* bias_acc, const Tok& tk,
                      const void* first_src, void* first_dst, int len_lo, cudaStream_t st) {
  constexpr size_t smem = bwd_smem<SP, HD>(sizeof(T));
  const auto go = [&](auto k) -> int {
    if (smem > 48 * 1024 && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -5;
    rb::launch_pdl(k, dim3(nh, b), dim3(SP * 2), smem, st, (const T*)dctx, (const T*)qkv, (const T*)bqkv, (const T*)probs,
                   (T*)dqkv, S, H, nh, p, seed, stream_id, bias_acc, tk, len_lo, FirstTok<T>{(const T*)first_src, (T*)first_dst});
    return 0;
  };
  if constexpr (SP > 64) return first_dst ? go(attention_bwd_blk_kernel<T, SP, HD, true>) : go(attention_bwd_blk_kernel<T, SP, HD, false>);
  else return first_dst ? go(attention_bwd_mma_kernel<T, SP, HD, true>) : go(attention_bwd_mma_kernel<T, SP, HD, false>);
}

// Tile sizes by sequence length.  All sequences of a padded batch have length S: one launch of the smallest tile that
// holds it.  Packed sequences have their own lengths: those of at most half the tile go to the next smaller one in a
// launch of their own, where twice as many fit an SM.
#define RB_ATT_LAUNCH(T, HD, FN, S, packed, ...)                                                                    \
  [&]() -> int {                                                                                                    \
    if ((S) <= 16) return FN<T, 16, HD>(__VA_ARGS__, 0, st);                                                        \
    if ((S) <= 32) return FN<T, 32, HD>(__VA_ARGS__, 0, st);                                                        \
    int rc_ = 0;                                                                                                    \
    if ((S) <= 64) {                                                                                                \
      if (packed) rc_ = FN<T, 32, HD>(__VA_ARGS__, 0, st);                                                          \
      return rc_ ? rc_ : FN<T, 64, HD>(__VA_ARGS__, (packed) ? 32 : 0, st);                                         \
    }                                                                                                               \
    if ((S) <= 128) {                                                                                               \
      if (packed) rc_ = FN<T, 64, HD>(__VA_ARGS__, 0, st);                                                          \
      return rc_ ? rc_ : FN<T, 128, HD>(__VA_ARGS__, (packed) ? 64 : 0, st);                                        \
    }                                                                                                               \
    if constexpr (HD == 64) {                                                                                       \
      if (packed) rc_ = FN<T, 128, HD>(__VA_ARGS__, 0, st);                                                         \
      return rc_ ? rc_ : FN<T, 256, HD>(__VA_ARGS__, (packed) ? 128 : 0, st);                                       \
    }                                                                                                               \
    return -4;                                                                                                      \
  }()

// ------------------------------------------------------------------------------------ sequences of 257..512 tokens
// Same math and the same fragment routines, blocked: a CTA of 4 warps owns 64 query rows (forward, dQ) or 64 key
// rows (dK, dV) of one (batch, head) and walks the other dimension in blocks of 128 through shared memory.
//   forward   two passes over the key blocks: running row maximum / sum first, then probabilities (stored for the
//             backward, as for short sequences), dropout and O += P~ V.
//   dQ        two passes as well (the softmax gradient needs the whole row's sum of dP * P before any dS):
//             dP = dO V^T per key block, then dS, written to a [b, nh, S, S] workspace, and dQ += dS K.
//   dK, dV    per block of 64 keys, over query blocks: dS and P~ tiles staged in shared memory (P~ rebuilt from
//             the stored probabilities and the counter-based dropout mask), dK += dS^T Q, dV += P~^T dO.
constexpr int QB = 64;     // rows owned by a CTA
constexpr int KBLK = 128;  // rows of the other dimension per step
constexpr int PPK = QB + 8;

// tokens first.. of sequence b from a [*, ld] matrix (pointer already at this head's first column) -> [n_tile][RP] tile
template <typename T>
__device__ __forceinline__ void stage_block(T* dst, const T* __restrict__ src, size_t ld, const T* __restrict__ bias,
                                            int first, int n_tile, const Tok& tk, int b, int S, int len) {
  for (int i = threadIdx.x; i < n_tile * (HD / 8); i += blockDim.x) {
    const int s = i >> 3, d = (i & 7) * 8;
    float v[8];
    const int row = first + s < len ? seq_row(tk, b, S, first + s) : -1;
    if (row >= 0) {
      load8(src + (size_t)row * ld + d, v);
      if (bias != nullptr) {
        float bb[8];
        load8(bias + d, bb);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] += bb[j];
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = 0.f;
    }
    store8(dst + s * RP + d, v);
  }
}

template <typename T>
__global__ void __launch_bounds__(128) attention_fwd_long_kernel(
    const T* __restrict__ qkv, const T* __restrict__ bqkv, const int* __restrict__ mask, T* __restrict__ ctx,
    T* __restrict__ probs, int S, int H, int nh, float p, const int* __restrict__ seed_ptr, uint32_t stream, const Tok tk) {
  extern __shared__ __align__(128) uint8_t sm_raw[];
  T* sQ = reinterpret_cast<T*>(sm_raw);
  T* sK = sQ + QB * RP;
  T* sV = sK + KBLK * RP;
  uint8_t* sCode = reinterpret_cast<uint8_t*>(sV + KBLK * RP);   // per key of the block: 0 beyond S, 1 attend, 2 masked
  const int h = blockIdx.x, b = blockIdx.y, q0 = blockIdx.z * QB;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const uint32_t seed = p > 0.f ? (uint32_t)(*seed_ptr) : 0u;
  const float inv_keep = p > 0.f ? 1.f / (1.f - p) : 1.f;
  const float scale = rsqrtf((float)HD);
  const T* base = qkv + h * HD;
  if (tk.slot != nullptr && b == (int)gridDim.y - 1 && q0 == 0) clear_zero_rows<T>(tk, ctx, H, h * HD, HD);
  const int len = seq_len(tk, b, S), lim = (len + 15) & ~15;
  if (q0 >= len) return;
  stage_block<T>(sQ, base, (size_t)3 * H, bqkv + h * HD, q0, QB, tk, b, S, len);
  const int r0 = warp * 16;
  const int i0 = q0 + r0 + g, i1 = i0 + 8;
  const int row0 = i0 < len ? seq_row(tk, b, S, i0) : -1, row1 = i1 < len ? seq_row(tk, b, S, i1) : -1;
  const int nkb = (len + KBLK - 1) / KBLK;
  float m0 = -1e30f, m1 = -1e30f, l0 = 0.f, l1 = 0.f;
  for (int kb = 0; kb < nkb; ++kb) {
    __syncthreads();
    stage_block<T>(sK, base + H, (size_t)3 * H, bqkv + H + h * HD, kb * KBLK, KBLK, tk, b, S, len);
    for (int j = threadIdx.x; j < KBLK; j += blockDim.x) {
      const int key = kb * KBLK + j;
      sCode[j] = key < len && seq_row(tk, b, S, key) >= 0 ? (mask[b * S + key] != 0 ? 1 : 2) : 0;
    }
    __syncthreads();
    float acc[KBLK / 8][4];
#pragma unroll
    for (int j = 0; j < KBLK / 8; ++j) { acc[j][0] = 0.f; acc[j][1] = 0.f; acc[j][2] = 0.f; acc[j][3] = 0.f; }
    rows_times_transposed<T, KBLK>(acc, sQ, sK, r0, lane, lim - kb * KBLK);
    float bm0 = -1e30f, bm1 = -1e30f;
#pragma unroll
    for (int j = 0; j < KBLK / 8; ++j) {
      if (kb * KBLK + 8 * j >= lim) continue;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int code = sCode[8 * j + 2 * t + e];
        acc[j][e] = code == 1 ? acc[j][e] * scale : -1e30f;
        acc[j][2 + e] = code == 1 ? acc[j][2 + e] * scale : -1e30f;
        if (code != 0) { bm0 = fmaxf(bm0, acc[j][e]); bm1 = fmaxf(bm1, acc[j][2 + e]); }
      }
    }
    const float n0 = fmaxf(m0, quad_max(bm0)), n1 = fmaxf(m1, quad_max(bm1));
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int j = 0; j < KBLK / 8; ++j) {
      if (kb * KBLK + 8 * j >= lim) continue;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (sCode[8 * j + 2 * t + e] != 0) { s0 += __expf(acc[j][e] - n0); s1 += __expf(acc[j][2 + e] - n1); }
      }
    }
    l0 = l0 * __expf(m0 - n0) + s0;
    l1 = l1 * __expf(m1 - n1) + s1;
    m0 = n0; m1 = n1;
  }
  l0 = quad_sum(l0); l1 = quad_sum(l1);
  const float inv0 = row0 >= 0 ? 1.f / l0 : 0.f, inv1 = row1 >= 0 ? 1.f / l1 : 0.f;
  const size_t prow0 = ((size_t)(b * nh + h) * S + i0) * S, prow1 = ((size_t)(b * nh + h) * S + i1) * S;
  const bool pair = (S & 1) == 0;
  float out[HD / 8][4];
#pragma unroll
  for (int jd = 0; jd < HD / 8; ++jd) { out[jd][0] = 0.f; out[jd][1] = 0.f; out[jd][2] = 0.f; out[jd][3] = 0.f; }
  for (int kb = 0; kb < nkb; ++kb) {
    __syncthreads();
    stage_block<T>(sK, base + H, (size_t)3 * H, bqkv + H + h * HD, kb * KBLK, KBLK, tk, b, S, len);
    stage_block<T>(sV, base + 2 * H, (size_t)3 * H, bqkv + 2 * H + h * HD, kb * KBLK, KBLK, tk, b, S, len);
    for (int j = threadIdx.x; j < KBLK; j += blockDim.x) {
      const int key = kb * KBLK + j;
      sCode[j] = key < len && seq_row(tk, b, S, key) >= 0 ? (mask[b * S + key] != 0 ? 1 : 2) : 0;
    }
    __syncthreads();
    float acc[KBLK / 8][4];
#pragma unroll
    for (int j = 0; j < KBLK / 8; ++j) { acc[j][0] = 0.f; acc[j][1] = 0.f; acc[j][2] = 0.f; acc[j][3] = 0.f; }
    rows_times_transposed<T, KBLK>(acc, sQ, sK, r0, lane, lim - kb * KBLK);
    uint32_t pf[KBLK / 16][4];
#pragma unroll
    for (int j = 0; j < KBLK / 8; ++j) {
      if (kb * KBLK + 8 * j >= lim) continue;
      const int c = 8 * j + 2 * t, key = kb * KBLK + c;
      float e00, e01, e10, e11;
      {
        const int c0 = sCode[c], c1 = sCode[c + 1];
        e00 = c0 != 0 ? __expf((c0 == 1 ? acc[j][0] * scale : -1e30f) - m0) * inv0 : 0.f;
        e01 = c1 != 0 ? __expf((c1 == 1 ? acc[j][1] * scale : -1e30f) - m0) * inv0 : 0.f;
        e10 = c0 != 0 ? __expf((c0 == 1 ? acc[j][2] * scale : -1e30f) - m1) * inv1 : 0.f;
        e11 = c1 != 0 ? __expf((c1 == 1 ? acc[j][3] * scale : -1e30f) - m1) * inv1 : 0.f;
      }
      const uint32_t u0 = Pack<T>::pack(e00, e01), u1 = Pack<T>::pack(e10, e11);
      store_pair<T>(probs, prow0 + key, u0, row0 >= 0 && key < S, key + 1 < S, pair);
      store_pair<T>(probs, prow1 + key, u1, row1 >= 0 && key < S, key + 1 < S, pair);
      float2 q0v = Pack<T>::unpack(u0), q1v = Pack<T>::unpack(u1);
      if (p > 0.f) {
        q0v.x = keep(seed, stream, (uint32_t)(prow0 + key), p) ? q0v.x * inv_keep : 0.f;
        q0v.y = keep(seed, stream, (uint32_t)(prow0 + key + 1), p) ? q0v.y * inv_keep : 0.f;
        q1v.x = keep(seed, stream, (uint32_t)(prow1 + key), p) ? q1v.x * inv_keep : 0.f;
        q1v.y = keep(seed, stream, (uint32_t)(prow1 + key + 1), p) ? q1v.y * inv_keep : 0.f;
      }
      pf[j >> 1][(j & 1) * 2 + 0] = Pack<T>::pack(q0v.x, q0v.y);
      pf[j >> 1][(j & 1) * 2 + 1] = Pack<T>::pack(q1v.x, q1v.y);
    }
    frag_times_rows<T, KBLK>(out, pf, sV, lane, lim - kb * KBLK);
  }
  write_rows<T>(out, ctx + h * HD, H, row0, row1, lane, nullptr);
}

template <typename T>
__global__ void __launch_bounds__(128) attention_bwd_long_dq_kernel(
    const T* __restrict__ dctx, const T* __restrict__ qkv, const T* __restrict__ bqkv, const T* __restrict__ probs,
    T* __restrict__ ds_ws, T* __restrict__ dqkv, int S, int H, int nh, float p, const int* __restrict__ seed_ptr,
    uint32_t stream, float* __restrict__ bias_acc, const Tok tk) {
  extern __shared__ __align__(128) uint8_t sm_raw[];
  T* sDO = reinterpret_cast<T*>(sm_raw);
  T* sK = sDO + QB * RP;
  T* sV = sK + KBLK * RP;
  float* sBias = reinterpret_cast<float*>(sV + KBLK * RP);   // [HD] column sums of this CTA's dQ rows
  const int h = blockIdx.x, b = blockIdx.y, q0 = blockIdx.z * QB;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const uint32_t seed = p > 0.f ? (uint32_t)(*seed_ptr) : 0u;
  const float inv_keep = p > 0.f ? 1.f / (1.f - p) : 1.f;
  const float scale = rsqrtf((float)HD);
  const T* base = qkv + h * HD;
  if (tk.slot != nullptr && b == (int)gridDim.y - 1 && q0 == 0) clear_zero_rows<T>(tk, dqkv, 3 * H, h * HD, HD);
  const int len = seq_len(tk, b, S), lim = (len + 15) & ~15;
  if (q0 >= len) return;
  if (bias_acc != nullptr)
    for (int i = threadIdx.x; i < HD; i += blockDim.x) sBias[i] = 0.f;
  stage_block<T>(sDO, dctx + h * HD, (size_t)H, nullptr, q0, QB, tk, b, S, len);
  const int r0 = warp * 16;
  const int i0 = q0 + r0 + g, i1 = i0 + 8;
  const int row0 = i0 < len ? seq_row(tk, b, S, i0) : -1, row1 = i1 < len ? seq_row(tk, b, S, i1) : -1;
  const int nkb = (len + KBLK - 1) / KBLK;
  const size_t prow0 = ((size_t)(b * nh + h) * S + i0) * S, prow1 = ((size_t)(b * nh + h) * S + i1) * S;
  const bool pair = (S & 1) == 0;
  float dot0 = 0.f, dot1 = 0.f;
  float out[HD / 8][4];
#pragma unroll
  for (int jd = 0; jd < HD / 8; ++jd) { out[jd][0] = 0.f; out[jd][1] = 0.f; out[jd][2] = 0.f; out[jd][3] = 0.f; }
  for (int pass = 0; pass < 2; ++pass) {
    for (int kb = 0; kb < nkb; ++kb) {
      __syncthreads();
      stage_block<T>(sV, base + 2 * H, (size_t)3 * H, bqkv + 2 * H + h * HD, kb * KBLK, KBLK, tk, b, S, len);
      if (pass == 1) stage_block<T>(sK, base + H, (size_t)3 * H, bqkv + H + h * HD, kb * KBLK, KBLK, tk, b, S, len);
      __syncthreads();
      float acc[KBLK / 8][4];
#pragma unroll
      for (int j = 0; j < KBLK / 8; ++j) { acc[j][0] = 0.f; acc[j][1] = 0.f; acc[j][2] = 0.f; acc[j][3] = 0.f; }
      rows_times_transposed<T, KBLK>(acc, sDO, sV, r0, lane, lim - kb * KBLK);
      uint32_t dsf[KBLK / 16][4];
#pragma unroll
      for (int j = 0; j < KBLK / 8; ++j) {
        if (kb * KBLK + 8 * j >= lim) continue;
        const int key = kb * KBLK + 8 * j + 2 * t;
        const bool k0 = key < S, k1 = key + 1 < S;
        const float2 pr0 = load_pair<T>(probs, prow0 + key, row0 >= 0 && k0, k1, pair);
        const float2 pr1 = load_pair<T>(probs, prow1 + key, row1 >= 0 && k0, k1, pair);
        float m00 = 1.f, m01 = 1.f, m10 = 1.f, m11 = 1.f;
        if (p > 0.f) {
          m00 = keep(seed, stream, (uint32_t)(prow0 + key), p) ? inv_keep : 0.f;
          m01 = keep(seed, stream, (uint32_t)(prow0 + key + 1), p) ? inv_keep : 0.f;
          m10 = keep(seed, stream, (uint32_t)(prow1 + key), p) ? inv_keep : 0.f;
          m11 = keep(seed, stream, (uint32_t)(prow1 + key + 1), p) ? inv_keep : 0.f;
        }
        const float a00 = acc[j][0] * m00, a01 = acc[j][1] * m01, a10 = acc[j][2] * m10, a11 = acc[j][3] * m11;
        if (pass == 0) {
          dot0 += a00 * pr0.x + a01 * pr0.y;
          dot1 += a10 * pr1.x + a11 * pr1.y;
        } else {
          const uint32_t d0 = Pack<T>::pack(pr0.x * (a00 - dot0) * scale, pr0.y * (a01 - dot0) * scale);
          const uint32_t d1 = Pack<T>::pack(pr1.x * (a10 - dot1) * scale, pr1.y * (a11 - dot1) * scale);
          store_pair<T>(ds_ws, prow0 + key, d0, row0 >= 0 && k0, k1, pair);
          store_pair<T>(ds_ws, prow1 + key, d1, row1 >= 0 && k0, k1, pair);
          dsf[j >> 1][(j & 1) * 2 + 0] = d0;
          dsf[j >> 1][(j & 1) * 2 + 1] = d1;
        }
      }
      if (pass == 1) frag_times_rows<T, KBLK>(out, dsf, sK, lane, lim - kb * KBLK);
    }
    if (pass == 0) { dot0 = quad_sum(dot0); dot1 = quad_sum(dot1); }
  }
  write_rows<T>(out, dqkv + h * HD, 3 * H, row0, row1, lane,
                bias_acc != nullptr ? sBias : nullptr);
  if (bias_acc != nullptr) {
    __syncthreads();
    const int cta = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    float* my_acc = bias_acc + (size_t)(cta % 8) * 3 * H;
    for (int i = threadIdx.x; i < HD; i += blockDim.x) atomicAdd(my_acc + h * HD + i, sBias[i]);
  }
}

template <typename T>
__global__ void __launch_bounds__(128) attention_bwd_long_dkv_kernel(
    const T* __restrict__ dctx, const T* __restrict__ qkv, const T* __restrict__ bqkv, const T* __restrict__ probs,
    const T* __restrict__ ds_ws, T* __restrict__ dqkv, int S, int H, int nh, float p, const int* __restrict__ seed_ptr,
    uint32_t stream, float* __restrict__ bias_acc, const Tok tk) {
  extern __shared__ __align__(128) uint8_t sm_raw[];
  T* sDS = reinterpret_cast<T*>(sm_raw);      // [query of the block][key of this CTA]
  T* sW = sDS + KBLK * PPK;
  T* sQ = sW + KBLK * PPK;
  T* sDO = sQ + KBLK * RP;
  float* sBias = reinterpret_cast<float*>(sDO + KBLK * RP);   // [2][HD] column sums of this CTA's dK, dV rows
  const int h = blockIdx.x, b = blockIdx.y, key0 = blockIdx.z * QB;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t seed = p > 0.f ? (uint32_t)(*seed_ptr) : 0u;
  const float inv_keep = p > 0.f ? 1.f / (1.f - p) : 1.f;
  const T* base = qkv + h * HD;
  if (tk.slot != nullptr && b == (int)gridDim.y - 1 && key0 == 0) {
    clear_zero_rows<T>(tk, dqkv, 3 * H, H + h * HD, HD);
    clear_zero_rows<T>(tk, dqkv, 3 * H, 2 * H + h * HD, HD);
  }
  const int len = seq_len(tk, b, S), lim = (len + 15) & ~15;
  if (key0 >= len) return;
  if (bias_acc != nullptr)
    for (int i = threadIdx.x; i < 2 * HD; i += blockDim.x) sBias[i] = 0.f;
  const bool vec = (S & 7) == 0;     // then every 8-key segment starts 16-byte aligned and lies inside the row
  const int nqb = (len + KBLK - 1) / KBLK;
  float outK[HD / 8][4], outV[HD / 8][4];
#pragma unroll
  for (int jd = 0; jd < HD / 8; ++jd) {
    outK[jd][0] = 0.f; outK[jd][1] = 0.f; outK[jd][2] = 0.f; outK[jd][3] = 0.f;
    outV[jd][0] = 0.f; outV[jd][1] = 0.f; outV[jd][2] = 0.f; outV[jd][3] = 0.f;
  }
  for (int qb = 0; qb < nqb; ++qb) {
    __syncthreads();
    stage_block<T>(sQ, base, (size_t)3 * H, bqkv + h * HD, qb * KBLK, KBLK, tk, b, S, len);
    stage_block<T>(sDO, dctx + h * HD, (size_t)H, nullptr, qb * KBLK, KBLK, tk, b, S, len);
    for (int i = threadIdx.x; i < KBLK * (QB / 8); i += blockDim.x) {
      const int qr = i >> 3, kc = (i & 7) * 8;
      const int q = qb * KBLK + qr, key = key0 + kc;
      float dsv[8], wv[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) { dsv[j] = 0.f; wv[j] = 0.f; }
      // rows of tokens that do not exist were never written; keys >= lim were not written either
      if (q < len && key < lim && key < S && seq_row(tk, b, S, q) >= 0) {
        const size_t idx = ((size_t)(b * nh + h) * S + q) * S + key;
        if (vec) {
          load8(ds_ws + idx, dsv);
          load8(probs + idx, wv);
        } else {
          for (int j = 0; j < 8; ++j)
            if (key + j < S) { dsv[j] = to_f(ds_ws[idx + j]); wv[j] = to_f(probs[idx + j]); }
        }
        if (p > 0.f) {
#pragma unroll
          for (int j = 0; j < 8; ++j) wv[j] = keep(seed, stream, (uint32_t)(idx + j), p) ? wv[j] * inv_keep : 0.f;
        }
      }
      store8(sDS + qr * PPK + kc, dsv);
      store8(sW + qr * PPK + kc, wv);
    }
    __syncthreads();
    transposed_times_rows<T, KBLK>(outK, sDS, PPK, warp * 16, sQ, lane, lim - qb * KBLK);
    transposed_times_rows<T, KBLK>(outV, sW, PPK, warp * 16, sDO, lane, lim - qb * KBLK);
  }
  const int k0 = key0 + warp * 16 + (lane >> 2);
  const int row0 = k0 < len ? seq_row(tk, b, S, k0) : -1, row1 = k0 + 8 < len ? seq_row(tk, b, S, k0 + 8) : -1;
  write_rows<T>(outK, dqkv + H + h * HD, 3 * H, row0, row1, lane,
                bias_acc != nullptr ? sBias : nullptr);
  write_rows<T>(outV, dqkv + 2 * H + h * HD, 3 * H, row0, row1, lane,
                bias_acc != nullptr ? sBias + HD : nullptr);
  if (bias_acc != nullptr) {
    __syncthreads();
    const int cta = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    float* my_acc = bias_acc + (size_t)(cta % 8) * 3 * H;
    for (int i = threadIdx.x; i < 2 * HD; i += blockDim.x)
      atomicAdd(my_acc + (1 + i / HD) * H + h * HD + (i % HD), sBias[i]);
  }
}

constexpr size_t fwd_long_smem(size_t esz) { return (size_t)(QB + 2 * KBLK) * RP * esz + KBLK; }
constexpr size_t dq_long_smem(size_t esz) { return (size_t)(QB + 2 * KBLK) * RP * esz + HD * sizeof(float); }
constexpr size_t dkv_long_smem(size_t esz) {
  return (size_t)2 * KBLK * PPK * esz + (size_t)2 * KBLK * RP * esz + 2 * HD * sizeof(float);
}

template <typename T>
static int launch_fwd_long(const void* qkv, const void* bqkv, const int* mask, void* ctx, void* probs, int b, int S, int H,
                           int nh, float p, const int* seed, unsigned stream_id, const Tok& tk, cudaStream_t st) {
  auto k = attention_fwd_long_kernel<T>;
  constexpr size_t smem = fwd_long_smem(sizeof(T));
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -5;
  k<<<dim3(nh, b, (S + QB - 1) / QB), 128, smem, st>>>((const T*)qkv, (const T*)bqkv, mask, (T*)ctx, (T*)probs, S, H, nh, p,
                                                        seed, stream_id, tk);
  return 0;
}

template <typename T>
static int launch_bwd_long(const void* dctx, const void* qkv, const void* bqkv, const void* probs, void* ds_ws, void* dqkv,
                           int b, int S, int H, int nh, float p, const int* seed, unsigned stream_id, float* bias_acc,
                           const Tok& tk, cudaStream_t st) {
  auto kq = attention_bwd_long_dq_kernel<T>;
  auto kkv = attention_bwd_long_dkv_kernel<T>;
  constexpr size_t sq = dq_long_smem(sizeof(T)), skv = dkv_long_smem(sizeof(T));
  if (cudaFuncSetAttribute(kq, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sq) != cudaSuccess) return -5;
  if (cudaFuncSetAttribute(kkv, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)skv) != cudaSuccess) return -5;
  const dim3 grid(nh, b, (S + QB - 1) / QB);
  kq<<<grid, 128, sq, st>>>((const T*)dctx, (const T*)qkv, (const T*)bqkv, (const T*)probs, (T*)ds_ws, (T*)dqkv, S, H, nh, p,
                            seed, stream_id, bias_acc, tk);
  kkv<<<grid, 128, skv, st>>>((const T*)dctx, (const T*)qkv, (const T*)bqkv, (const T*)probs, (const T*)ds_ws, (T*)dqkv, S,
                              H, nh, p, seed, stream_id, bias_acc, tk);
  return 0;
}

}  // namespace amma
}  // namespace rb

using namespace rb;

// dtype: 1 = bf16, 2 = fp16.  Requires H / nh == 64 or 32, H % 8 == 0, 1 <= S <= 256 (head dim 32: <= 128); returns -4
// otherwise.  tok_slot / tok_len / tok_meta (all or none): packed tokens, see token_map.cuh.
static bool mma_args_ok(int dtype, int b, int S, int H, int nh) {
  if (S < 1 || S > 256 || H % nh || H % 8 || (dtype != RB_BF16 && dtype != RB_F16)) return false;
  if (H / nh != 64 && !(H / nh == 32 && S <= 128)) return false;
  return S <= 128 || (long long)b * nh * S * S < (1LL << 32);   // dropout counters are 32-bit element indices
}

static int attention_fwd_any(int dtype, const void* qkv, const void* bqkv, const int* mask, void* ctx, void* probs,
                             int b, int S, int H, int nh, float p, const int* seed, unsigned stream_id,
                             const int* tok_slot, const int* tok_len, const int* tok_meta, const void* first_src,
                             void* first_dst, cudaStream_t st) {
  if (!mma_args_ok(dtype, b, S, H, nh)) return -4;
  const amma::Tok tk{tok_slot, tok_len, tok_meta};
  const bool packed = tok_slot != nullptr;
  int rc;
#define RB_FWD(T, HD) RB_ATT_LAUNCH(T, HD, amma::launch_fwd, S, packed, qkv, bqkv, mask, ctx, probs, b, S, H, nh, p, seed, stream_id, tk, first_src, first_dst)
  if (H / nh == 64) rc = dtype == RB_BF16 ? RB_FWD(__nv_bfloat16, 64) : RB_FWD(__half, 64);
  else rc = dtype == RB_BF16 ? RB_FWD(__nv_bfloat16, 32) : RB_FWD(__half, 32);
#undef RB_FWD
  if (rc) return rc;
  RB_LAUNCH_CHECK();
  return 0;
}

RB_API int rb_attention_fwd_mma(int dtype, const void* qkv, const void* bqkv, const int* mask, void* ctx, void* probs,
                                int b, int S, int H, int nh, float p, const int* seed, unsigned stream_id,
                                const int* tok_slot, const int* tok_len, const int* tok_meta, cudaStream_t st) {
  return attention_fwd_any(dtype, qkv, bqkv, mask, ctx, probs, b, S, H, nh, p, seed, stream_id, tok_slot, tok_len, tok_meta,
                           nullptr, nullptr, st);
}

// First-token variant, packed rows only: ctx is [b, H], and first_dst [b, H] receives the first tokens' rows of first_src.
RB_API int rb_attention_fwd_first(int dtype, const void* qkv, const void* bqkv, const int* mask, void* ctx, void* probs,
                                  int b, int S, int H, int nh, float p, const int* seed, unsigned stream_id,
                                  const int* tok_slot, const int* tok_len, const int* tok_meta, const void* first_src,
                                  void* first_dst, cudaStream_t st) {
  if (tok_slot == nullptr || first_src == nullptr || first_dst == nullptr) return -3;
  return attention_fwd_any(dtype, qkv, bqkv, mask, ctx, probs, b, S, H, nh, p, seed, stream_id, tok_slot, tok_len, tok_meta,
                           first_src, first_dst, st);
}

// bias_acc (nullable): 8 replicas x [3H] fp32; when given, the column sums of dqkv (the q/k/v bias gradients) are
// accumulated there so that no separate pass over dqkv is needed.
static int attention_bwd_any(int dtype, const void* dctx, const void* qkv, const void* bqkv, const void* probs,
                             void* dqkv, int b, int S, int H, int nh, float p, const int* seed, unsigned stream_id,
                             float* bias_acc, const int* tok_slot, const int* tok_len, const int* tok_meta,
                             const void* first_src, void* first_dst, cudaStream_t st) {
  if (!mma_args_ok(dtype, b, S, H, nh)) return -4;
  const amma::Tok tk{tok_slot, tok_len, tok_meta};
  const bool packed = tok_slot != nullptr;
  int rc;
#define RB_BWD(T, HD) RB_ATT_LAUNCH(T, HD, amma::launch_bwd, S, packed, dctx, qkv, bqkv, probs, dqkv, b, S, H, nh, p, seed, stream_id, bias_acc, tk, first_src, first_dst)
  if (H / nh == 64) rc = dtype == RB_BF16 ? RB_BWD(__nv_bfloat16, 64) : RB_BWD(__half, 64);
  else rc = dtype == RB_BF16 ? RB_BWD(__nv_bfloat16, 32) : RB_BWD(__half, 32);
#undef RB_BWD
  if (rc) return rc;
  RB_LAUNCH_CHECK();
  return 0;
}

RB_API int rb_attention_bwd_mma(int dtype, const void* dctx, const void* qkv, const void* bqkv, const void* probs,
                                void* dqkv, int b, int S, int H, int nh, float p, const int* seed, unsigned stream_id,
                                float* bias_acc, const int* tok_slot, const int* tok_len, const int* tok_meta,
                                cudaStream_t st) {
  return attention_bwd_any(dtype, dctx, qkv, bqkv, probs, dqkv, b, S, H, nh, p, seed, stream_id, bias_acc, tok_slot, tok_len,
                           tok_meta, nullptr, nullptr, st);
}

// First-token variant, packed rows only: dctx is [b, H]; the packed rows of first_dst receive the rows of first_src [b, H] at
// the first tokens and zeros elsewhere.
RB_API int rb_attention_bwd_first(int dtype, const void* dctx, const void* qkv, const void* bqkv, const void* probs,
                                  void* dqkv, int b, int S, int H, int nh, float p, const int* seed, unsigned stream_id,
                                  float* bias_acc, const int* tok_slot, const int* tok_len, const int* tok_meta,
                                  const void* first_src, void* first_dst, cudaStream_t st) {
  if (tok_slot == nullptr || first_src == nullptr || first_dst == nullptr) return -3;
  return attention_bwd_any(dtype, dctx, qkv, bqkv, probs, dqkv, b, S, H, nh, p, seed, stream_id, bias_acc, tok_slot, tok_len,
                           tok_meta, first_src, first_dst, st);
}

// Sequences of 257..512 tokens, head dim 64 (same requirements otherwise).  The backward needs ds_ws, a [b, nh, S, S]
// scratch of the activation dtype (the softmax gradient, written by its first kernel and read by its second); two launches.
static bool long_args_ok(int dtype, int b, int S, int H, int nh) {
  if (S <= 128 || S > 512 || H % nh || H % 8 || H / nh != amma::HD || (dtype != RB_BF16 && dtype != RB_F16)) return false;
  return (long long)b * nh * S * S < (1LL << 32);   // dropout counters are 32-bit element indices
}

RB_API int rb_attention_fwd_long(int dtype, const void* qkv, const void* bqkv, const int* mask, void* ctx, void* probs,
                                 int b, int S, int H, int nh, float p, const int* seed, unsigned stream_id,
                                 const int* tok_slot, const int* tok_len, const int* tok_meta, cudaStream_t st) {
  if (!long_args_ok(dtype, b, S, H, nh)) return -4;
  const amma::Tok tk{tok_slot, tok_len, tok_meta};
  const int rc = dtype == RB_BF16
                     ? amma::launch_fwd_long<__nv_bfloat16>(qkv, bqkv, mask, ctx, probs, b, S, H, nh, p, seed, stream_id, tk, st)
                     : amma::launch_fwd_long<__half>(qkv, bqkv, mask, ctx, probs, b, S, H, nh, p, seed, stream_id, tk, st);
  if (rc) return rc;
  RB_LAUNCH_CHECK();
  return 0;
}

RB_API int rb_attention_bwd_long(int dtype, const void* dctx, const void* qkv, const void* bqkv, const void* probs,
                                 void* ds_ws, void* dqkv, int b, int S, int H, int nh, float p, const int* seed,
                                 unsigned stream_id, float* bias_acc, const int* tok_slot, const int* tok_len, const int* tok_meta,
                                cudaStream_t st) {
  if (!long_args_ok(dtype, b, S, H, nh) || ds_ws == nullptr) return -4;
  const amma::Tok tk{tok_slot, tok_len, tok_meta};
  const int rc = dtype == RB_BF16
                     ? amma::launch_bwd_long<__nv_bfloat16>(dctx, qkv, bqkv, probs, ds_ws, dqkv, b, S, H, nh, p, seed,
                                                            stream_id, bias_acc, tk, st)
                     : amma::launch_bwd_long<__half>(dctx, qkv, bqkv, probs, ds_ws, dqkv, b, S, H, nh, p, seed, stream_id,
                                                     bias_acc, tk, st);
  if (rc) return rc;
  RB_LAUNCH_CHECK();
  return 0;
}
