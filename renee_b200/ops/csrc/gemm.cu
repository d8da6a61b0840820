// GEMMs for sm_100a: one persistent tcgen05 / TMEM kernel family with the element-wise neighbours of every linear
// layer of the encoder, and the three products of the classifier step, fused into the epilogue.  They stand in for the cuBLAS calls behind the reference's HF
// nn.Linear layers and its FP32Linear (main.py:126-129, dl_base.py:104-111) and for the ATen kernels around
// them (bias add, GELU, dropout, residual add, GELU backward, bias-gradient column sums).
//
//   layout NT  C[M,N] = A[M,K] · B[N,K]^T   forward   (activations x weight^T)       A, B K-major
//   layout NN  C[M,N] = A[M,K] · B[K,N]     dgrad     (output gradient x weight)     A K-major, B MN-major
//   layout TN  C[M,N] = A[K,M]^T · B[K,N]   wgrad     (output gradient^T x input)    A, B MN-major, split-K
//
//   epilogues  STORE                C = acc
//              BIAS_GELU            F = acc + bias ;  C = gelu(F)                    (FFN-1 forward; F kept for backward)
//              BIAS_DROPOUT_RESID   C = R + dropout(acc + bias)                      (out-proj / FFN-2 forward: the LayerNorm input)
//              ADD                  C = acc + R                                      (dgrad joined with the residual gradient)
//              GELU_BWD             C = acc * gelu'(R) ;  column sums of C -> bias gradient accumulators
//              SPLITK               fp32 partials reduced in L2, the last CTA of a tile converts and stores
//              SIGMOID_POS          C = sigmoid(acc) - Y: the classifier's logit gradient; Y from a label-sorted list of
//                                   positives applied to the staged tile in shared memory before it is stored; on
//                                   loss-sampling steps also the sum of softplus(acc) (parity: dl_base.py:572-594)
//              DX                   dX += scale * acc by vector reductions into an fp32 matrix (contraction over the
//                                   labels of a chunk, split over the CTAs); the last CTA raises the peers' flags
//              DW_SGD               classifier weights: W and momentum tiles [128 x 64] come in by TMA under the main loop,
//                                   m = mo m + (acc + wd w), w -= lr m (stochastic rounding optional) in shared memory,
//                                   both tiles leave by TMA; dW = Gt X is never stored (parity: dl_base.py:623-633, 343-344)
//              TOPK                 nothing is stored: every epilogue thread keeps the 8 largest entries of its row
//                                   over all the tiles its CTA visits and writes them as candidates at the end; topk.cu
//                                   reduces the candidates to the k best and recomputes the labels of a thread that
//                                   may have dropped one (prediction: X W^T is never materialised; parity:
//                                   dl_base.py:745-756)
//
// Structure.  Persistent CTAs walk the work items (tile x K-split).  576 threads: warp 0 TMA producer, warp 1
// TMEM owner + MMA issuer, warps 2..17 epilogue (four groups of four warps, one TMEM lane quarter per warp, one
// 64-column panel of the tile per group).  The shared-memory ring keeps streaming across item boundaries and TMEM
// holds two accumulators, so the epilogue of item i runs under the main loop of item i + 1.
//
// Two tile shapes.  NCTA = 1: a CTA owns a 128 x BN tile.  NCTA = 2 (`cta_group::2`): the two CTAs of a cluster
// of two own a 256 x BN tile; each loads its 128 rows of A and HALF of the B columns, the leader CTA issues
// MMAs that read both CTAs' shared memory and write 128 accumulator rows into each CTA's TMEM.  For the same MMA
// work the pair fetches and keeps 128 + BN/2 rows per k block and CTA instead of 128 + BN.  Loads are plain TMA tile
// loads (no multicast); a pair's loads count their bytes on the leader's barrier and one `tcgen05.commit` arrives on
// both CTAs' barriers.  (8192 x 768 x 2304, plain store: tensor pipe 49 % busy over the whole launch, L2 31 %, DRAM 7 %.)
//
// Epilogue.  Output tiles are staged in 128-byte-swizzled shared-memory panels ([128 rows x 64 columns] of 16-bit
// elements) and written with TMA stores, which clip at the matrix edge; tile-shaped inputs (residual, stored
// pre-activation) are fetched into the same panels by TMA while the tile's main loop still runs and are updated
// in place.  Every global access of the epilogue is therefore a full-line bulk copy.
// A warp owns 32 rows of its group's panel: it fetches, stages and stores them by itself and waits for no other warp.
// What does not need the accumulator -- the dropout hashes, the bias, the residual's way to registers, the positives of the
// tile's labels -- is done while the main loop runs; the accumulator comes in fragments of 8 columns, the next one on its way.
// (With panels shared by four warps, a barrier of all sixteen per tile and these loads behind the accumulator, 4928 tokens:
// FFN1 bias + GELU 31.8 -> 28.1 us, FFN2 dgrad + GELU backward 33.5 -> 28.5, FFN2 forward + dropout + residual 25.4 -> 21.3,
// output projection 14.3 -> 11.1; plain products of these shapes take 20.8, 20.8, 19.9 and 9.0.)  What is left of an epilogue
// in a multi-round launch is shared-memory bandwidth: a 256 x 256 pair tile of K = 768 moves 48 KB per k block and CTA through
// it for the MMAs and 32 KB for the loads, and two 16-bit outputs another 256 KB.
//
// Every wait is bounded (tc.cuh): a protocol error ends with a status word, never with a hang.  Barriers without a time limit
// are only met by warps that all come to them whatever their bounded waits said.
#include <type_traits>
#include "peer.cuh"
#include "token_map.cuh"
#include "topk.cuh"

namespace rb {
namespace eg {

constexpr int BM = 128;                         // accumulator rows per CTA
constexpr int BK = 64;
constexpr int A_BYTES = BM * BK * 2;            // 16 KB
constexpr int PANEL_BYTES = BM * 64 * 2;        // one staging panel: 128 rows x 64 x 16 bit
constexpr int SUB_ROWS = 32;                    // a warp's rows of it: it stages, stores and fetches them by itself
constexpr int SUB_BYTES = SUB_ROWS * 64 * 2;
constexpr int EGROUPS = 4;                      // epilogue groups of four warps (one per TMEM lane quarter)
constexpr int N_PANELS = EGROUPS;               // one staging panel per epilogue group
constexpr int EPI_WARPS = 4 * EGROUPS;
constexpr int EPI_THREADS = 32 * EPI_WARPS;
constexpr int THREADS = 64 + EPI_THREADS;       // producer warp, MMA warp, sixteen epilogue warps
constexpr int ACC_BUFS = 2;
constexpr int ACC_STRIDE = 256;                 // TMEM columns between the two accumulators
constexpr int TMEM_COLS = ACC_BUFS * ACC_STRIDE;

// Shared memory: the operand ring plus, for epilogues that stage tiles, one panel per epilogue group.  Bytes in flight
// cover the loads' latency, so the ring takes everything else (192 KB).
constexpr int RING_BYTES = 192 * 1024;          // operand bytes in flight per CTA
constexpr int MAX_STAGES = 8;                   // a stage is 16 KB of A + BN / NCTA rows of B: 24 KB (8 stages) .. 48 KB (4)

enum Layout : int { L_NT = 0, L_NN = 1, L_TN = 2 };
enum Epi : int { E_STORE = 0, E_BIAS_GELU = 1, E_BIAS_DROPOUT_RESID = 2, E_ADD = 3, E_GELU_BWD = 4, E_SPLITK = 5, E_TOPK = 6, E_SIGMOID_POS = 7, E_DX = 8, E_DW_SGD = 9 };

// DW_SGD updates two tile-shaped tensors in place (weights and momentum): two panels per group, a 160 KB ring.
constexpr int SMEM_BUDGET = 224 * 1024;         // ring + panels
constexpr bool staged_epi(int epi) { return epi != E_SPLITK && epi != E_TOPK && epi != E_DX; }
constexpr int panel_count(int epi) { return !staged_epi(epi) ? 0 : (epi == E_DW_SGD ? 2 * N_PANELS : N_PANELS); }
constexpr int ring_bytes(int epi) {
  return SMEM_BUDGET - panel_count(epi) * PANEL_BYTES < RING_BYTES ? SMEM_BUDGET - panel_count(epi) * PANEL_BYTES : RING_BYTES;
}
template <int EPI> struct Cfg {
  static constexpr bool kStaged = staged_epi(EPI);
  static constexpr int kPanels = panel_count(EPI);
  static constexpr int kRing = ring_bytes(EPI);
  static constexpr int kSmem = kRing + kPanels * PANEL_BYTES + 1024 + 512;   // alignment, barriers
};

struct Params {
  int M, N;                      // output rows / columns
  int BN;                        // N tile: 64, 128 or 256 (NCTA = 2: 128 or 256)
  int n_m_tiles, n_n_tiles;      // tiles of (128 NCTA) x BN
  int splits, kb_total, kb_per_split;
  void* C; int ldc;              // direct stores of the split-K fix-up only
  const void* bias;              // [N]                             BIAS_GELU, BIAS_DROPOUT_RESID
  float p; const int* seed; uint32_t stream;        // dropout      BIAS_DROPOUT_RESID
  float* colacc; int col_tot; int col_off;          // GELU_BWD: replicas of [col_tot] floats, this vector at col_off
  float* sk_scratch; unsigned* sk_counters;         // SPLITK: [tiles][128 NCTA x BN] fp32 (zero between launches), [tiles]
  float* cand_val; int* cand_idx; int cand_ld;      // TOPK: [M, cand_ld] candidates, 8 per (unit, epilogue group)
  // SIGMOID_POS (classifier logits + gradient): label-sorted positives, label id of row 0, all-gather flags to wait for
  const int* pos_rows; const int* pos_labels; const int* nnz_ptr; int label0;
  const uint32_t* wait_flags; int wait_n; const uint32_t* step_ptr;
  float* loss_acc;               // SIGMOID_POS, loss-sampling steps: += sum of softplus(z) over the valid logits
  // DX (classifier input gradient): fp32 accumulation target, loss scale, completion signal to the peers
  float* dX; int ldX; const float* hp;
  unsigned* done_counter; void* peer_flags[16]; int n_peers; int flag_index;
  // DW_SGD (classifier weights): momentum, weight decay, rounding mode; the row stride numbers the elements for the
  // rounding hash; the learning rate and the seed come from hp
  float mo, wd; int stochastic_round; int ldW;
  // Packed tokens (token_map.cuh): M (layouts NT, NN) or K (TN) counts token rows, and the number that exists is only
  // known on the device; tok numbers the dropout counters of packed rows
  const int* tok_meta; const int* tok;
  int* status;
};

constexpr int kColReplicas = 8;   // must equal the replica count of the deferred column reductions (encoder_ops.cu)

template <typename T> __device__ __forceinline__ uint4 pack8(const float* v) { return pack16x8<T>(v); }
template <typename T> __device__ __forceinline__ void unpack8(const uint4& raw, float* out) {
  const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
  for (int i = 0; i < 8; ++i) out[i] = to_f(e[i]);
}

// The n staging warps of a row quarter come together (barrier 1 is that of all epilogue warps).
__device__ __forceinline__ void meet_rows(int quarter, int n) {
  asm volatile("bar.sync %0, %1;" ::"r"(2 + quarter), "r"(32 * n) : "memory");
}

// First positions of the sorted a[0 .. n) whose values are >= k_lo and >= k_hi, by one warp: each half-warp probes 16 places
// per step, so ten thousand entries take 4 dependent loads where two binary searches in a row took 28.
__device__ __forceinline__ void warp_bounds(const int* __restrict__ a, int n, int k_lo, int k_hi, int lane, int& lo, int& hi) {
  const int i = lane & 15, key = lane < 16 ? k_lo : k_hi;
  int l = 0, h = n;
  while (__any_sync(0xffffffffu, l < h)) {
    const int len = h - l;
    const bool less = len > 0 && a[l + (int)((long long)len * (i + 1) / 17)] < key;
    const int c = __popc((__ballot_sync(0xffffffffu, less) >> (lane & 16)) & 0xffffu);      // the probes ascend
    const int nl = c > 0 ? l + (int)((long long)len * c / 17) + 1 : l;
    const int nh = c < 16 ? l + (int)((long long)len * (c + 1) / 17) : h;
    if (len > 0) { l = nl; h = nh; }
  }
  lo = __shfl_sync(0xffffffffu, l, 0);
  hi = __shfl_sync(0xffffffffu, l, 16);
}

// sigmoids of 8 logits with one reciprocal per pair: 1 / a = b / (a b).  Below -40 the result is 0 in 16 bits either way, and
// the bound keeps the product of two denominators finite.  A NaN stays one and does not reach its neighbour, whose logit
// belongs to another row of the batch: one test of the 8 (a test per pair cost 18 % of the kernel at 64-deep products).
__device__ __forceinline__ void sigmoid8(const float* z, float* s) {
  float den[8], pair[4];
#pragma unroll
  for (int j = 0; j < 8; ++j) den[j] = 1.f + __expf(-max_nan(z[j], -40.f));
#pragma unroll
  for (int j = 0; j < 4; ++j) pair[j] = den[2 * j] * den[2 * j + 1];
  const float any = (pair[0] + pair[1]) + (pair[2] + pair[3]);
  if (any != any) {
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] = 1.f / den[j];
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float r = 1.f / pair[j];
      s[2 * j] = r * den[2 * j + 1];
      s[2 * j + 1] = r * den[2 * j];
    }
  }
}

// Byte offset of the 16-byte chunk `chunk` (8 columns) of row r inside a 128-byte-swizzled panel.
__device__ __forceinline__ uint32_t panel_off(int r, int chunk) { return (uint32_t)r * 128u + (uint32_t)((chunk ^ (r & 7)) << 4); }

// (M tile, N tile) of an item's tile.  TOPK walks two M tiles side by side: the units of even number take one, the
// others the other, so that the (much larger) N operand is read from HBM once per pair of M tiles instead of once per M
// tile, and a unit still stays with one M tile until its N tiles are done (topk.cuh has the same numbering).
template <int EPI> __device__ __forceinline__ void tile_coords(int tile, int n_m, int n_n, int& mt, int& nt) {
  if (EPI == E_TOPK) topk_tile(tile, n_m, n_n, mt, nt);
  else { mt = tile / n_n; nt = tile - mt * n_n; }
}

template <typename T, int LAYOUT, int EPI, int NCTA>
__global__ void __launch_bounds__(THREADS, 1)
enc_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmR,
                const __grid_constant__ CUtensorMap tmF, const Params p) {
  using C_ = Cfg<EPI>;
  constexpr int RING = C_::kRing;
  constexpr bool A_MN = (LAYOUT == L_TN);
  constexpr bool B_MN = (LAYOUT != L_NT);
  constexpr int FMT = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
  constexpr bool HAS_IN = (EPI == E_BIAS_DROPOUT_RESID || EPI == E_ADD || EPI == E_GELU_BWD || EPI == E_DW_SGD);   // tile-shaped input R
  constexpr bool STAGED = C_::kStaged;                                                           // outputs through panels
  constexpr bool HELD_IN = HAS_IN && EPI != E_DW_SGD;      // ... of one tensor: read into registers under the main loop
  constexpr uint32_t IN_BYTES = EPI == E_DW_SGD ? 2 * SUB_BYTES : SUB_BYTES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* panels = smem + RING;                           // [N_PANELS][PANEL_BYTES], 1024-byte aligned
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(panels + C_::kPanels * PANEL_BYTES);
  uint64_t* empty_bar = full_bar + MAX_STAGES;
  uint64_t* tmem_full_bar = empty_bar + MAX_STAGES;      // [ACC_BUFS]
  uint64_t* tmem_empty_bar = tmem_full_bar + ACC_BUFS;   // [ACC_BUFS]  (used in the leader CTA)
  uint64_t* in_bar = tmem_empty_bar + ACC_BUFS;          // [EPI_WARPS]  a warp's part of the R panel has landed
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(in_bar + EPI_WARPS);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);
  volatile int* s_last = s_abort + 1;

  const int warp = tc::warp_id();
  const int lane = threadIdx.x & 31;
  const uint32_t rank = NCTA == 2 ? tc::cluster_ctarank() : 0u;
  const int unit = NCTA == 2 ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;          // which persistent worker
  const int n_units = NCTA == 2 ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const int b_rows = p.BN / NCTA;                                                 // B rows (N index) this CTA loads
  const int STAGE = A_BYTES + b_rows * BK * 2;                                    // 24, 32 or 48 KB
  const int STAGES = min(MAX_STAGES, RING / STAGE);
  const uint32_t stage_tx = (uint32_t)NCTA * (uint32_t)STAGE;

  if (threadIdx.x == 0) {
    tc::prefetch_tmap(&tmA);
    tc::prefetch_tmap(&tmB);
    if (STAGED) tc::prefetch_tmap(&tmC);
    if (HAS_IN) tc::prefetch_tmap(&tmR);
    if (EPI == E_BIAS_GELU || EPI == E_DW_SGD) tc::prefetch_tmap(&tmF);
    for (int s = 0; s < MAX_STAGES; ++s) { tc::mbar_init(full_bar + s, 1); tc::mbar_init(empty_bar + s, 1); }
    for (int a = 0; a < ACC_BUFS; ++a) { tc::mbar_init(tmem_full_bar + a, 1); tc::mbar_init(tmem_empty_bar + a, 4 * EGROUPS * NCTA); }
    for (int a = 0; a < EPI_WARPS; ++a) tc::mbar_init(in_bar + a, 1);
    *s_abort = 0;
    *s_last = 0;
    tc::fence_barrier_init();
  }
  if (warp == 1) {
    if (NCTA == 2) tc::tmem_alloc_pair(tmem_ptr_smem, TMEM_COLS); else tc::tmem_alloc(tmem_ptr_smem, TMEM_COLS);
  }
  tc::tc_fence_before();
  __syncthreads();
  if (NCTA == 2) tc::cluster_sync_all();            // the peer's barriers exist before anything arrives on them
  tc::tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  bool aborted = false;
  // everything above touched no global memory: it may have run under the tail of the previous kernel
  grid_dep_wait();
  grid_dep_launch();
  // extents of this launch: the host's, or with packed tokens the device's row count (every thread reads the same word)
  const int kb_total = p.kb_total, kb_per_split = p.kb_per_split, splits = p.splits;
  int M = p.M, n_m_tiles = p.n_m_tiles;
  if (LAYOUT != L_TN && p.tok_meta != nullptr) {
    M = __ldcg(p.tok_meta + TOK_ROWS);
    n_m_tiles = (M + BM * NCTA - 1) / (BM * NCTA);
  }
  const int n_items = n_m_tiles * p.n_n_tiles * splits;
  // items of this unit: every n_units-th, or for the logits (few N tiles per M tile) a run of neighbours, so that the
  // positives of an M tile are looked up once
  constexpr bool RUNS = EPI == E_SIGMOID_POS;
  const int per_unit = (n_items + n_units - 1) / n_units;
  const int it0 = RUNS ? unit * per_unit : unit, it1 = RUNS ? min(n_items, it0 + per_unit) : n_items, its = RUNS ? 1 : n_units;

  if (warp == 0 && tc::elect_one()) {
    // ---------------- TMA producer: one continuous stream of (item, k block) stages
    int s = 0;
    uint32_t ph = 0;
    if (EPI == E_SIGMOID_POS && p.wait_flags != nullptr) {
      // all-gather prologue: every rank has pushed its rows of X into this GPU's buffer and raised its flag; the
      // loads below go through the async proxy, hence the proxy fence after the acquire
      const uint32_t want = *p.step_ptr;
      for (int q = 0; q < p.wait_n; ++q)
        if (!wait_flag(p.wait_flags + q, want, p.status, 100 + q)) aborted = true;
      asm volatile("fence.proxy.async;" ::: "memory");
    }
    for (int item = it0; item < it1 && !aborted; item += its) {
      const int tile = item / splits, split = item - tile * splits;
      int mt, nt;
      tile_coords<EPI>(tile, n_m_tiles, p.n_n_tiles, mt, nt);
      const int m0 = mt * (BM * NCTA) + (int)rank * BM;
      const int n0 = nt * p.BN + (int)rank * b_rows;
      const int kb0 = split * kb_per_split, kb1 = min(kb_total, kb0 + kb_per_split);
      for (int kb = kb0; kb < kb1; ++kb, s = (s + 1 == STAGES ? 0 : s + 1), ph ^= (s == 0 ? 1u : 0u)) {
        if (!tc::mbar_wait(empty_bar + s, ph ^ 1, aborted, p.status, tc::SITE_EMPTY, kb)) break;
        uint8_t* sA = smem + s * STAGE;
        uint8_t* sB = sA + A_BYTES;
        if (NCTA == 1) {
          tc::mbar_expect_tx(full_bar + s, stage_tx);
          if (A_MN) {
            tc::tma_load_2d(sA, &tmA, full_bar + s, m0, kb * BK);
            tc::tma_load_2d(sA + 8192, &tmA, full_bar + s, m0 + 64, kb * BK);
          } else {
            tc::tma_load_2d(sA, &tmA, full_bar + s, kb * BK, m0);
          }
          if (B_MN) {
            for (int i = 0; i < b_rows / 64; ++i) tc::tma_load_2d(sB + i * 8192, &tmB, full_bar + s, n0 + 64 * i, kb * BK);
          } else {
            tc::tma_load_2d(sB, &tmB, full_bar + s, kb * BK, n0);
          }
        } else {
          // the leader's barrier counts the bytes of both CTAs' loads; only the leader announces them
          const uint32_t lbar = tc::leader_addr(tc::smem_u32(full_bar + s));
          if (rank == 0) tc::mbar_expect_tx(full_bar + s, stage_tx);
          if (A_MN) {
            tc::tma_load_2d_pair(sA, &tmA, lbar, m0, kb * BK);
            tc::tma_load_2d_pair(sA + 8192, &tmA, lbar, m0 + 64, kb * BK);
          } else {
            tc::tma_load_2d_pair(sA, &tmA, lbar, kb * BK, m0);
          }
          if (B_MN) {
            for (int i = 0; i < b_rows / 64; ++i) tc::tma_load_2d_pair(sB + i * 8192, &tmB, lbar, n0 + 64 * i, kb * BK);
          } else {
            tc::tma_load_2d_pair(sB, &tmB, lbar, kb * BK, n0);
          }
        }
      }
    }
  } else if (warp == 1 && rank == 0 && tc::elect_one()) {
    // ---------------- MMA issuer (leader CTA): accumulator (t_local & 1), reused once the epilogue(s) drained it
    const uint32_t idesc = tc::make_idesc(FMT, A_MN ? 1 : 0, B_MN ? 1 : 0, BM * NCTA, p.BN);
    int s = 0, t_local = 0;
    uint32_t ph = 0;
    for (int item = it0; item < it1 && !aborted; item += its, ++t_local) {
      const int tile = item / splits, split = item - tile * splits;
      const int kb0 = split * kb_per_split, kb1 = min(kb_total, kb0 + kb_per_split);
      const int buf = t_local & 1;
      const uint32_t use = (uint32_t)(t_local >> 1);
      if (!tc::mbar_wait(tmem_empty_bar + buf, (use & 1) ^ 1, aborted, p.status, tc::SITE_TMEM_EMPTY, item)) break;
      tc::tc_fence_after();
      const uint32_t d_tmem = tmem_base + (uint32_t)buf * ACC_STRIDE;
      for (int kb = kb0; kb < kb1; ++kb, s = (s + 1 == STAGES ? 0 : s + 1), ph ^= (s == 0 ? 1u : 0u)) {
        if (!tc::mbar_wait(full_bar + s, ph, aborted, p.status, tc::SITE_FULL, kb)) break;
        tc::tc_fence_after();
        const uint32_t sA = tc::smem_u32(smem + s * STAGE);
        const uint32_t sB = sA + A_BYTES;
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) {
          const uint64_t ad = A_MN ? tc::make_smem_desc(sA + k * 2048, 8192, 1024) : tc::make_smem_desc(sA + k * 32, 16, 1024);
          const uint64_t bd = B_MN ? tc::make_smem_desc(sB + k * 2048, 8192, 1024) : tc::make_smem_desc(sB + k * 32, 16, 1024);
          if (NCTA == 2) tc::umma_f16_pair(d_tmem, ad, bd, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
          else tc::umma_f16(d_tmem, ad, bd, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
        }
        if (NCTA == 2) tc::umma_commit_pair(empty_bar + s); else tc::umma_commit(empty_bar + s);
      }
      if (aborted) break;
      if (NCTA == 2) tc::umma_commit_pair(tmem_full_bar + buf); else tc::umma_commit(tmem_full_bar + buf);
    }
  } else if (warp >= 2) {
    // ---------------- epilogue: group g = (warp - 2) / 4 owns columns [64 g, 64 g + 64) of the CTA's 128 rows
    const int quarter = warp & 3;
    const int g = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;                    // row of the CTA's accumulator = TMEM lane
    // staged epilogues: group g takes the 64-column panel g of the tile (BN / 64 groups have one, the others idle);
    // the others split the tile's columns into BN / EGROUPS (at least 32) per group
    const bool staging = STAGED && g < (p.BN >> 6);
    const int g_col = g * 64;
    const int ucols = p.BN / EGROUPS < 32 ? 32 : p.BN / EGROUPS;
    const bool u_active = g * ucols < p.BN;
    uint8_t* pan = panels + g * PANEL_BYTES + quarter * SUB_BYTES;              // this warp's 32 rows of the staging panel
    uint8_t* pan2 = panels + (N_PANELS + g) * PANEL_BYTES + quarter * SUB_BYTES;   // DW_SGD: the momentum beside the weights
    uint64_t* my_in_bar = in_bar + (warp - 2);
    uint32_t seed = 0u;
    float inv_keep = 1.f;
    if (EPI == E_BIAS_DROPOUT_RESID && p.p > 0.f) { seed = (uint32_t)(*p.seed); inv_keep = 1.f / (1.f - p.p); }
    int t_local = 0;
    uint32_t in_count = 0;                                // R panels fetched so far (parity of my_in_bar)
    // TOPK: this thread's 8 best (value, column) of its row so far, sorted descending; cur_m = row block they belong to
    float tv[8] = {};
    int ti[8] = {};
    int cur_m = -1;
    const auto topk_flush = [&]() {                       // the list of this unit and column group for row block cur_m
      const int frow = cur_m * (BM * NCTA) + (int)rank * BM + r;
      if (cur_m < 0 || frow >= M || !u_active) return;
      const size_t at = (size_t)frow * p.cand_ld + (size_t)(unit * EGROUPS + g) * 8;
      float4* cv = reinterpret_cast<float4*>(p.cand_val + at);
      int4* ci = reinterpret_cast<int4*>(p.cand_idx + at);
      cv[0] = make_float4(tv[0], tv[1], tv[2], tv[3]); cv[1] = make_float4(tv[4], tv[5], tv[6], tv[7]);
      ci[0] = make_int4(ti[0], ti[1], ti[2], ti[3]); ci[1] = make_int4(ti[4], ti[5], ti[6], ti[7]);
    };
    // SIGMOID_POS: the positives of this warp's 32 labels of M tile pos_m are, of a window of 32 entries of the label-sorted
    // list that the lanes hold, those in range, and entries pos_more .. pos_end behind it
    int pos_m = -1, pos_l = -1, pos_c = 0, pos_more = 0, pos_end = 0;
    float loss = 0.f;                                     // SIGMOID_POS: this thread's share of sum softplus(z)
    for (int item = it0; item < it1; item += its, ++t_local) {
      const int tile = item / splits;
      int mt, nt;
      tile_coords<EPI>(tile, n_m_tiles, p.n_n_tiles, mt, nt);
      if (EPI == E_TOPK && mt != cur_m) {
        topk_flush();
        __syncwarp();                                      // lanes of rows past M return early
#pragma unroll
        for (int k = 0; k < 8; ++k) { tv[k] = -INFINITY; ti[k] = -1; }
        cur_m = mt;
      }
      const int m0 = mt * (BM * NCTA) + (int)rank * BM;
      const int n0 = nt * p.BN;
      const int row = m0 + r;
      const int sub0 = m0 + quarter * SUB_ROWS;            // first row of this warp
      const int pcol = n0 + g_col;                         // first column of this group's panel
      const int buf = t_local & 1;
      const uint32_t use = (uint32_t)(t_local >> 1);
      // Under the main loop: everything that the accumulator is not needed for
      uint32_t bias2 = 0u;                                 // this lane's two of the panel's 64 bias values
      uint32_t kept[2] = {0xffffffffu, 0xffffffffu};       // dropout decisions of the 64 columns
      if (STAGED && staging) {
        if (tc::elect_one()) {                             // always the same lane: it waits for the stores it issued
          tc::tma_store_wait_read<0>();                    // the panel is free once the previous store has read it
          if (HAS_IN) {
            tc::mbar_expect_tx(my_in_bar, IN_BYTES);
            tc::tma_load_2d(pan, &tmR, my_in_bar, pcol, sub0);
            if (EPI == E_DW_SGD) {
              tc::tma_load_2d(pan2, &tmF, my_in_bar, pcol, sub0);
              // the next tile's weights and momentum on their way to L2: 1.3 M labels x 768, batch 512, 1680 -> 1661 us; 312330 x
              // 768, batch 90, 385 -> 375.  (The same for the weights that the logits and top-k products stream made them slower,
              // 51 -> 63 us at 131072 x 256: their ring already keeps 24 MB on the way.)
              if (item + its < it1) {
                const int mt2 = (item + its) / p.n_n_tiles, nt2 = (item + its) - mt2 * p.n_n_tiles;
                const int row2 = mt2 * (BM * NCTA) + (int)rank * BM + quarter * SUB_ROWS;
                if (row2 < M) {
                  tc::tma_prefetch_2d(&tmR, nt2 * p.BN + g_col, row2);
                  tc::tma_prefetch_2d(&tmF, nt2 * p.BN + g_col, row2);
                }
              }
            }
          }
        }
        if ((EPI == E_BIAS_GELU || EPI == E_BIAS_DROPOUT_RESID) && pcol + 2 * lane < p.N)
          bias2 = __ldg(reinterpret_cast<const uint32_t*>(reinterpret_cast<const T*>(p.bias) + pcol) + lane);
        if (EPI == E_BIAS_DROPOUT_RESID && p.p > 0.f) {
          // dropout counters number the padded layout's rows
          const int drop_row = p.tok != nullptr && row < M ? __ldcg(p.tok + row) : row;
          const uint32_t e0 = (uint32_t)(drop_row * p.N + pcol);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t bits = 0u;
#pragma unroll 8
            for (int j = 0; j < 32; ++j) bits |= (keep(seed, p.stream, e0 + 32 * h + j, p.p) ? 1u : 0u) << j;
            kept[h] = bits;
          }
        }
        if (EPI == E_SIGMOID_POS && p.pos_labels != nullptr && mt != pos_m) {
          // A unit's tiles ascend, so where positives are sparse the window that one search found serves the next tiles too
          // (1.3 M labels x 1024 rows, 64-deep: 0.5 positives per 32 labels; with a search of four dependent loads per M tile
          // the launches took 67 us, without any positives 43)
          const int k_lo = p.label0 + sub0, k_hi = p.label0 + min(sub0 + SUB_ROWS, M), nnz = *p.nnz_ptr;
          const bool held = pos_m >= 0 && mt > pos_m && __shfl_sync(0xffffffffu, pos_l, 31) >= k_hi;
          pos_m = mt;
          if (!held) {
            int first;
            warp_bounds(p.pos_labels, nnz, k_lo, k_hi, lane, first, pos_end);
            const int e = first + lane;
            pos_l = e < nnz ? p.pos_labels[e] : 0x7fffffff;
            pos_c = e < nnz ? p.pos_rows[e] : 0;
            pos_more = first + 32;
          } else {
            pos_end = 0;                                   // the window reaches past this tile's labels
          }
        }
      }
      bool ok = true;
      uint4 in_row[HELD_IN ? 8 : 1];                       // the tile-shaped input of this thread's row
      if (STAGED && staging && HAS_IN) {
        ok = tc::mbar_wait(my_in_bar, in_count & 1, aborted, p.status, tc::SITE_FULL, 2000 + g);
        ++in_count;
        if constexpr (HELD_IN) {
#pragma unroll
          for (int chunk = 0; chunk < 8; ++chunk) in_row[chunk] = *reinterpret_cast<const uint4*>(pan + panel_off(lane, chunk));
        }
      }
      ok = tc::mbar_wait(tmem_full_bar + buf, use & 1, aborted, p.status, tc::SITE_TMEM_FULL, item) && ok;
      if constexpr (STAGED) {
        // A staging warp whose wait has run out stores nothing from here on (every later wait of it returns at once).  It leaves by
        // itself, except from the logits: there the warps of the same 32 rows meet below at barriers without a time limit, and a
        // neighbour whose wait ended just in time would stand there for ever.  So it still comes to all of them.
        if (!__all_sync(0xffffffffu, ok)) {
          if (EPI != E_SIGMOID_POS) break;
          aborted = true;                                  // in every lane
          if (staging && p.pos_labels != nullptr && pos_end > pos_more) {
            meet_rows(quarter, p.BN >> 6);
            meet_rows(quarter, p.BN >> 6);
          }
          continue;
        }
      } else {
        if (!ok) *s_abort = 1;
        asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");
        if (*s_abort) break;                               // the same answer in every epilogue warp
      }
      tc::tc_fence_after();
      if (STAGED && staging) {
        const uint32_t tbase = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)buf * ACC_STRIDE + (uint32_t)g_col;
        uint4 keep2[EPI == E_BIAS_GELU ? 8 : 1];           // BIAS_GELU: the second output, packed, until the first has left
        uint32_t frag[2][8];                               // 8 accumulator columns at work, 8 on their way
        tc::tmem_issue8(tbase, frag[0]);
        __syncwarp();                                      // lane 0 has seen the panel free (!HAS_IN)
#pragma unroll
        for (int chunk = 0; chunk < 8; ++chunk) {
          tc::tmem_wait8(frag[chunk & 1]);
          if (chunk < 7) tc::tmem_issue8(tbase + 8 * (chunk + 1), frag[(chunk + 1) & 1]);
          const int c = pcol + 8 * chunk;
          uint4* slot = reinterpret_cast<uint4*>(pan + panel_off(lane, chunk));
          float a[8], o[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) a[j] = __uint_as_float(frag[chunk & 1][j]);
          if (EPI == E_STORE) {
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = a[j];
          } else if (EPI == E_SIGMOID_POS) {
            if (p.loss_acc != nullptr && row < M) {
              // sampled loss (dl_base.py:579-583): softplus of every logit here; minus the logits at the positives
              // by a separate small kernel
#pragma unroll
              for (int j = 0; j < 8; ++j)
                if (c + j < p.N) loss += fmaxf(a[j], 0.f) + log1pf(__expf(-fabsf(a[j])));
            }
            sigmoid8(a, o);
            if (c + 8 > p.N) {                         // the columns behind the batch are written as zeros
#pragma unroll
              for (int j = 0; j < 8; ++j) if (c + j >= p.N) o[j] = 0.f;
            }
          } else if (EPI == E_BIAS_GELU || EPI == E_BIAS_DROPOUT_RESID) {
            uint4 braw;
            braw.x = __shfl_sync(0xffffffffu, bias2, 4 * chunk); braw.y = __shfl_sync(0xffffffffu, bias2, 4 * chunk + 1);
            braw.z = __shfl_sync(0xffffffffu, bias2, 4 * chunk + 2); braw.w = __shfl_sync(0xffffffffu, bias2, 4 * chunk + 3);
            float b[8];
            unpack8<T>(braw, b);
            if (EPI == E_BIAS_GELU) {
#pragma unroll
              for (int j = 0; j < 8; ++j) o[j] = a[j] + b[j];
              const uint4 f16 = pack8<T>(o);
              *slot = f16;
              unpack8<T>(f16, o);                        // the backward pass differentiates at the stored value
#pragma unroll
              for (int j = 0; j < 8; j += 2) f2_get(gelu2(f2(o[j], o[j + 1])), a[j], a[j + 1]);
              keep2[EPI == E_BIAS_GELU ? chunk : 0] = pack8<T>(a);
            } else {
              float res[8];
              unpack8<T>(in_row[HELD_IN ? chunk : 0], res);
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                float t = a[j] + b[j];
                if (p.p > 0.f) t = (kept[chunk >> 2] >> (8 * (chunk & 3) + j)) & 1u ? t * inv_keep : 0.f;
                o[j] = res[j] + t;
              }
            }
          } else if (EPI == E_ADD) {
            float res[8];
            unpack8<T>(in_row[HELD_IN ? chunk : 0], res);
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = a[j] + res[j];
          } else if (EPI == E_DW_SGD) {
            // momentum SGD on the tile: m = mo m + (dW + wd w), w -= lr m, with m rounded to 16 bit first.  One element
            // at a time this was some 40 instructions per element, more than the tile's bytes take: two per instruction.
            // The noise of the rounding takes a hash per element, half of what is left.  1.3 M labels x 768, batch 512:
            // 2.01 -> 1.76 ms (1.68 with one hash per pair, which gives other weights for the same seed).
            uint4* slot2 = reinterpret_cast<uint4*>(pan2 + panel_off(lane, chunk));
            float w[8], mm[8];
            unpack8<T>(*slot, w);
            unpack8<T>(*slot2, mm);
            const F2 nlr = f2(-p.hp[HP_LR_XFC]), mo2 = f2(p.mo), wd2 = f2(p.wd);
            const uint32_t sr_seed = reinterpret_cast<const uint32_t*>(p.hp)[HP_SEED];
            const uint32_t e = (uint32_t)row * (uint32_t)p.ldW + (uint32_t)c;
#pragma unroll
            for (int j = 0; j < 8; j += 2)
              f2_get(f2_fma(mo2, f2(mm[j], mm[j + 1]), f2_fma(wd2, f2(w[j], w[j + 1]), f2(a[j], a[j + 1]))), mm[j], mm[j + 1]);
            const uint4 m16 = pack8<T>(mm);
            unpack8<T>(m16, mm);
#pragma unroll
            for (int j = 0; j < 8; j += 2) f2_get(f2_fma(nlr, f2(mm[j], mm[j + 1]), f2(w[j], w[j + 1])), o[j], o[j + 1]);
            *slot2 = m16;
            if (p.stochastic_round) {
              uint4 w16;                               // every element has a hash of its own number
              uint32_t* wp = reinterpret_cast<uint32_t*>(&w16);
#pragma unroll
              for (int j = 0; j < 8; j += 2)
                wp[j >> 1] = sr_pack2<T>(o[j], o[j + 1], mix32(sr_seed, 0x5152u, e + j), mix32(sr_seed, 0x5152u, e + j + 1));
              *slot = w16;
            } else {
              *slot = pack8<T>(o);
            }
          } else {   // E_GELU_BWD
            float f[8];
            unpack8<T>(in_row[HELD_IN ? chunk : 0], f);
#pragma unroll
            for (int j = 0; j < 8; j += 2) f2_get(f2(a[j], a[j + 1]) * gelu_grad2(f2(f[j], f[j + 1])), o[j], o[j + 1]);
          }
          if (EPI != E_BIAS_GELU && EPI != E_DW_SGD) *slot = pack8<T>(o);
        }
        if (EPI == E_SIGMOID_POS && p.pos_labels != nullptr) {
          // subtract 1 at the tile's positives while it is still in shared memory: entries of the label-sorted list whose
          // label is one of this warp's 32 rows and whose batch row is one of the panel's 64 columns
          __syncwarp();                                    // every row of the warp's part is written
          const int lab0 = p.label0 + sub0, n_lab = min(SUB_ROWS, M - sub0);
          const auto apply = [&](int pl, int pc, uint8_t* part, int col0) {
            const int bcol = pc - col0, pr = pl - lab0;
            if (pr >= 0 && pr < n_lab && bcol >= 0 && bcol < 64 && pc < p.N) {
              T* cell = reinterpret_cast<T*>(part + panel_off(pr, bcol >> 3)) + (bcol & 7);
              *cell = from_f<T>(to_f(*cell) - 1.f);        // duplicates are removed by the collator: one writer per cell
            }
          };
          apply(pos_l, pos_c, pan, pcol);
          if (pos_end > pos_more) {
            // Labels that many rows have (the first 32 of a Zipf-distributed 1.3 M hold 5000 of 21000 positives): the warps of
            // these 32 rows share the entries out, each applying its own to all panels of the tile, 8 on their way per lane.
            // Every panel's warp scanning all of them made the launch with those labels take 192 us, where the others take 47.
            // (The same list, hence the same two meetings per tile, in each of these warps.)
            const int np = p.BN >> 6;
            meet_rows(quarter, np);
            for (int e0 = pos_more + 32 * g + lane; e0 < pos_end; e0 += 256 * np) {
              int pl[8], pc[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                const int e = e0 + 32 * np * u;
                pl[u] = e < pos_end ? p.pos_labels[e] : 0x7fffffff;
                pc[u] = e < pos_end ? p.pos_rows[e] : 0;
              }
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                const int pg = (pc[u] - n0) >> 6;          // panel of the tile
                if (pg >= 0 && pg < np) apply(pl[u], pc[u], panels + pg * PANEL_BYTES + quarter * SUB_BYTES, n0 + 64 * pg);
              }
            }
            tc::fence_proxy_async();
            meet_rows(quarter, np);
          }
        }
        tc::fence_proxy_async();                 // generic-proxy writes of the panel before the async-proxy store
        __syncwarp();
        if (sub0 < M && tc::elect_one()) {
          tc::tma_store_2d(EPI == E_BIAS_GELU ? &tmF : &tmC, pan, pcol, sub0);
          if (EPI == E_DW_SGD) tc::tma_store_2d(&tmF, pan2, pcol, sub0);
          tc::tma_store_commit();
        }
        if (EPI == E_BIAS_GELU) {
          // second output through the same panel: C = gelu(F), held in registers
          if (tc::elect_one()) tc::tma_store_wait_read<0>();
          __syncwarp();
#pragma unroll
          for (int chunk = 0; chunk < 8; ++chunk)
            *reinterpret_cast<uint4*>(pan + panel_off(lane, chunk)) = keep2[EPI == E_BIAS_GELU ? chunk : 0];
          tc::fence_proxy_async();
          __syncwarp();
          if (sub0 < M && tc::elect_one()) {
            tc::tma_store_2d(&tmC, pan, pcol, sub0);
            tc::tma_store_commit();
          }
        }
        if (EPI == E_GELU_BWD && p.colacc != nullptr && sub0 < M && pcol + 2 * lane < p.N) {
          // bias gradient: each lane adds two columns of the staged (rounded) rows; rows past the packed tokens hold what an
          // earlier pass left
          const int n_rows = min(SUB_ROWS, M - sub0);
          F2 cs = f2(0.f);
          for (int i = 0; i < n_rows; ++i) {
            const uint32_t w = *reinterpret_cast<const uint32_t*>(pan + panel_off(i, lane >> 2) + 4 * (lane & 3));
            const T* e = reinterpret_cast<const T*>(&w);
            cs = cs + f2(to_f(e[0]), to_f(e[1]));
          }
          float c0, c1;
          f2_get(cs, c0, c1);
          float* at = p.colacc + (size_t)(blockIdx.x % kColReplicas) * p.col_tot + p.col_off + pcol + 2 * lane;
          atomicAdd(at, c0);
          atomicAdd(at + 1, c1);
        }
      }
      if (EPI == E_TOPK) {
        const uint32_t ttk = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)buf * ACC_STRIDE + (uint32_t)(g * ucols);
        {
          for (int cc = 0; u_active && cc < ucols; cc += 32) {
            float v[32];
            __syncwarp();                                  // the load is warp-wide; lanes leave the body below apart
            tc::tmem_ld32(ttk + cc, v);
            const int c0 = n0 + g * ucols + cc;
            // Most fragments hold nothing for any of the warp's rows once the lists are warm: one maximum over the 32
            // values decides.  A NaN must pass the test (it ranks above every number), hence max.NaN.
            float m8[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) m8[q] = max_nan(max_nan(v[4 * q], v[4 * q + 1]), max_nan(v[4 * q + 2], v[4 * q + 3]));
            const float top = max_nan(max_nan(max_nan(m8[0], m8[1]), max_nan(m8[2], m8[3])),
                                      max_nan(max_nan(m8[4], m8[5]), max_nan(m8[6], m8[7])));
            const bool some = !(top <= tv[7]);
            const bool cold = __any_sync(0xffffffffu, some && tv[7] == -INFINITY);
            if (!some) continue;
            if (!cold) {
              // Warm lists: a lane has one or two candidates among its 32 values, but hardly two lanes in the same column.
              // Every lane steps through its own (bit j of hits), so the warp takes as many insertions as its busiest lane
              // has candidates, not one per column that any lane has one in (half of them, still, at the 14th fragment).
              uint32_t hits = 0u;
#pragma unroll
              for (int j = 0; j < 32; ++j) hits |= (v[j] <= tv[7] ? 0u : 1u) << j;
              if (c0 + 32 > p.N) hits &= c0 < p.N ? (1u << (p.N - c0)) - 1u : 0u;
              while (hits != 0u) {
                const int j = __ffs(hits) - 1;
                hits &= hits - 1u;
                float q16[16], q8[8], q4[4];
#pragma unroll
                for (int i = 0; i < 16; ++i) q16[i] = (j & 1) ? v[2 * i + 1] : v[2 * i];
#pragma unroll
                for (int i = 0; i < 8; ++i) q8[i] = (j & 2) ? q16[2 * i + 1] : q16[2 * i];
#pragma unroll
                for (int i = 0; i < 4; ++i) q4[i] = (j & 4) ? q8[2 * i + 1] : q8[2 * i];
                const float q0 = (j & 8) ? q4[1] : q4[0], q1 = (j & 8) ? q4[3] : q4[2];
                const float x = topk_store_value((j & 16) ? q1 : q0);
                const int col = c0 + j;
#pragma unroll
                for (int k = 7; k >= 0; --k) {           // strict: of equal values the lower column stays
                  const bool up = k > 0 && x > tv[k > 0 ? k - 1 : 0];      // the entry above moves down
                  const bool here = x > tv[k];
                  const float nv = up ? tv[k > 0 ? k - 1 : 0] : x;
                  const int ni = up ? ti[k > 0 ? k - 1 : 0] : col;
                  if (here) { tv[k] = nv; ti[k] = ni; }
                }
              }
              continue;
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              if (m8[q] <= tv[7]) continue;
#pragma unroll
              for (int j = 4 * q; j < 4 * q + 4; ++j) {
                const float x = topk_store_value(v[j]);
                if (x > tv[7] && c0 + j < p.N) {         // strict: of equal values the lower column stays
                  tv[7] = x; ti[7] = c0 + j;
#pragma unroll
                  for (int k = 7; k > 0; --k) {
                    if (tv[k] > tv[k - 1]) {
                      const float a = tv[k]; tv[k] = tv[k - 1]; tv[k - 1] = a;
                      const int b = ti[k]; ti[k] = ti[k - 1]; ti[k - 1] = b;
                    }
                  }
                }
              }
            }
          }
        }
      }
      if (EPI == E_DX) {
        const float scale = p.hp[HP_SCALE];
        const uint32_t tdx = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)buf * ACC_STRIDE + (uint32_t)(g * ucols);
        for (int c0 = 0; u_active && c0 < ucols; c0 += 32) {
          float v[32];
          tc::tmem_ld32(tdx + c0, v);
          const int col0 = n0 + g * ucols + c0;
          if (row < M) {
            float* d = p.dX + (size_t)row * p.ldX + col0;
#pragma unroll
            for (int j4 = 0; j4 < 8; ++j4)
              if (col0 + 4 * j4 < p.N)
                red_add_f32x4(d + 4 * j4, v[4 * j4] * scale, v[4 * j4 + 1] * scale, v[4 * j4 + 2] * scale, v[4 * j4 + 3] * scale);
          }
        }
      }
      if (EPI == E_SPLITK) {
        const uint32_t tsk = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)buf * ACC_STRIDE + (uint32_t)(g * ucols);
        for (int c0 = 0; u_active && c0 < ucols; c0 += 32) {
          float v[32];
          tc::tmem_ld32(tsk + c0, v);
          const int c_in_tile = g * ucols + c0;
          const int col0 = n0 + c_in_tile;
          if (row < M) {
            if (splits == 1) {
#pragma unroll
              for (int j8 = 0; j8 < 4; ++j8)
                if (col0 + 8 * j8 < p.N)
                  *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.C) + (size_t)row * p.ldc + col0 + 8 * j8) = pack8<T>(v + 8 * j8);
            } else {
              float* s = p.sk_scratch + (size_t)tile * (BM * NCTA * p.BN) + (size_t)((int)rank * BM + r) * p.BN + c_in_tile;
#pragma unroll
              for (int j4 = 0; j4 < 8; ++j4)
                if (col0 + 4 * j4 < p.N) red_add_f32x4(s + 4 * j4, v[4 * j4], v[4 * j4 + 1], v[4 * j4 + 2], v[4 * j4 + 3]);
            }
          }
        }
      }
      // every tcgen05.ld of this item has completed (tmem_ld32 waits): hand the accumulator back to the MMA warp
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (NCTA == 2) tc::mbar_arrive_leader(tmem_empty_bar + buf); else tc::mbar_arrive(tmem_empty_bar + buf);
      }
      if (EPI == E_SPLITK && splits > 1) {
        // split-K fix-up: the CTA that adds the last partial of its half of a tile converts the sum and re-zeroes
        // the scratch (each CTA of a pair counts its own half)
        unsigned* cnt = p.sk_counters + (size_t)tile * NCTA + rank;
        __threadfence();
        asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");
        if (threadIdx.x == 64) *s_last = (atomicAdd(cnt, 1u) == (unsigned)(splits - 1)) ? 1 : 0;
        asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");
        if (*s_last) {
          // this CTA's 128 x BN block of the tile's scratch is contiguous: walk it with coalesced 16-byte accesses,
          // several loads in flight per thread
          __threadfence();
          T* C = reinterpret_cast<T*>(p.C);
          float4* blk = reinterpret_cast<float4*>(p.sk_scratch + (size_t)tile * (BM * NCTA * p.BN) + (size_t)((int)rank * BM) * p.BN);
          const int n4 = BM * p.BN / 4;
          const int bn4 = p.BN / 4;
          const int et = (int)threadIdx.x - 64;
          for (int base = et; base < n4; base += EPI_THREADS * 4) {
            float4 x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int i4 = base + EPI_THREADS * u;
              x[u] = i4 < n4 ? __ldcg(blk + i4) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int i4 = base + EPI_THREADS * u;
              if (i4 < n4) {
                __stcg(blk + i4, make_float4(0.f, 0.f, 0.f, 0.f));
                const int rr = i4 / bn4, cc = (i4 - rr * bn4) * 4;
                const int grow = m0 + rr, gcol = n0 + cc;
                if (grow < M && gcol < p.N) {
                  uint2 o;
                  T* e = reinterpret_cast<T*>(&o);
                  e[0] = from_f<T>(x[u].x); e[1] = from_f<T>(x[u].y); e[2] = from_f<T>(x[u].z); e[3] = from_f<T>(x[u].w);
                  *reinterpret_cast<uint2*>(C + (size_t)grow * p.ldc + gcol) = o;
                }
              }
            }
          }
          if (threadIdx.x == 64) *cnt = 0u;
        }
      }
    }
    if (STAGED && staging && tc::elect_one()) tc::tma_store_wait_read<0>();   // the stores have read shared memory; they complete before the grid does
    if (EPI == E_SIGMOID_POS && p.loss_acc != nullptr) {
      loss = warp_sum(loss);
      if (lane == 0 && loss != 0.f) atomicAdd(p.loss_acc, loss);
    }
    if (EPI == E_DX && p.done_counter != nullptr) {
      // reduce-scatter epilogue: the last CTA of this rank's dX GEMM tells every rank that the partial sums in this
      // rank's buffer are complete
      __threadfence_system();
      asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");
      if (threadIdx.x == 64) {
        if (atomicAdd(p.done_counter, 1u) == gridDim.x - 1) {
          *p.done_counter = 0u;
          __threadfence_system();
          const uint32_t tagv = *p.step_ptr;
          for (int q = 0; q < p.n_peers; ++q) st_release_sys(reinterpret_cast<uint32_t*>(p.peer_flags[q]) + p.flag_index, tagv);
        }
      }
    }
    if (EPI == E_TOPK) topk_flush();
  }
  tc::tc_fence_before();
  __syncthreads();
  if (NCTA == 2) tc::cluster_sync_all();                   // the peer no longer reads this CTA's memory or barriers
  if (warp == 1) {
    tc::tc_fence_after();
    if (NCTA == 2) tc::tmem_dealloc_pair(tmem_base, TMEM_COLS); else tc::tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

}  // namespace eg
}  // namespace rb

// ------------------------------------------------------------------------------------ LayerNorm of a stored input
// y = LN(pre) with the row statistics kept for the backward pass; `pre` was written by the BIAS_DROPOUT_RESID
// epilogue.  One warp per row, 16-byte accesses.
namespace rb {
namespace eg {
template <typename T, int NV>
__global__ void __launch_bounds__(128) ln_fwd_kernel(const T* __restrict__ pre, const T* __restrict__ gamma,
                                                     const T* __restrict__ beta, T* __restrict__ y,
                                                     float* __restrict__ mean, float* __restrict__ rstd, int rows, int H,
                                                     float eps, const int* __restrict__ tok_meta) {
  grid_dep_wait();            // launched with launch_pdl: nothing above touches global memory
  grid_dep_launch();          // the kernel that follows may start its set-up now; it waits for this grid before reading
  const int lane = threadIdx.x & 31;
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (row >= (tok_meta != nullptr ? __ldcg(tok_meta + TOK_ROWS) : rows)) return;
  float v[NV][8];
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = (lane + 32 * i) * 8;
    if (col < H) {
      load8(pre + (size_t)row * H + col, v[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) sum += v[i][j];
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
      for (int j = 0; j < 8; ++j) { const float d = v[i][j] - mu; sq += d * d; }
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
}  // namespace eg
}  // namespace rb

using namespace rb;
using namespace rb::eg;

struct Maps { CUtensorMap a, b, c, r, f; };

// Programmatic dependent launch (a kernel's set-up overlaps the previous kernel's tail): on by default.
RB_API void rb_enc_gemm_set_pdl(int on) { pdl_flag() = on ? 1 : 0; }

template <typename T, int LAYOUT, int EPI, int NCTA>
static int launch_enc_gemm(const Maps& m, const Params& p, int units, cudaStream_t st) {
  static bool attr_set = false;
  auto k = enc_gemm_kernel<T, LAYOUT, EPI, NCTA>;
  constexpr int smem = Cfg<EPI>::kSmem;
  if (!attr_set) {
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -5;
    attr_set = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(NCTA * units, 1, 1);
  cfg.blockDim = dim3(THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int n_attr = 0;
  if (NCTA == 2) {
    attr[n_attr].id = cudaLaunchAttributeClusterDimension;
    attr[n_attr].val.clusterDim.x = 2;
    attr[n_attr].val.clusterDim.y = 1;
    attr[n_attr].val.clusterDim.z = 1;
    ++n_attr;
  }
  if (pdl_flag()) {
    attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
    ++n_attr;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n_attr;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k, m.a, m.b, m.c, m.r, m.f, p);
  return e == cudaSuccess ? 0 : (int)e;
}

template <typename T, int NCTA>
static int dispatch_enc_gemm(int layout, int epi, const Maps& m, const Params& p, int units, cudaStream_t st) {
  if (layout == L_NT) {
    if (epi == E_STORE) return launch_enc_gemm<T, L_NT, E_STORE, NCTA>(m, p, units, st);
    if (epi == E_BIAS_GELU) return launch_enc_gemm<T, L_NT, E_BIAS_GELU, NCTA>(m, p, units, st);
    if (epi == E_BIAS_DROPOUT_RESID) return launch_enc_gemm<T, L_NT, E_BIAS_DROPOUT_RESID, NCTA>(m, p, units, st);
    if (epi == E_TOPK) return launch_enc_gemm<T, L_NT, E_TOPK, NCTA>(m, p, units, st);
    if (epi == E_SIGMOID_POS) return launch_enc_gemm<T, L_NT, E_SIGMOID_POS, NCTA>(m, p, units, st);
  } else if (layout == L_NN) {
    if (epi == E_STORE) return launch_enc_gemm<T, L_NN, E_STORE, NCTA>(m, p, units, st);
    if (epi == E_ADD) return launch_enc_gemm<T, L_NN, E_ADD, NCTA>(m, p, units, st);
    if (epi == E_GELU_BWD) return launch_enc_gemm<T, L_NN, E_GELU_BWD, NCTA>(m, p, units, st);
    if (epi == E_DW_SGD) return launch_enc_gemm<T, L_NN, E_DW_SGD, NCTA>(m, p, units, st);
  } else if (layout == L_TN) {
    if (epi == E_SPLITK) return launch_enc_gemm<T, L_TN, E_SPLITK, NCTA>(m, p, units, st);
    if (epi == E_DX) return launch_enc_gemm<T, L_TN, E_DX, NCTA>(m, p, units, st);
  }
  return -4;
}

// Tile shape and K-splits from a cost model calibrated on B200 (clocks per CTA; grids of 256 x 256 pair tiles down to
// 128 x 64, K = 64 .. 3072, chained launches):
//   * a k block costs the largest of MMA time (2.25 BN: shared memory, read by the MMAs and written by the loads, keeps the
//     tensor pipe from its 2 BN), operand bytes of the CTA over the rate at which an SM receives them (75 bytes per clock
//     with most SMs busy), and about 290 clocks of issue and barrier traffic;
//   * work is spread over the units (SMs, or SM pairs) in rounds; a round cannot be shorter than a tile's epilogue, and a
//     share of the epilogue is added to it (epi_share);
//   * about 3000 clocks of start-up per kernel (TMEM allocation, barrier set-up, first load), 600 more for pairs;
//   * the epilogue of a CTA's last tile is exposed: epi_clocks, by 64-column panels;
//   * a K-split costs about 10000 clocks (partial sums through L2 atomics, the last CTA's conversion pass).
struct Plan { int ncta, bn, splits, tiles; };

static int g_max_units = 0;
// Experiments: cap the number of persistent workers (0 = one per SM / SM pair).
RB_API void rb_enc_gemm_set_max_units(int n) { g_max_units = n; }

static double epi_clocks(int epi, int bn) {
  const double n = bn / 64.0;
  switch (epi) {
    case E_STORE: return 800 + 480 * n;
    case E_ADD: return 1000 + 560 * n;
    case E_BIAS_DROPOUT_RESID: return 2500 + 800 * n;
    case E_BIAS_GELU: return 3000 + 1700 * n;
    case E_GELU_BWD: return 2800 + 1550 * n;
    case E_SIGMOID_POS: return 1000 + 1200 * n;
    case E_DW_SGD: return 1500 + 1500 * n;
    default: return 800;                       // SPLITK, DX, TOPK
  }
}
// Share of a tile's epilogue that its round is longer than the main loop: shared-memory traffic of the panels, and for the
// dropout epilogue the hashes of a tile that does not have the epilogue warps to itself.
static double epi_share(int epi) { return epi == E_BIAS_DROPOUT_RESID ? 0.6 : 0.35; }

static Plan make_plan(int layout, int epi, int M, int N, int K, int bn_forced, int ncta_forced) {
  const int sms = sm_count();
  const int kb = (K + BK - 1) / BK;
  Plan best{1, 128, 1, 1};
  double best_cost = -1.0;
  for (int ncta = 1; ncta <= 2; ++ncta) {
    if (ncta_forced && ncta != ncta_forced) continue;
    for (int bn = 256; bn >= 64; bn >>= 1) {
      if (bn_forced && bn != bn_forced) continue;
      if (ncta == 2 && bn < 128) continue;
      if (!bn_forced && bn > 64 && bn / 2 >= N) continue;            // a narrower tile already covers every column
      const int tiles = ((M + BM * ncta - 1) / (BM * ncta)) * ((N + bn - 1) / bn);
      const int units = sms / ncta;
      int max_splits = layout == L_TN ? (kb < 16 ? kb : 16) : 1;
      int first_split = 1;
      if (epi == E_DX) {                      // partial sums are reduced into the output directly: split as far as the units go
        first_split = units / tiles < 1 ? 1 : (units / tiles > kb ? kb : units / tiles);
        max_splits = first_split;
      }
      for (int splits = first_split; splits <= max_splits; splits = (splits == max_splits ? max_splits + 1 : splits * 2)) {
        const int kb_per = (kb + splits - 1) / splits;
        const int eff_splits = (kb + kb_per - 1) / kb_per;
        if (eff_splits != splits && splits > 1 && epi != E_DX) continue;
        const long items = (long)tiles * eff_splits;
        const long rounds = (items + units - 1) / units;
        const double busy = (double)(items < units ? items : units) * ncta / sms;      // fraction of the SMs at work
        const double bytes = A_BYTES + (double)(bn / ncta) * BK * 2;
        double t_kb = bytes / (busy > 0.5 ? 75.0 : 150.0);
        if (t_kb < 290.0) t_kb = 290.0;
        if (t_kb < 2.25 * bn) t_kb = 2.25 * bn;
        const double tail = epi_clocks(epi, bn);
        double round = kb_per * t_kb + epi_share(epi) * tail;
        if (round < tail) round = tail;
        double cost = 3000.0 + (ncta == 2 ? 600.0 : 0.0) + rounds * round + tail + (eff_splits > 1 && epi != E_DX ? 10000.0 : 0.0);
        if (epi == E_TOPK) cost += 120.0 * (items < units ? items : units);      // every unit leaves candidates to select from
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = Plan{ncta, bn, eff_splits, tiles}; }
      }
    }
  }
  return best;
}

// What rb_enc_gemm will use for (M, N, K): tile shape, K-splits for layout TN, and the sizes of the split-K
// scratch (floats) and counters (words) it needs when splits > 1.
RB_API int rb_enc_gemm_plan(int layout, int epi, int M, int N, int K, int bn_forced, int ncta_forced, int* ncta_out,
                            int* bn_out, int* splits_out, long long* scratch_floats, int* counter_words) {
  const Plan pl = make_plan(layout, epi, M, N, K, bn_forced, ncta_forced);
  *ncta_out = pl.ncta; *bn_out = pl.bn; *splits_out = pl.splits;
  *scratch_floats = (long long)pl.tiles * BM * pl.ncta * pl.bn;
  *counter_words = pl.tiles * pl.ncta;
  return 0;
}

// C = op(A) op(B) with a fused epilogue; see the head of this file.  Leading dimensions in elements.
//   layout 0 (NT): A[M, lda>=K], B[N, ldb>=K];  1 (NN): A[M, lda>=K], B[K, ldb>=N];  2 (TN): A[K, lda>=M], B[K, ldb>=N]
//   dtype: RB_BF16 or RB_F16 (operands, C, bias, R and F all have it; accumulation is fp32)
//   R [M, ldr]: residual (BIAS_DROPOUT_RESID, ADD) or stored pre-activation (GELU_BWD); F [M, ldf]: pre-activation
//   output (BIAS_GELU).  Layout TN with more than one K-split needs sk_scratch / sk_counters of the sizes
//   rb_enc_gemm_plan reports (zero on entry, left zero).  bn_forced / ncta_forced: 0 = choose.
//   tok_meta / tok (nullable; layouts NT and NN): packed tokens (token_map.cuh).  M is then the capacity in rows and the
//   kernel takes the row count from tok_meta; plan_rows (0 = the capacity) is the count to plan tiles for.
// Returns 0, or -3 for an unsupported shape (the caller then uses the library GEMM).
RB_API int rb_enc_gemm(int dtype, int layout, int epi, const void* A, const void* B, void* C, int M, int N, int K, int lda,
                       int ldb, int ldc, const void* bias, const void* R, int ldr, void* F, int ldf, float p_drop,
                       const int* seed, unsigned stream_id, float* colacc, int col_tot, int col_off, float* sk_scratch,
                       unsigned* sk_counters, int bn_forced, int ncta_forced, const int* tok_meta, const int* tok,
                       int plan_rows, int* status, cudaStream_t st) {
  if (dtype != RB_BF16 && dtype != RB_F16) return -1;
  if (M < 1 || N < 1 || K < 1 || N % 8 || lda % 8 || ldb % 8 || ldc % 8 || ldr % 8 || ldf % 8) return -3;
  if (layout == L_TN && M % 8) return -3;
  if ((epi == E_BIAS_GELU || epi == E_BIAS_DROPOUT_RESID) && bias == nullptr) return -3;
  if ((epi == E_BIAS_DROPOUT_RESID || epi == E_ADD || epi == E_GELU_BWD) && R == nullptr) return -3;
  if (epi == E_BIAS_GELU && F == nullptr) return -3;
  if (epi == E_BIAS_DROPOUT_RESID && p_drop > 0.f && seed == nullptr) return -3;
  const bool bf16 = dtype == RB_BF16;
  if (layout == L_TN && tok_meta != nullptr) return -3;
  const Plan pl = make_plan(layout, epi, plan_rows > 0 ? plan_rows : M, N, K, bn_forced, ncta_forced);
  const int BN = pl.bn, b_rows = BN / pl.ncta;
  Maps m;
  int rc;
  if (layout == L_TN) rc = tc::make_tmap_2d(&m.a, A, K, M, lda, 64, 64, bf16);
  else rc = tc::make_tmap_2d(&m.a, A, M, K, lda, 64, BM, bf16);
  if (rc) return rc;
  if (layout == L_NT) rc = tc::make_tmap_2d(&m.b, B, N, K, ldb, 64, b_rows, bf16);
  else rc = tc::make_tmap_2d(&m.b, B, K, N, ldb, 64, 64, bf16);
  if (rc) return rc;
  // output / input panels: [32 rows x 64 columns] boxes of the row-major [M, N] matrices, one per epilogue warp
  rc = tc::make_tmap_2d(&m.c, C, M, N, ldc, 64, SUB_ROWS, bf16);
  if (rc) return rc;
  m.r = m.c;
  m.f = m.c;
  if (R != nullptr && (rc = tc::make_tmap_2d(&m.r, R, M, N, ldr, 64, SUB_ROWS, bf16)) != 0) return rc;
  if (F != nullptr && (rc = tc::make_tmap_2d(&m.f, F, M, N, ldf, 64, SUB_ROWS, bf16)) != 0) return rc;
  Params p{};
  p.M = M; p.N = N; p.BN = BN;
  p.n_m_tiles = (M + BM * pl.ncta - 1) / (BM * pl.ncta); p.n_n_tiles = (N + BN - 1) / BN;
  p.kb_total = (K + BK - 1) / BK;
  p.splits = pl.splits;
  p.kb_per_split = (p.kb_total + p.splits - 1) / p.splits;
  if (p.splits > 1 && (sk_scratch == nullptr || sk_counters == nullptr)) return -3;
  p.C = C; p.ldc = ldc; p.bias = bias;
  p.p = p_drop; p.seed = seed; p.stream = stream_id;
  p.colacc = colacc; p.col_tot = col_tot; p.col_off = col_off;
  p.sk_scratch = sk_scratch; p.sk_counters = sk_counters; p.status = status;
  p.tok_meta = tok_meta; p.tok = tok;
  const int n_items = p.n_m_tiles * p.n_n_tiles * p.splits;
  int max_units = sm_count() / pl.ncta;
  if (g_max_units > 0 && g_max_units < max_units) max_units = g_max_units;
  const int units = n_items < max_units ? n_items : max_units;
  if (pl.ncta == 2)
    rc = bf16 ? dispatch_enc_gemm<__nv_bfloat16, 2>(layout, epi, m, p, units, st) : dispatch_enc_gemm<__half, 2>(layout, epi, m, p, units, st);
  else
    rc = bf16 ? dispatch_enc_gemm<__nv_bfloat16, 1>(layout, epi, m, p, units, st) : dispatch_enc_gemm<__half, 1>(layout, epi, m, p, units, st);
  if (rc) return rc;
  RB_LAUNCH_CHECK();
  return 0;
}

// Units of a TOPK launch.  An even number as soon as a unit gets several items: two M tiles are walked side by side and
// a unit must stay with one of them (topk.cuh).
static int topk_units(const Plan& pl, int n_m, int n_n) {
  const int max_units = sm_count() / pl.ncta;
  const long n_items = (long)n_m * n_n;
  return n_items <= max_units ? (int)n_items : (max_units > 1 ? max_units & ~1 : 1);
}

// Layout of the candidates that rb_xfc_topk_candidates leaves for (B, Ls, D): out[0] CTAs per tile, [1] N tile,
// [2] units, [3] N tiles, [4] M tiles, [5] floats (and ints) per row.
RB_API int rb_xfc_topk_plan(int B, int Ls, int D, int* out) {
  if (B < 1 || Ls < 1 || D < 1) return -3;
  const Plan pl = make_plan(L_NT, E_TOPK, B, Ls, D, 0, 0);
  const int n_m = (B + BM * pl.ncta - 1) / (BM * pl.ncta), n_n = (Ls + pl.bn - 1) / pl.bn;
  const int units = topk_units(pl, n_m, n_n);
  out[0] = pl.ncta; out[1] = pl.bn; out[2] = units; out[3] = n_n; out[4] = n_m; out[5] = units * EGROUPS * 8;
  return 0;
}

// Prediction: candidates for the k largest entries of every row of X W^T without materialising the product.
//   X [B, ldx >= D], W [Ls, ldw >= D] (16-bit, same dtype); cand_val / cand_idx [B, rb_xfc_topk_plan's row length]:
// every (unit, epilogue group) writes the 8 best (value, column of W) that it met in a row, in descending order, value
// -inf and column -1 where it met fewer.  topk.cu turns them into the k best.
RB_API int rb_xfc_topk_candidates(int dtype, const void* X, const void* W, int B, int Ls, int D, int ldx, int ldw,
                                  float* cand_val, int* cand_idx, int* status, cudaStream_t st) {
  if (dtype != RB_BF16 && dtype != RB_F16) return -1;
  if (B < 1 || Ls < 1 || D < 1 || ldx % 8 || ldw % 8) return -3;
  const bool bf16 = dtype == RB_BF16;
  const Plan pl = make_plan(L_NT, E_TOPK, B, Ls, D, 0, 0);
  const int BN = pl.bn, b_rows = BN / pl.ncta;
  Maps m;
  int rc = tc::make_tmap_2d(&m.a, X, B, D, ldx, 64, BM, bf16);
  if (rc) return rc;
  rc = tc::make_tmap_2d(&m.b, W, Ls, D, ldw, 64, b_rows, bf16);
  if (rc) return rc;
  m.c = m.a; m.r = m.a; m.f = m.a;
  Params p{};
  p.M = B; p.N = Ls; p.BN = BN;
  p.n_m_tiles = (B + BM * pl.ncta - 1) / (BM * pl.ncta); p.n_n_tiles = (Ls + BN - 1) / BN;
  p.kb_total = (D + BK - 1) / BK; p.splits = 1; p.kb_per_split = p.kb_total;
  const int units = topk_units(pl, p.n_m_tiles, p.n_n_tiles);
  p.cand_val = cand_val; p.cand_idx = cand_idx; p.cand_ld = units * EGROUPS * 8; p.status = status;
  rc = pl.ncta == 2
           ? (bf16 ? dispatch_enc_gemm<__nv_bfloat16, 2>(L_NT, E_TOPK, m, p, units, st) : dispatch_enc_gemm<__half, 2>(L_NT, E_TOPK, m, p, units, st))
           : (bf16 ? dispatch_enc_gemm<__nv_bfloat16, 1>(L_NT, E_TOPK, m, p, units, st) : dispatch_enc_gemm<__half, 1>(L_NT, E_TOPK, m, p, units, st));
  if (rc) return rc;
  RB_LAUNCH_CHECK();
  return 0;
}

template <int DUMMY = 0>
static int launch_planned(const Plan& pl, bool bf16, int layout, int epi, const Maps& m, Params& p, int K, cudaStream_t st) {
  p.BN = pl.bn;
  p.n_m_tiles = (p.M + BM * pl.ncta - 1) / (BM * pl.ncta); p.n_n_tiles = (p.N + pl.bn - 1) / pl.bn;
  p.kb_total = (K + BK - 1) / BK;
  p.splits = pl.splits;
  p.kb_per_split = (p.kb_total + p.splits - 1) / p.splits;
  const long n_items = (long)p.n_m_tiles * p.n_n_tiles * p.splits;
  int max_units = sm_count() / pl.ncta;
  if (g_max_units > 0 && g_max_units < max_units) max_units = g_max_units;
  const int units = n_items < max_units ? (int)n_items : max_units;
  return pl.ncta == 2
             ? (bf16 ? dispatch_enc_gemm<__nv_bfloat16, 2>(layout, epi, m, p, units, st) : dispatch_enc_gemm<__half, 2>(layout, epi, m, p, units, st))
             : (bf16 ? dispatch_enc_gemm<__nv_bfloat16, 1>(layout, epi, m, p, units, st) : dispatch_enc_gemm<__half, 1>(layout, epi, m, p, units, st));
}

// Classifier logits + gradient on the persistent GEMM: Gt[Lc, ldG] = sigmoid(W X^T) - Y for the fp16 label chunk
// W[Lc, D] and the gathered embeddings X[B, D]; columns B .. ldG of Gt are written as zeros.  Positives: label-sorted
// (row, label) pairs, labels numbered from label0 at row 0 of W; they are subtracted in shared memory before the tile
// is stored.  wait_flags != null: the loads wait until flags[0 .. wait_n) have reached *step_ptr (all-gather landed).
// Replaces, in the reference, torch.matmul + sigmoid_ + index_put_ (dl_base.py:572, 593-594) / the CUTLASS
// sigmoid-GEMM (xfc_gemm_kernel.cu:59-100).
RB_API int rb_xfc_logits_grad_v2(const void* W, int Lc, int D, const void* X, int B, void* Gt, int ldG, const int* pos_rows,
                                 const int* pos_labels, const int* nnz_ptr, int label0, const unsigned* wait_flags,
                                 int wait_n, const unsigned* step_ptr, float* loss_acc, int* status, cudaStream_t st) {
  if (D % 8 || ldG % 8 || Lc < 1 || B < 1 || ldG < B) return -3;
  const Plan pl = make_plan(L_NT, E_SIGMOID_POS, Lc, B, D, 0, 0);
  Maps m;
  int rc = tc::make_tmap_2d(&m.a, W, Lc, D, D, 64, BM, false);
  if (rc) return rc;
  rc = tc::make_tmap_2d(&m.b, X, B, D, D, 64, pl.bn / pl.ncta, false);
  if (rc) return rc;
  rc = tc::make_tmap_2d(&m.c, Gt, Lc, ldG, ldG, 64, SUB_ROWS, false);
  if (rc) return rc;
  m.r = m.c; m.f = m.c;
  Params p{};
  p.M = Lc; p.N = B; p.status = status;
  p.pos_rows = pos_rows; p.pos_labels = pos_labels; p.nnz_ptr = nnz_ptr; p.label0 = label0;
  p.wait_flags = wait_flags; p.wait_n = wait_n; p.step_ptr = step_ptr; p.loss_acc = loss_acc;
  rc = launch_planned(pl, false, L_NT, E_SIGMOID_POS, m, p, D, st);
  if (rc) return rc;
  RB_LAUNCH_CHECK();
  return 0;
}

// dX[B, D] += hp[SCALE] * Gt^T W over the label chunk (fp32, vector reductions; dX zeroed before the first chunk).
// done_counter != null: the last CTA stores *step_ptr into word flag_index of every peer's flag array.
RB_API int rb_xfc_dx_v2(const void* Gt, int ldG, const void* W, int Lc, int D, int B, float* dX, const float* hp,
                        unsigned* done_counter, void* const* peer_flags, int n_peers, int flag_index,
                        const unsigned* step_ptr, int* status, cudaStream_t st) {
  if (D % 8 || ldG % 8 || Lc < 1 || B < 1 || n_peers > 16) return -3;
  const Plan pl = make_plan(L_TN, E_DX, B, D, Lc, 0, 0);
  Maps m;
  int rc = tc::make_tmap_2d(&m.a, Gt, Lc, B, ldG, 64, 64, false);
  if (rc) return rc;
  rc = tc::make_tmap_2d(&m.b, W, Lc, D, D, 64, 64, false);
  if (rc) return rc;
  m.c = m.a; m.r = m.a; m.f = m.a;
  Params p{};
  p.M = B; p.N = D; p.status = status;
  p.dX = dX; p.ldX = D; p.hp = hp;
  if (done_counter != nullptr) {
    p.done_counter = done_counter; p.n_peers = n_peers; p.flag_index = flag_index; p.step_ptr = step_ptr;
    for (int q = 0; q < n_peers; ++q) p.peer_flags[q] = peer_flags[q];
  }
  rc = launch_planned(pl, false, L_TN, E_DX, m, p, Lc, st);
  if (rc) return rc;
  RB_LAUNCH_CHECK();
  return 0;
}

// Classifier weight update on the persistent GEMM: dW = Gt X over the batch (never stored), then momentum SGD on the
// [128 x 64] tiles of W and Mom [Lc, D] (fp16) in shared memory: both tiles come in by TMA under the main loop and
// leave by TMA; lr and the rounding seed are read from hp on the device.
// Replaces, in the reference, the fused dW GEMM + SGD epilogue (xfc_gemm_kernel.cu:102-151).
RB_API int rb_xfc_dw_sgd_v2(const void* Gt, int ldG, const void* X, int B, void* W, void* Mom, int Lc, int D,
                            const float* hp, float mo, float wd, int stochastic_round, int bn_forced, int ncta_forced,
                            int* status, cudaStream_t st) {
  if (D % 8 || ldG % 8 || Lc < 1 || B < 1) return -3;
  const Plan pl = make_plan(L_NN, E_DW_SGD, Lc, D, B, bn_forced, ncta_forced);
  Maps m;
  int rc = tc::make_tmap_2d(&m.a, Gt, Lc, B, ldG, 64, BM, false);
  if (rc) return rc;
  rc = tc::make_tmap_2d(&m.b, X, B, D, D, 64, 64, false);
  if (rc) return rc;
  rc = tc::make_tmap_2d(&m.c, W, Lc, D, D, 64, SUB_ROWS, false);
  if (rc) return rc;
  m.r = m.c;
  rc = tc::make_tmap_2d(&m.f, Mom, Lc, D, D, 64, SUB_ROWS, false);
  if (rc) return rc;
  Params p{};
  p.M = Lc; p.N = D; p.status = status;
  p.hp = hp; p.mo = mo; p.wd = wd; p.stochastic_round = stochastic_round; p.ldW = D;
  rc = launch_planned(pl, false, L_NN, E_DW_SGD, m, p, B, st);
  if (rc) return rc;
  RB_LAUNCH_CHECK();
  return 0;
}

#define EG_DISPATCH_NV(H, ...)                                                     \
  {                                                                                \
    const int nv_ = ((H) + 255) / 256;                                             \
    if (nv_ <= 1) { constexpr int NV = 1; __VA_ARGS__; }                           \
    else if (nv_ <= 2) { constexpr int NV = 2; __VA_ARGS__; }                      \
    else if (nv_ <= 3) { constexpr int NV = 3; __VA_ARGS__; }                      \
    else if (nv_ <= 4) { constexpr int NV = 4; __VA_ARGS__; }                      \
    else if (nv_ <= 8) { constexpr int NV = 8; __VA_ARGS__; }                      \
    else return -2;                                                                \
  }

RB_API int rb_ln_fwd(int dtype, const void* pre, const void* gamma, const void* beta, void* y, float* mean, float* rstd,
                     int rows, int H, float eps, const int* tok_meta, cudaStream_t st) {
  if (H % 8 || rows < 1) return -3;
  const int blocks = (rows + 3) / 4;
  switch (dtype) {
    case RB_F32: { using T = float; EG_DISPATCH_NV(H, (launch_pdl(ln_fwd_kernel<T, NV>, dim3(blocks), dim3(128), 0, st, (const T*)pre, (const T*)gamma, (const T*)beta, (T*)y, mean, rstd, rows, H, eps, tok_meta))); break; }
    case RB_BF16: { using T = __nv_bfloat16; EG_DISPATCH_NV(H, (launch_pdl(ln_fwd_kernel<T, NV>, dim3(blocks), dim3(128), 0, st, (const T*)pre, (const T*)gamma, (const T*)beta, (T*)y, mean, rstd, rows, H, eps, tok_meta))); break; }
    case RB_F16: { using T = __half; EG_DISPATCH_NV(H, (launch_pdl(ln_fwd_kernel<T, NV>, dim3(blocks), dim3(128), 0, st, (const T*)pre, (const T*)gamma, (const T*)beta, (T*)y, mean, rstd, rows, H, eps, tok_meta))); break; }
    default: return -1;
  }
  RB_LAUNCH_CHECK();
  return 0;
}
