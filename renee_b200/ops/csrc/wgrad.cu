// The weight gradients of one transformer layer in one launch: dW_i [M_i, N_i] = dY_i^T X_i for up to MAX_PROBS linears
// that share the token dimension (q/k/v, output projection, FFN1, FFN2), 16-bit operands, fp32 accumulation, sm_100a.
//
// Each of them alone is a poor fit for the chip: at 768 columns they have 9 to 36 tiles of 256 x 256 for 74 SM pairs, so
// they were split over the tokens, reduced through fp32 atomics in L2 and converted by a last pass -- 29 us per launch,
// 116 us per layer, at 4900 tokens, where the products take 44 us at the measured cuBLAS rate.  Here the work of all of
// them is shared out evenly: as many whole tiles per pair of SMs as all pairs get, all walking the tokens in step so that
// the operands they share come from L2, and before that the left-over tiles, as one line of (tile, k block) pairs cut into
// equal runs ("stream-K").  (All tiles in one line, without the whole ones: 64 us per layer at 4900 tokens, 140 at 10200;
// the units then read the operands, 250 MB at 10200 tokens, at unrelated places.)  A tile that a cut falls into is reduced
// across units.  A unit that holds part of such a tile writes its fp32
// sums to its own place in a scratch and counts itself; the one that finds all others counted adds their sums to its
// accumulators, which are still in TMEM, and stores the tile.  Nobody waits for anybody, and the scratch needs no
// initial value.  Measured per layer: 57 us at 4900 tokens
// (4 x 29 as single split-K launches), 95 at 10200 (164); steps 256 x 32 2.74 -> 2.57 ms, 128 x 128 5.08 -> 4.80 ms.
//
// Same structure as gemm.cu: cta_group::2 tiles of 256 x 256 (128 accumulator rows per CTA), warp 0 TMA producer, warp 1
// MMA issuer, sixteen epilogue warps (a thread owns one row and 64 columns), two accumulators in TMEM, a 7-stage ring that
// keeps streaming across tiles, every wait bounded.  With packed tokens the number of k blocks comes from the device.
#include "tc.cuh"
#include "token_map.cuh"

namespace rb {
namespace wg {

constexpr int BM = 128, BN = 256, BK = 64;
constexpr int STAGE = BM * BK * 2 + (BN / 2) * BK * 2;    // per CTA: 128 rows of A, half of the 256 columns of B
constexpr int STAGES = 7;
constexpr int EPI_WARPS = 16, EPI_THREADS = 32 * EPI_WARPS, THREADS = 64 + EPI_THREADS;
constexpr int TMEM_COLS = 512;
constexpr int MAX_PROBS = 5;                                // a layer's four and one that the layer behind it left over
constexpr int MIN_RUN = 8;                                 // k blocks per unit at least: bounds the pieces of a tile
constexpr int SMEM = STAGES * STAGE + 1024 + 512;
constexpr size_t PIECE_FLOATS = (size_t)BM * BN;           // one CTA's half of a tile

struct Maps { CUtensorMap a[MAX_PROBS], b[MAX_PROBS]; };
struct Prob { int M, N, n_n, first; void* C; int ldc; };   // first: number of its first tile
struct Params {
  Prob prob[MAX_PROBS];
  int n_probs, n_tiles, K;
  const int* tok_meta;
  float* scratch;          // [units][2 pieces][2 CTAs][BM x BN]
  unsigned* counters;      // [n_tiles][2 CTAs], zero between launches
  int* status;
};

template <typename T>
__global__ void __launch_bounds__(THREADS, 1) wgrad_group_kernel(const __grid_constant__ Maps maps, const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmem_full_bar = empty_bar + STAGES;     // [2]
  uint64_t* tmem_empty_bar = tmem_full_bar + 2;     // [2]
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(tmem_empty_bar + 2);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);
  volatile int* s_last = s_abort + 1;
  const int warp = tc::warp_id(), lane = threadIdx.x & 31;
  const uint32_t rank = tc::cluster_ctarank();
  const int unit = (int)(blockIdx.x >> 1), n_units = (int)(gridDim.x >> 1);
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { tc::mbar_init(full_bar + s, 1); tc::mbar_init(empty_bar + s, 1); }
    for (int a = 0; a < 2; ++a) { tc::mbar_init(tmem_full_bar + a, 1); tc::mbar_init(tmem_empty_bar + a, 2 * EPI_WARPS); }
    *s_abort = 0;
    *s_last = 0;
    tc::fence_barrier_init();
  }
  if (warp == 1) tc::tmem_alloc_pair(tmem_ptr_smem, TMEM_COLS);
  tc::tc_fence_before();
  __syncthreads();
  tc::cluster_sync_all();
  tc::tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  bool aborted = false;
  grid_dep_wait();
  grid_dep_launch();
  // Work of this unit: a run [x0, x1) of the line of n_cut * kb (tile, k block) pairs of the first n_cut tiles, then every
  // n_units-th of the other tiles as a whole
  const int rows = p.tok_meta != nullptr ? __ldcg(p.tok_meta + TOK_ROWS) : p.K;
  const int kb = (rows + BK - 1) / BK;
  const int n_cut = p.n_tiles % n_units;
  const int total = n_cut * kb;
  const int run = max(min(MIN_RUN, kb), (total + n_units - 1) / n_units);
  const int x0 = min(total, unit * run), x1 = min(total, x0 + run);
  // The pieces of the run, then the whole tiles: tile, k blocks [k0, k1); x advances along the line, then by whole tiles
  const int x_end = x1 + (p.n_tiles - n_cut) / n_units;
  const auto piece = [&](int x, int& tile, int& k0, int& k1) -> int {     // returns the x that follows
    if (x < x1) {
      tile = x / kb; k0 = x - tile * kb; k1 = min(kb, k0 + x1 - x);
      return x + (k1 - k0);
    }
    tile = n_cut + (x - x1) * n_units + unit; k0 = 0; k1 = kb;
    return x + 1;
  };
  const auto find = [&](int tile, int& m0, int& n0) -> int {
    int i = 0;
    while (i + 1 < p.n_probs && tile >= p.prob[i + 1].first) ++i;
    const int t = tile - p.prob[i].first, n_n = p.prob[i].n_n;
    m0 = (t / n_n) * (2 * BM) + (int)rank * BM;
    n0 = (t % n_n) * BN;
    return i;
  };

  if (warp == 0 && tc::elect_one()) {
    int s = 0;
    uint32_t ph = 0;
    for (int x = x0; x < x_end && !aborted;) {
      int tile, k0, k1, m0, n0;
      x = piece(x, tile, k0, k1);
      const int i = find(tile, m0, n0);
      const int nb = n0 + (int)rank * (BN / 2);
      for (int k = k0; k < k1; ++k, s = (s + 1 == STAGES ? 0 : s + 1), ph ^= (s == 0 ? 1u : 0u)) {
        if (!tc::mbar_wait(empty_bar + s, ph ^ 1, aborted, p.status, tc::SITE_EMPTY, k)) break;
        uint8_t* sA = smem + s * STAGE;
        uint8_t* sB = sA + BM * BK * 2;
        const uint32_t lbar = tc::leader_addr(tc::smem_u32(full_bar + s));
        if (rank == 0) tc::mbar_expect_tx(full_bar + s, 2 * STAGE);
        tc::tma_load_2d_pair(sA, &maps.a[i], lbar, m0, k * BK);
        tc::tma_load_2d_pair(sA + 8192, &maps.a[i], lbar, m0 + 64, k * BK);
        tc::tma_load_2d_pair(sB, &maps.b[i], lbar, nb, k * BK);
        tc::tma_load_2d_pair(sB + 8192, &maps.b[i], lbar, nb + 64, k * BK);
      }
    }
  } else if (warp == 1 && rank == 0 && tc::elect_one()) {
    constexpr int FMT = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
    const uint32_t idesc = tc::make_idesc(FMT, 1, 1, 2 * BM, BN);
    int s = 0, t_local = 0;
    uint32_t ph = 0;
    for (int x = x0; x < x_end && !aborted; ++t_local) {
      int tile, k0, k1;
      x = piece(x, tile, k0, k1);
      const int buf = t_local & 1;
      if (!tc::mbar_wait(tmem_empty_bar + buf, (uint32_t)((t_local >> 1) & 1) ^ 1u, aborted, p.status, tc::SITE_TMEM_EMPTY, tile)) break;
      tc::tc_fence_after();
      const uint32_t d = tmem_base + (uint32_t)buf * 256u;
      for (int k = k0; k < k1; ++k, s = (s + 1 == STAGES ? 0 : s + 1), ph ^= (s == 0 ? 1u : 0u)) {
        if (!tc::mbar_wait(full_bar + s, ph, aborted, p.status, tc::SITE_FULL, k)) break;
        tc::tc_fence_after();
        const uint32_t sA = tc::smem_u32(smem + s * STAGE), sB = sA + BM * BK * 2;
#pragma unroll
        for (int q = 0; q < BK / 16; ++q)
          tc::umma_f16_pair(d, tc::make_smem_desc(sA + q * 2048, 8192, 1024), tc::make_smem_desc(sB + q * 2048, 8192, 1024), idesc,
                            (k > k0 || q > 0) ? 1u : 0u);
        tc::umma_commit_pair(empty_bar + s);
      }
      if (aborted) break;
      tc::umma_commit_pair(tmem_full_bar + buf);
    }
  } else if (warp >= 2) {
    const int quarter = warp & 3, g = (warp - 2) >> 2, r = quarter * 32 + lane, et = (int)threadIdx.x - 64;
    int t_local = 0;
    for (int x = x0; x < x_end; ++t_local) {
      int tile, k0, k1, m0, n0;
      x = piece(x, tile, k0, k1);
      const Prob& pr = p.prob[find(tile, m0, n0)];
      const int buf = t_local & 1;
      const bool whole = k0 == 0 && k1 == kb;
      const int u_lo = (int)(((long long)tile * kb) / run), u_hi = (int)(((long long)tile * kb + kb - 1) / run);
      unsigned* cnt = p.counters + 2 * tile + rank;
      const unsigned others = (unsigned)(u_hi - u_lo);
      if (!tc::mbar_wait(tmem_full_bar + buf, (uint32_t)((t_local >> 1) & 1), aborted, p.status, tc::SITE_TMEM_FULL, tile)) *s_abort = 1;
      if (!whole && et == 0) {
        // if every other piece of the tile is in the scratch already, this one needs no place there
        unsigned c;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(cnt) : "memory");
        *s_last = c == others ? 1 : 0;
      }
      asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");
      if (*s_abort) break;                                   // the same answer in every epilogue warp
      tc::tc_fence_after();
      const uint32_t tacc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)buf * 256u + (uint32_t)(g * 64);
      bool last = whole || *s_last != 0;
      if (!last) {
        // piece 0 of a unit is the tile its run starts in, piece 1 the one its run ends in
        float4* out = reinterpret_cast<float4*>(p.scratch + (size_t)((unit * 2 + (t_local > 0 ? 1 : 0)) * 2 + (int)rank) * PIECE_FLOATS) + et;
#pragma unroll
        for (int hc = 0; hc < 2; ++hc) {
          float v[32];
          tc::tmem_ld32(tacc + 32 * hc, v);
#pragma unroll
          for (int q = 0; q < 8; ++q)
            __stcg(out + (size_t)(8 * hc + q) * EPI_THREADS, make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]));
        }
        __threadfence();
        asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");
        if (et == 0) *s_last = atomicAdd(cnt, 1u) == others ? 1 : 0;
        asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");
        last = *s_last != 0;
      }
      if (last) {
        __threadfence();
        const int row = m0 + r;
        uint16_t* crow = reinterpret_cast<uint16_t*>(pr.C) + (size_t)row * pr.ldc;
#pragma unroll
        for (int hc = 0; hc < 2; ++hc) {
          float v[32];
          tc::tmem_ld32(tacc + 32 * hc, v);
          if (!whole) {
            for (int u = u_lo; u <= u_hi; ++u) {
              if (u == unit) continue;
              // the tile is unit u's first one unless its run began in an earlier tile
              const int piece = u * run >= tile * kb ? 0 : 1;
              const float4* in = reinterpret_cast<const float4*>(p.scratch + (size_t)((u * 2 + piece) * 2 + (int)rank) * PIECE_FLOATS) + et;
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                const float4 f = __ldcg(in + (size_t)(8 * hc + q) * EPI_THREADS);
                v[4 * q] += f.x; v[4 * q + 1] += f.y; v[4 * q + 2] += f.z; v[4 * q + 3] += f.w;
              }
            }
          }
          if (row < pr.M) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int c = n0 + g * 64 + 32 * hc + 8 * q;
              if (c < pr.N) *reinterpret_cast<uint4*>(crow + c) = pack16x8<T>(v + 8 * q);
            }
          }
        }
        if (!whole && et == 0) *cnt = 0u;
      }
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive_leader(tmem_empty_bar + buf);
      // s_last is written again for the next piece only after every warp has read it
      if (!whole) asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::cluster_sync_all();
  if (warp == 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

template <typename T>
static int launch(const Maps& m, const Params& p, cudaStream_t st) {
  auto k = wgrad_group_kernel<T>;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess) return -5;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sm_count() / 2 * 2, 1, 1);
  cfg.blockDim = dim3(THREADS, 1, 1);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_flag() ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k, m, p);
  return e == cudaSuccess ? 0 : (int)e;
}

}  // namespace wg
}  // namespace rb

using namespace rb;

// Bytes of scratch that rb_wgrad_group needs.  It also needs two (zeroed) counter words per 256 x 256 tile of its problems.
RB_API long long rb_wgrad_group_scratch_bytes(void) { return (long long)(sm_count() / 2) * 4 * (long long)wg::PIECE_FLOATS * 4; }

// dW_i [M_i, ldc_i >= N_i] = A_i [K, lda_i >= M_i]^T B_i [K, ldb_i >= N_i] for i < n.  dims: per problem M, N, lda, ldb, ldc (all
// multiples of 8); K token rows, or with tok_meta (token_map.cuh) at most K.
RB_API int rb_wgrad_group(int dtype, int n, const void* const* A, const void* const* B, void* const* C, const int* dims, int K,
                          const int* tok_meta, float* scratch, unsigned* counters, int n_counters, int* status, cudaStream_t st) {
  if (dtype != RB_BF16 && dtype != RB_F16) return -1;
  if (n < 1 || n > wg::MAX_PROBS || K < 1 || scratch == nullptr || counters == nullptr || sm_count() < 2) return -3;
  wg::Maps m;
  wg::Params p{};
  int tiles = 0;
  for (int i = 0; i < n; ++i) {
    const int M = dims[5 * i], N = dims[5 * i + 1], lda = dims[5 * i + 2], ldb = dims[5 * i + 3], ldc = dims[5 * i + 4];
    if (M < 1 || N < 1 || M % 8 || N % 8 || lda % 8 || ldb % 8 || ldc % 8 || (reinterpret_cast<uintptr_t>(C[i]) & 15)) return -3;
    int rc = tc::make_tmap_2d(&m.a[i], A[i], K, M, lda, 64, 64, dtype == RB_BF16);
    if (rc) return rc;
    rc = tc::make_tmap_2d(&m.b[i], B[i], K, N, ldb, 64, 64, dtype == RB_BF16);
    if (rc) return rc;
    const int n_n = (N + wg::BN - 1) / wg::BN;
    p.prob[i] = wg::Prob{M, N, n_n, tiles, C[i], ldc};
    tiles += ((M + 2 * wg::BM - 1) / (2 * wg::BM)) * n_n;
  }
  for (int i = n; i < wg::MAX_PROBS; ++i) { m.a[i] = m.a[0]; m.b[i] = m.b[0]; p.prob[i] = p.prob[0]; }
  if (2 * tiles > n_counters || (long long)tiles * ((K + wg::BK - 1) / wg::BK) > (1LL << 30)) return -3;
  p.n_probs = n; p.n_tiles = tiles; p.K = K; p.tok_meta = tok_meta; p.scratch = scratch; p.counters = counters; p.status = status;
  const int rc = dtype == RB_BF16 ? wg::launch<__nv_bfloat16>(m, p, st) : wg::launch<__half>(m, p, st);
  if (rc) return rc;
  RB_LAUNCH_CHECK();
  return 0;
}
