// A step's inputs from page-locked host memory to their device buffers in one launch: up to four int32 arrays (token ids, mask,
// rows and labels of the positives), the hyper-parameter block and the number of positives.
//
// As five copies and a fill these took 40 us at the head of every training step (1 to 4 us each and 2 us between them), whatever
// their size: 256 x 32 tokens are 67 KB.  The kernel reads the host arrays over the bus directly, 16 bytes per thread and
// access where both sides are aligned, with everything in flight at once; the hyper-parameters travel as kernel arguments.
// What is left is the bus: 7.6 us for 5 KB, 8.4 for 67 KB, 12.4 for 300 KB.  Steps of 32 x 32 tokens with a two-layer encoder
// 224 -> 212 us, 256 x 32 tokens 2.39 -> 2.36 ms.
#include "common.cuh"

namespace rb {
constexpr int STAGE_SEGS = 4, STAGE_HP = 8;
struct StageArgs {
  const int* src[STAGE_SEGS];
  int* dst[STAGE_SEGS];
  int n[STAGE_SEGS];             // 32-bit words
  float hp[STAGE_HP];
  float* hp_dst;
  int* nnz_dst;
  int nnz;
};

__global__ void __launch_bounds__(256) stage_inputs_kernel(const StageArgs a) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  if (t < STAGE_HP && a.hp_dst != nullptr) a.hp_dst[t] = a.hp[t];
  if (t == 0 && a.nnz_dst != nullptr) *a.nnz_dst = a.nnz;
#pragma unroll
  for (int s = 0; s < STAGE_SEGS; ++s) {
    const int n = a.n[s];
    const bool wide = ((reinterpret_cast<uintptr_t>(a.src[s]) | reinterpret_cast<uintptr_t>(a.dst[s])) & 15) == 0;
    const int nv = wide ? n / 4 : 0;
    for (int i = t; i < nv; i += step) reinterpret_cast<int4*>(a.dst[s])[i] = reinterpret_cast<const int4*>(a.src[s])[i];
    for (int i = 4 * nv + t; i < n; i += step) a.dst[s][i] = a.src[s][i];
  }
}
}  // namespace rb

using namespace rb;

// 1: what was recorded before the event has run; 0: not yet (wait == 0); else minus a CUDA error.  This thread's part in the capture
// of another thread is relaxed for the call: a query or a wait of this kind ends a capture in the default (global) mode.
RB_API int rb_event_passed(cudaEvent_t ev, int wait) {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaError_t e = cudaThreadExchangeStreamCaptureMode(&mode);
  if (e != cudaSuccess) return -(int)e;
  e = wait ? cudaEventSynchronize(ev) : cudaEventQuery(ev);
  const cudaError_t back = cudaThreadExchangeStreamCaptureMode(&mode);
  if (e == cudaErrorNotReady) { (void)cudaGetLastError(); return back == cudaSuccess ? 0 : -(int)back; }
  if (e == cudaSuccess) e = back;
  return e == cudaSuccess ? 1 : -(int)e;
}

// src[i]: page-locked host memory, n[i] words, i < n_segs <= 4.  hp_host (nullable): STAGE_HP floats, read here; nnz_dst nullable.
RB_API int rb_stage_inputs(int n_segs, const void* const* src, void* const* dst, const int* n, const float* hp_host, float* hp_dst,
                           int* nnz_dst, int nnz, cudaStream_t st) {
  if (n_segs < 0 || n_segs > STAGE_SEGS) return -3;
  StageArgs a{};
  long long words = STAGE_HP * 4;
  for (int i = 0; i < n_segs; ++i) {
    if (n[i] < 0 || (n[i] > 0 && (src[i] == nullptr || dst[i] == nullptr))) return -3;
    a.src[i] = static_cast<const int*>(src[i]);
    a.dst[i] = static_cast<int*>(dst[i]);
    a.n[i] = n[i];
    words = words > n[i] ? words : n[i];
  }
  if (hp_host != nullptr) {
    for (int i = 0; i < STAGE_HP; ++i) a.hp[i] = hp_host[i];
    a.hp_dst = hp_dst;
  }
  a.nnz_dst = nnz_dst;
  a.nnz = nnz;
  long long blocks = (words / 4 + 255) / 256;               // one access per thread and array, up to a few CTAs per SM
  if (blocks > sm_count() * 4) blocks = sm_count() * 4;
  stage_inputs_kernel<<<(int)(blocks < 1 ? 1 : blocks), 256, 0, st>>>(a);
  RB_LAUNCH_CHECK();
  return 0;
}
