// Encoder optimizer kernels over flat buffers:
//   grad_check     raises the found-inf flag if any gradient element is non-finite
//   adamw          fused AdamW (decoupled decay) with gradient unscaling, bias correction, the skip on
//                  found-inf, and the write of the low-precision compute copy of the parameters
//   scaler_update  loss-scale state machine (growth / back-off), Adam step counter, flag reset
// They replace apex FusedAdam + torch GradScaler's foreach kernels as the reference uses them
// (main.py:180-181, dl_base.py:372-374).  All step-varying scalars are read from the device-resident
// hyper-parameter block, so the launches can be replayed from a CUDA graph with no host round trip.
#include "common.cuh"

namespace rb {

template <typename T>
__global__ void __launch_bounds__(256) grad_check_kernel(const T* __restrict__ g, size_t n_vec, float* __restrict__ hp) {
  bool bad = false;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_vec; i += (size_t)gridDim.x * blockDim.x) {
    float a[8];
    load8(g + i * 8, a);
#pragma unroll
    for (int j = 0; j < 8; ++j) bad |= !isfinite(a[j]);
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) hp[HP_FOUND_INF] = 1.0f;
}

// 8 floats in one 256-bit access where the buffer starts on a 32-byte boundary (the flat buffers do), two otherwise.  AdamW is
// bound by HBM (28 bytes per parameter): 66.4 M parameters 320 -> 301 us (5.8 -> 6.2 TB/s) with the wide accesses.
template <bool WIDE> __device__ __forceinline__ void load8w(const float* p, float (&v)[8]) {
  if (WIDE)
    asm volatile("ld.global.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(p) : "memory");
  else load8(p, v);
}
template <bool WIDE> __device__ __forceinline__ void store8w(float* p, const float (&v)[8]) {
  if (WIDE)
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
  else store8(p, v);
}

template <typename TG, typename TP, bool WIDE>
__global__ void __launch_bounds__(256) adamw_kernel(float* __restrict__ p32, float* __restrict__ m, float* __restrict__ v,
                                                    const TG* __restrict__ g, TP* __restrict__ p16, size_t n_vec,
                                                    size_t n_decay, const float* __restrict__ hp, float beta1, float beta2,
                                                    float eps, float wd, float grad_mult) {
  if (hp[HP_FOUND_INF] != 0.f) return;
  const float lr = hp[HP_LR_ENC];
  const float step = hp[HP_ADAM_STEP] + 1.0f;
  const float inv_scale = hp[HP_INV_SCALE] * grad_mult;
  const float bc1 = 1.f - powf(beta1, step);
  const float bc2 = 1.f - powf(beta2, step);
  const float inv_bc1 = 1.f / bc1, inv_bc2 = 1.f / bc2;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_vec; i += (size_t)gridDim.x * blockDim.x) {
    const size_t e = i * 8;
    float gg[8], pp[8], mm[8], vv[8];
    load8(g + e, gg);
    load8w<WIDE>(p32 + e, pp);
    load8w<WIDE>(m + e, mm);
    load8w<WIDE>(v + e, vv);
    const float decay = (e < n_decay) ? 1.f - lr * wd : 1.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float gr = gg[j] * inv_scale;
      mm[j] = beta1 * mm[j] + (1.f - beta1) * gr;
      vv[j] = beta2 * vv[j] + (1.f - beta2) * gr * gr;
      const float denom = sqrtf(vv[j] * inv_bc2) + eps;
      pp[j] = pp[j] * decay - lr * (mm[j] * inv_bc1) / denom;
    }
    store8w<WIDE>(p32 + e, pp);
    store8w<WIDE>(m + e, mm);
    store8w<WIDE>(v + e, vv);
    if (p16 != nullptr) store8(p16 + e, pp);
  }
}

__global__ void scaler_update_kernel(float* hp, int enabled, float growth, float backoff, float interval) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  if (hp[HP_FOUND_INF] != 0.f) {
    if (enabled) hp[HP_SCALE] *= backoff;
    hp[HP_TRACKER] = 0.f;
  } else {
    hp[HP_ADAM_STEP] += 1.f;
    hp[HP_TRACKER] += 1.f;
    if (enabled && hp[HP_TRACKER] >= interval) {
      hp[HP_SCALE] *= growth;
      hp[HP_TRACKER] = 0.f;
    }
  }
  hp[HP_INV_SCALE] = 1.f / hp[HP_SCALE];
  hp[HP_FOUND_INF] = 0.f;
}

}  // namespace rb

using namespace rb;

static int flat_blocks(size_t n_vec) {
  size_t b = (n_vec + 255) / 256;
  return (int)(b > rb::sm_count() * 8 ? rb::sm_count() * 8 : (b == 0 ? 1 : b));
}

RB_API int rb_grad_check(int dtype, const void* g, long long n, float* hp, cudaStream_t st) {
  if (n % 8) return -3;
  const size_t n_vec = (size_t)n / 8;
  switch (dtype) {
    case RB_F32: grad_check_kernel<float><<<flat_blocks(n_vec), 256, 0, st>>>((const float*)g, n_vec, hp); break;
    case RB_BF16: grad_check_kernel<__nv_bfloat16><<<flat_blocks(n_vec), 256, 0, st>>>((const __nv_bfloat16*)g, n_vec, hp); break;
    case RB_F16: grad_check_kernel<__half><<<flat_blocks(n_vec), 256, 0, st>>>((const __half*)g, n_vec, hp); break;
    default: return -1;
  }
  RB_LAUNCH_CHECK();
  return 0;
}

// p16 may be null (fp32 encoder: the master buffer is the compute copy)
RB_API int rb_adamw(int dtype, float* p32, float* m, float* v, const void* g, void* p16, long long n, long long n_decay,
                    const float* hp, float beta1, float beta2, float eps, float wd, float grad_mult, cudaStream_t st) {
  if (n % 8 || n_decay % 8) return -3;
  const size_t n_vec = (size_t)n / 8;
  const int blocks = flat_blocks(n_vec);
  const bool wide = ((reinterpret_cast<uintptr_t>(p32) | reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v)) & 31) == 0;
#define RB_ADAMW(T, W) adamw_kernel<T, T, W><<<blocks, 256, 0, st>>>(p32, m, v, (const T*)g, (T*)p16, n_vec, (size_t)n_decay, hp, beta1, beta2, eps, wd, grad_mult)
  switch (dtype) {
    case RB_F32: if (wide) RB_ADAMW(float, true); else RB_ADAMW(float, false); break;
    case RB_BF16: if (wide) RB_ADAMW(__nv_bfloat16, true); else RB_ADAMW(__nv_bfloat16, false); break;
    case RB_F16: if (wide) RB_ADAMW(__half, true); else RB_ADAMW(__half, false); break;
    default: return -1;
  }
#undef RB_ADAMW
  RB_LAUNCH_CHECK();
  return 0;
}

RB_API int rb_scaler_update(float* hp, int enabled, float growth, float backoff, int interval, cudaStream_t st) {
  scaler_update_kernel<<<1, 32, 0, st>>>(hp, enabled, growth, backoff, (float)interval);
  RB_LAUNCH_CHECK();
  return 0;
}
