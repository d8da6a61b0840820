// Shared device helpers for the sm_100a kernels of renee_b200.
#pragma once
#include <type_traits>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#define RB_API extern "C" __attribute__((visibility("default")))

// dtype codes shared with the Python side (renee_b200/ops/cuda.py)
enum RbDtype : int { RB_F32 = 0, RB_BF16 = 1, RB_F16 = 2 };

// Slots of the device-resident hyper-parameter block (renee_b200/optim/hparams.py)
enum RbHp : int {
  HP_LR_XFC = 0, HP_LR_ENC = 1, HP_SEED = 2,
  HP_SCALE = 8, HP_INV_SCALE = 9, HP_FOUND_INF = 10, HP_TRACKER = 11, HP_ADAM_STEP = 12
};

#define RB_LAUNCH_CHECK() do { cudaError_t e_ = cudaGetLastError(); if (e_ != cudaSuccess) return (int)e_; } while (0)

namespace rb {

__device__ __forceinline__ float to_f(float x) { return x; }
__device__ __forceinline__ float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }
__device__ __forceinline__ float to_f(__half x) { return __half2float(x); }

template <typename T> __device__ __forceinline__ T from_f(float x);
template <> __device__ __forceinline__ float from_f<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ __forceinline__ __half from_f<__half>(float x) { return __float2half_rn(x); }

// 8 floats rounded to a 16-bit type, two per conversion instruction
template <typename T> __device__ __forceinline__ uint4 pack16x8(const float* v) {
  uint4 raw;
  uint32_t* w = reinterpret_cast<uint32_t*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&h);
    } else {
      const __half2 h = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
  }
  return raw;
}

// 8 consecutive elements of T, moved with the widest aligned access available
template <typename T> struct Vec8 {
  T v[8];
};

template <typename T>
__device__ __forceinline__ void load8(const T* __restrict__ p, float (&out)[8]) {
  if constexpr (sizeof(T) == 2) {
    uint4 raw = *reinterpret_cast<const uint4*>(p);
    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = to_f(e[i]);
  } else {
    float4 a = *reinterpret_cast<const float4*>(p);
    float4 b = *reinterpret_cast<const float4*>(p + 4);
    out[0] = a.x; out[1] = a.y; out[2] = a.z; out[3] = a.w;
    out[4] = b.x; out[5] = b.y; out[6] = b.z; out[7] = b.w;
  }
}

template <typename T>
__device__ __forceinline__ void store8(T* __restrict__ p, const float (&in)[8]) {
  if constexpr (sizeof(T) == 2) {
    *reinterpret_cast<uint4*>(p) = pack16x8<T>(in);
  } else {
    *reinterpret_cast<float4*>(p) = make_float4(in[0], in[1], in[2], in[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(in[4], in[5], in[6], in[7]);
  }
}

// 8 elements kept in their storage format (4 registers for 16-bit types) and expanded on demand:
// lets a kernel hold several vectors across a reduction without paying 8 registers per vector.
template <typename T> struct Raw8 { uint4 v; };
template <> struct Raw8<float> { float4 a, b; };

template <typename T> __device__ __forceinline__ Raw8<T> load_raw8(const T* __restrict__ p) {
  Raw8<T> r;
  r.v = *reinterpret_cast<const uint4*>(p);
  return r;
}
template <> __device__ __forceinline__ Raw8<float> load_raw8<float>(const float* __restrict__ p) {
  Raw8<float> r;
  r.a = *reinterpret_cast<const float4*>(p);
  r.b = *reinterpret_cast<const float4*>(p + 4);
  return r;
}
template <typename T> __device__ __forceinline__ void unpack8(const Raw8<T>& r, float (&out)[8]) {
  const T* e = reinterpret_cast<const T*>(&r.v);
#pragma unroll
  for (int i = 0; i < 8; ++i) out[i] = to_f(e[i]);
}
template <> __device__ __forceinline__ void unpack8<float>(const Raw8<float>& r, float (&out)[8]) {
  out[0] = r.a.x; out[1] = r.a.y; out[2] = r.a.z; out[3] = r.a.w;
  out[4] = r.b.x; out[5] = r.b.y; out[6] = r.b.z; out[7] = r.b.w;
}

// Rounds through T (what a store followed by a load would give)
template <typename T> __device__ __forceinline__ float round_through(float x) { return to_f(from_f<T>(x)); }

// fp32 -> fp16 with stochastic rounding: add uniform noise below the 13 mantissa bits fp16 drops, then
// truncate.  Unbiased for values in fp16's normal range, which keeps updates smaller than half an ulp
// of W from being lost systematically late in the learning-rate schedule.
// Two neighbours at once, packed; rx and ry are the random words of the two (fp16 drops 13 bits, bf16 16).  The masking
// keeps an infinity one; the conversion truncates what lies below fp16's range.
template <typename T> __device__ __forceinline__ uint32_t sr_pack2(float x, float y, uint32_t rx, uint32_t ry) {
  constexpr uint32_t kNoise = std::is_same<T, __half>::value ? 0x1FFFu : 0xFFFFu;
  const float a = __uint_as_float((__float_as_uint(x) + (rx & kNoise)) & ~kNoise);
  const float b = __uint_as_float((__float_as_uint(y) + (ry & kNoise)) & ~kNoise);
  uint32_t r;
  if (std::is_same<T, __half>::value) asm("cvt.rz.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  else asm("cvt.rz.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// One 16-byte reduction instead of four 4-byte ones (p must be 16-byte aligned)
__device__ __forceinline__ void red_add_f32x4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// Two fp32 values per instruction (add / mul / fma .f32x2): IEEE arithmetic, half the issue slots.
struct F2 { unsigned long long v; };
__device__ __forceinline__ F2 f2(float a, float b) { F2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
__device__ __forceinline__ void f2_get(F2 x, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v)); }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { F2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { F2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

// Exact (erf) GELU and its derivative for two values, by the tail of the normal distribution: |z|, -Q(|z|) = -0.5 erfc(|z| /
// sqrt 2) and e = exp(-z^2 / 2).  erfc(x) = t (a1 + t (a2 + t (a3 + t (a4 + t a5)))) exp(-x^2) with t = 1 / (1 + p x)
// (Abramowitz & Stegun 7.1.26, |error| <= 1.5e-7): the negative tail comes out of the product directly, without the
// cancellation of 1 + erf.  The factors are moved: ax = |z| sqrt(log2(e) / 2), so that the exponential is one instruction, and
// 0.5 and the sign sit in the coefficients.  GELU and its gradient then need no choice between Q and 1 - Q (which was 4 of 25
// instructions per pair; the kernels around them are bound by instruction issue rather than by HBM):
//   gelu(z) = z [z >= 0] - |z| Q      gelu'(z) = [z >= 0] - sign(z) Q + z e / sqrt(2 pi)
// At the infinities as torch: gelu(inf) = inf; gelu(-inf) and both derivatives are 0 times infinity, a NaN, so that a
// pre-activation that has overflowed 16 bits is seen behind the FFN whatever its sign (max(z, 0) made a 0 of -inf; the kernels of
// their own at 4320 x 3072 in fp16: forward 12.4 -> 13.1 us, with the sign test of the derivative backward 24.5 -> 23.8).
__device__ __forceinline__ F2 normal_tail2(F2 z, F2& az, F2& e) {
  float z0, z1;
  f2_get(z, z0, z1);
  // a finite bound, so that |z| Q of an infinite z is 0 (a NaN stays one)
  float a0, a1;
  asm("min.NaN.f32 %0, %1, 0f7F7FFFFF;" : "=f"(a0) : "f"(fabsf(z0)));
  asm("min.NaN.f32 %0, %1, 0f7F7FFFFF;" : "=f"(a1) : "f"(fabsf(z1)));
  az = f2(a0, a1);
  const F2 ax = az * f2(0.84932180028801904f);
  float d0, d1, t0, t1, e0, e1;
  f2_get(f2_fma(f2(0.3275911f * 0.83255461115769776f), ax, f2(1.f)), d0, d1);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t0) : "f"(d0));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t1) : "f"(d1));
  const F2 t = f2(t0, t1);
  F2 p = f2(-0.5f * 1.061405429f);
  p = f2_fma(p, t, f2(0.5f * 1.453152027f));
  p = f2_fma(p, t, f2(-0.5f * 1.421413741f));
  p = f2_fma(p, t, f2(0.5f * 0.284496736f));
  p = f2_fma(p, t, f2(-0.5f * 0.254829592f));
  f2_get(ax * ax, e0, e1);
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(-e0));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(-e1));
  e = f2(e0, e1);
  return p * t * e;
}
__device__ __forceinline__ F2 gelu2(F2 z) {
  float z0, z1;
  f2_get(z, z0, z1);
  F2 az, e;
  const F2 nq = normal_tail2(z, az, e);
  return f2_fma(az, nq, z * f2(z0 < 0.f ? 0.f : 1.f, z1 < 0.f ? 0.f : 1.f));
}
__device__ __forceinline__ F2 gelu_grad2(F2 z) {
  float z0, z1, q0, q1;
  f2_get(z, z0, z1);
  F2 az, e;
  f2_get(normal_tail2(z, az, e), q0, q1);
  // the step and the tail's sign by one comparison: by copysign, the derivative at -0 was 1.5
  const F2 cdf = f2(z0 < 0.f ? 0.f : 1.f, z1 < 0.f ? 0.f : 1.f) + f2(z0 < 0.f ? -q0 : q0, z1 < 0.f ? -q1 : q1);
  return f2_fma(z * f2(0.39894228040143268f), e, cdf);
}

// Number of SMs of the current device (queried once per process; all GPUs of a job are alike)
inline int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1)
      n = 1;
  }
  return n;
}

// Programmatic dependent launch: a kernel launched with the programmatic-stream-serialization attribute may
// start (set up barriers, allocate TMEM, fetch descriptors) while its predecessor in the stream is still running,
// once every CTA of the predecessor has executed launch_dependents (or exited); it must execute grid_dep_wait
// before its first access to global memory, which blocks until the predecessor has completed and its writes are
// visible.  Without the launch attribute both instructions do nothing.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Host side: one switch for the whole library and a launch helper that sets the attribute.  A kernel launched
// through launch_pdl MUST execute grid_dep_wait() before its first access to global memory.
inline int& pdl_flag() {
  static int on = 1;
  return on;
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                              Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_flag() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// Counter-based dropout RNG; must stay bit-identical to renee_b200/ops/rng.py::mix32
__device__ __forceinline__ uint32_t mix32(uint32_t seed, uint32_t stream, uint32_t idx) {
  uint32_t x = idx * 0x9E3779B1u + seed;
  x ^= x >> 16; x *= 0x85EBCA6Bu; x ^= x >> 13; x *= 0xC2B2AE35u; x ^= x >> 16;
  x += stream * 0x27D4EB2Fu;
  x ^= x >> 15; x *= 0x2C1B3C6Du; x ^= x >> 12; x *= 0x297A2D39u; x ^= x >> 15;
  return x;
}
// The rule is (h >> 8) / 2^24 >= p in reals.  Scaling p by 2^24 is exact, so comparing the 24-bit integer with
// ceil(p 2^24), which the compiler keeps outside the loop, is the same decision without an integer-to-float conversion
// per element: those run at 16 per clock and SM and bounded the LayerNorm backward and the attention kernels.
__device__ __forceinline__ bool keep(uint32_t seed, uint32_t stream, uint32_t idx, float p) {
  return (mix32(seed, stream, idx) >> 8) >= (uint32_t)ceilf(p * 16777216.0f);
}

}  // namespace rb
