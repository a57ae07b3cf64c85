// Shared device/host helpers for the gdn2_b200 kernels (sm_100a only).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/gdn2_b200.h"

namespace gdn2 {

constexpr int kDim = GDN2_DIM;
constexpr int kTokenInterval = GDN2_TOKEN_INTERVAL;

// ---- typed scalar loads / stores through float --------------------------------
// bf16 -> fp32 is a 16-bit shift (exact); spelled out so that it runs on the integer pipe
__device__ __forceinline__ float to_float(__nv_bfloat16 x) {
  return __uint_as_float(uint32_t(__bfloat16_as_ushort(x)) << 16);
}
__device__ __forceinline__ float to_float(__half x) { return __half2float(x); }
__device__ __forceinline__ float to_float(float x) { return x; }

template <typename T>
__device__ __forceinline__ T from_float(float x);
template <>
__device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float x) {
  return __float2bfloat16_rn(x);
}
template <>
__device__ __forceinline__ __half from_float<__half>(float x) {
  return __float2half_rn(x);
}
template <>
__device__ __forceinline__ float from_float<float>(float x) {
  return x;
}

// two values converted at once (one instruction for both)
template <typename T> struct Pair;
template <> struct Pair<__nv_bfloat16> {
  using type = __nv_bfloat162;
  __device__ static __forceinline__ type make(float lo, float hi) { return __floats2bfloat162_rn(lo, hi); }
};
template <> struct Pair<__half> {
  using type = __half2;
  __device__ static __forceinline__ type make(float lo, float hi) { return __floats2half2_rn(lo, hi); }
};

template <typename T>
__device__ __forceinline__ float ldf(const void* base, int64_t index) {
  return to_float(static_cast<const T*>(base)[index]);
}
template <typename T>
__device__ __forceinline__ void stf(void* base, int64_t index, float value) {
  static_cast<T*>(base)[index] = from_float<T>(value);
}

// ---- state tile I/O: 128-bit when the base is 16-byte aligned ------------------
__device__ __forceinline__ void load4(const float* p, bool vec, float (&x)[4]) {
  if (vec) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w;
  } else {
    x[0] = p[0]; x[1] = p[1]; x[2] = p[2]; x[3] = p[3];
  }
}
__device__ __forceinline__ void store4(float* p, bool vec, const float (&x)[4]) {
  if (vec) {
    *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
  } else {
    p[0] = x[0]; p[1] = x[1]; p[2] = x[2]; p[3] = x[3];
  }
}

// 4 consecutive sequence elements, kept packed until they are needed (a prefetch then costs 2 or 4
// registers per group instead of 4 floats)
template <typename T> struct Raw4 { using type = uint2; };
template <> struct Raw4<float> { using type = float4; };
template <typename T>
__device__ __forceinline__ typename Raw4<T>::type load4_raw(const void* base, int64_t idx) {
  return *reinterpret_cast<const typename Raw4<T>::type*>(static_cast<const T*>(base) + idx);
}
template <typename T>
__device__ __forceinline__ void unpack4(typename Raw4<T>::type raw, float (&out)[4]);
template <>
__device__ __forceinline__ void unpack4<__nv_bfloat16>(uint2 raw, float (&out)[4]) {
  out[0] = __uint_as_float(raw.x << 16); out[1] = __uint_as_float(raw.x & 0xffff0000u);
  out[2] = __uint_as_float(raw.y << 16); out[3] = __uint_as_float(raw.y & 0xffff0000u);
}
template <>
__device__ __forceinline__ void unpack4<__half>(uint2 raw, float (&out)[4]) {
  const __half2* hh = reinterpret_cast<const __half2*>(&raw);
  const float2 a = __half22float2(hh[0]), c = __half22float2(hh[1]);
  out[0] = a.x; out[1] = a.y; out[2] = c.x; out[3] = c.y;
}
template <>
__device__ __forceinline__ void unpack4<float>(float4 raw, float (&out)[4]) {
  out[0] = raw.x; out[1] = raw.y; out[2] = raw.z; out[3] = raw.w;
}

// two of them
template <typename T> struct Raw2 { using type = uint32_t; };
template <> struct Raw2<float> { using type = float2; };
template <typename T>
__device__ __forceinline__ float2 unpack2(typename Raw2<T>::type raw);
template <>
__device__ __forceinline__ float2 unpack2<__nv_bfloat16>(uint32_t raw) {
  return make_float2(__uint_as_float(raw << 16), __uint_as_float(raw & 0xffff0000u));
}
template <>
__device__ __forceinline__ float2 unpack2<__half>(uint32_t raw) {
  return __half22float2(*reinterpret_cast<const __half2*>(&raw));
}
template <>
__device__ __forceinline__ float2 unpack2<float>(float2 raw) { return raw; }

__device__ __forceinline__ float exp2_approx(float x) {  // one special-function result
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Two fp32 operations per instruction (each rounded like the scalar one): the elementwise phases of the chunk kernels
// are bound by instruction issue.
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "add.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "mov.b64 rc, {%6, %7};\n\tfma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 twice(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 minus2(float2 a, float2 b) { return fma2(b, twice(-1.f), a); }
__device__ __forceinline__ float2 exp2_2(float2 x) { return make_float2(exp2_approx(x.x), exp2_approx(x.y)); }

// ---- layer prologue (optional, fused into the forward kernels) ------------------------------
// bit flags of the `prologue` argument of the *_fused entry points
constexpr int kPrologueNorm = GDN2_PROLOGUE_NORMALIZE_QK;   // q, k are raw projections: L2-normalise them
constexpr int kPrologueGate = GDN2_PROLOGUE_ACTIVATE_GATES; // beta, w, g are pre-activations
constexpr float kPrologueEps = 1e-6f;

// The activations inside the forward kernels run on the special-function unit (ex2 / lg2 / rcp
// approximations, about 1e-6 relative, far below the 16-bit inputs' own rounding): the library routines
// (expf, log1pf, a full division) made the prologue half of the prep kernel's code and two thirds again
// of its time.  (The stand-alone activation kernel of a training step is memory-bound and keeps them.)
__device__ __forceinline__ float prologue_sigmoid(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.f + __expf(-x)));
  return r;
}
// log-decay g = -softplus(x) = -log(1 + e^x).  Small e^x: the series e - e^2/2 + e^3/3 (its first
// dropped term is below 2^-26 of the sum there; lg2 of a number next to 1 would lose the digits);
// softplus(x) equals x to fp32 precision beyond 20.
__device__ __forceinline__ float prologue_log_decay(float x) {
  const float e = __expf(fminf(x, 20.f));
  const float series = e * (1.f - e * (0.5f - e * 0.33333334f));
  const float direct = __logf(1.f + e);
  return x > 20.f ? -x : -(e < 0.00390625f ? series : direct);
}

// ---- host-side status helpers ---------------------------------------------------
void record_cuda_error(cudaError_t err);  // defined in api.cu
int check_launch();                       // cudaGetLastError -> status
int multiprocessors(int* count);          // SMs of the current device, looked up once per device (api.cu)
cudaError_t ensure_dynamic_smem(const void* kernel, int bytes);  // once per (kernel, device) opt-in (api.cu)
bool profiling();  // per-kernel timing is on: the kernels of a call then run one by one (api.cu)
void profile_mark(int index, cudaStream_t stream);  // records timing event `index` when profiling is on (api.cu)

// ---- kernels of one call that overlap -----------------------------------------------
// The second one is launched `beside` the first: it may begin once all CTAs of the first have begun (let_others_begin, at
// the start of the first) where those leave room, needs nothing of what the first writes, and calls outlast_others at its
// end: what follows on the stream waits for the second alone.  Everything before the first is over by then.  Its last CTA
// waits and no other, since one that waits keeps its place on the SM from the CTAs after it.  (H16, all waiting / the last:
// 60 sequences of 30 tokens packed with one of 4096 317 / 277 us, in training 1068 / 1012, 40 of 5 with 2048 and 1024 137 /
// 113.)  Both do nothing in a launch of their own.
__device__ __forceinline__ void let_others_begin() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void outlast_others() {
  if (blockIdx.x + 1 == gridDim.x) asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <typename... Params, typename... Args>
inline int launch_beside(void (*kernel)(Params...), unsigned blocks, int threads, int smem, cudaStream_t stream,
                         const Args&... args) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(blocks);
  config.blockDim = dim3(unsigned(threads));
  config.dynamicSmemBytes = size_t(smem);
  config.stream = stream;
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  config.attrs = &attribute;
  config.numAttrs = 1;
  const cudaError_t err = cudaLaunchKernelEx(&config, kernel, args...);
  if (err == cudaSuccess) return GDN2_OK;
  (void)cudaGetLastError();
  record_cuda_error(err);
  return GDN2_ERR_LAUNCH;
}

inline bool valid_seq_dtype(int d) { return d == GDN2_BF16 || d == GDN2_FP16; }
inline bool valid_gate_dtype(int d, int seq) { return d == seq || d == GDN2_FP32; }

// Dispatch a callable templated on <T, G> over the runtime dtype codes.
#define GDN2_DISPATCH_TYPES(dtype, g_dtype, ...)                         \
  do {                                                                   \
    if ((dtype) == GDN2_BF16) {                                          \
      using T = __nv_bfloat16;                                           \
      if ((g_dtype) == GDN2_FP32) { using G = float; __VA_ARGS__; }      \
      else { using G = __nv_bfloat16; __VA_ARGS__; }                     \
    } else {                                                             \
      using T = __half;                                                  \
      if ((g_dtype) == GDN2_FP32) { using G = float; __VA_ARGS__; }      \
      else { using G = __half; __VA_ARGS__; }                            \
    }                                                                    \
  } while (0)

}  // namespace gdn2
