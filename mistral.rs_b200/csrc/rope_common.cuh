// rope_common.cuh — 8-element slices of 16- and 32-bit vectors, and the rotary embedding of such a slice (paged_attn.cu, step_resident.cu).
#pragma once
#include "common.cuh"

#include <cuda_fp8.h>

namespace mrs {

template <typename T> struct Vec8;
template <> struct Vec8<__half> {
  __device__ static __forceinline__ void load(const __half *p, float *f) {
    const uint4 v = *(const uint4 *)p;
    const __half2 *h = (const __half2 *)&v;
#pragma unroll
    for (int i = 0; i < 4; i++) { const float2 t = __half22float2(h[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
  }
  __device__ static __forceinline__ float one(const __half *p) { return __half2float(*p); }
  __device__ static __forceinline__ void store(__half *p, const float *f) {
    uint4 v;
    __half2 *h = (__half2 *)&v;
#pragma unroll
    for (int i = 0; i < 4; i++) h[i] = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
    *(uint4 *)p = v;
  }
};
template <> struct Vec8<__nv_bfloat16> {
  __device__ static __forceinline__ void load(const __nv_bfloat16 *p, float *f) {
    const uint4 v = *(const uint4 *)p;
    const __nv_bfloat162 *h = (const __nv_bfloat162 *)&v;
#pragma unroll
    for (int i = 0; i < 4; i++) { const float2 t = __bfloat1622float2(h[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
  }
  __device__ static __forceinline__ float one(const __nv_bfloat16 *p) { return __bfloat162float(*p); }
  __device__ static __forceinline__ void store(__nv_bfloat16 *p, const float *f) {
    uint4 v;
    __nv_bfloat162 *h = (__nv_bfloat162 *)&v;
#pragma unroll
    for (int i = 0; i < 4; i++) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    *(uint4 *)p = v;
  }
};
template <> struct Vec8<float> {
  __device__ static __forceinline__ void load(const float *p, float *f) {
    const float4 a = *(const float4 *)p, b = *(const float4 *)(p + 4);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  }
  __device__ static __forceinline__ float one(const float *p) { return *p; }
  __device__ static __forceinline__ void store(float *p, const float *f) {
    *(float4 *)p = make_float4(f[0], f[1], f[2], f[3]);
    *(float4 *)(p + 4) = make_float4(f[4], f[5], f[6], f[7]);
  }
};
// FP8-E4M3 cache bytes (cache_dtype 3, REF mistralrs-paged-attn/src/cuda/ffi.rs dtype codes): value = float(e4m3);
// the per-tensor scales are folded into the logits (k_scale) and the output (v_scale)
struct fp8_t { uint8_t b; };
__device__ __forceinline__ float fp8_to_float(uint8_t b) {
  const __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)b, __NV_E4M3);
  return __half2float(*(const __half *)&h);
}
template <> struct Vec8<fp8_t> {
  __device__ static __forceinline__ void load(const fp8_t *p, float *f) {
    const uint2 v = *(const uint2 *)p;
    const uint8_t *b = (const uint8_t *)&v;
#pragma unroll
    for (int i = 0; i < 8; i++) f[i] = fp8_to_float(b[i]);
  }
  __device__ static __forceinline__ float one(const fp8_t *p) { return fp8_to_float(p->b); }
};

// round through T (what storing a tensor of dtype T would do)
template <typename T> __device__ __forceinline__ float rnd(float v);
template <> __device__ __forceinline__ float rnd<__half>(float v) { return __half2float(__float2half_rn(v)); }
template <> __device__ __forceinline__ float rnd<__nv_bfloat16>(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
template <> __device__ __forceinline__ float rnd<float>(float v) { return v; }
template <typename T> __device__ __forceinline__ T from_float(float v);
template <> __device__ __forceinline__ __half from_float<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ float from_float<float>(float v) { return v; }

// NeoX RoPE of the 8-element slice held by lane `gl` (elements d0..d0+7 of a head), with the
// reference kernel's per-operation rounding in T (rotary.cu:10-34).  The partner slice
// (d +- D/2) lives in lane gl ^ (LPT/2).
template <typename T, int D>
__device__ __forceinline__ void rope_slice(float *x, const T *cosp, const T *sinp, int gl) {
  constexpr int LPT = D / 8;
  const bool upper = gl >= LPT / 2;
  const int o0 = (upper ? gl - LPT / 2 : gl) * 8;  // rot offset of this slice
  float c[8], sn[8];
  Vec8<T>::load(cosp + o0, c);
  Vec8<T>::load(sinp + o0, sn);
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const float other = __shfl_xor_sync(0xffffffffu, x[i], LPT / 2);
    // out_x = fma(x, cos, -T(y*sin)); out_y = fma(y, cos, T(x*sin)) with one rounding in T, as the
    // reference kernel is compiled (tests/golden/ref_golden.npz)
    const float b = rnd<T>(other * sn[i]);     // y*sin (lower) / x*sin (upper)
    x[i] = (float)__hfma((T)x[i], (T)c[i], (T)(upper ? b : -b));
  }
}
// GPT-J / GGUF-llama pairing: (x[2i], x[2i+1]) rotate together and both live in this lane's slice;
// cos/sin index d/2.  Same per-operation rounding as rope_slice (REF rotary.cu:10-34, is_neox = 0).
template <typename T, int D>
__device__ __forceinline__ void rope_slice_interleaved(float *x, const T *cosp, const T *sinp, int gl) {
  const int o0 = gl * 4;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float c = Vec8<T>::one(cosp + o0 + i), sn = Vec8<T>::one(sinp + o0 + i);
    const float xv = x[2 * i], yv = x[2 * i + 1];
    const float ys = rnd<T>(yv * sn), xs = rnd<T>(xv * sn);
    x[2 * i] = (float)__hfma((T)xv, (T)c, (T)(-ys));
    x[2 * i + 1] = (float)__hfma((T)yv, (T)c, (T)xs);
  }
}
template <typename T, int D>
__device__ __forceinline__ void rope_any(float *x, const T *cosp, const T *sinp, int gl, bool interleaved) {
  if (interleaved) rope_slice_interleaved<T, D>(x, cosp, sinp, gl);
  else rope_slice<T, D>(x, cosp, sinp, gl);
}

}  // namespace mrs
