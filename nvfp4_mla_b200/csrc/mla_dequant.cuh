// Whole-cache dequantisation: ckv = e2m1 * block_scale * ckv_scale, kpe = e4m3 * kpe_scale, to fp32 or bf16.
// The two multiplies are separate fp32 roundings in exactly that order (never fused), which makes the fp32 result
// bit-identical to the torch expression `lut[code] * sf.float() * ckv_scale`.
//
// HBM-bound: 352 bytes in, 2304 (fp32) or 1152 (bf16) bytes out per token. One warp per token per step; for fp32 lane l
// owns channels 4l .. 4l+3 of each 128-channel quarter, for bf16 channels 8l .. 8l+7 of each half, so every store
// instruction of the warp writes 512 contiguous bytes.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include "mla_common.cuh"
#include "ptx_sm100.cuh"

namespace mla {

__device__ __forceinline__ float2 f16x2_to_f32x2(uint32_t h) {  // exact
  __half2 p;
  memcpy(&p, &h, sizeof p);
  return __half22float2(p);
}
__device__ __forceinline__ float e4m3_value(uint8_t x) {
  __nv_fp8_e4m3 f;
  f.__x = x;
  return float(f);
}

// The outputs are written once and not read here: streaming stores.
template <typename T> struct Dequant;
template <> struct Dequant<float> {
  static __device__ __forceinline__ void put(float* p, uint32_t codes, float scale, float ckv_scale) {  // four channels
    uint32_t e0, e1;  // as two FP16 pairs (exact; FP16 -> fp32 is exact too)
    asm("{\n.reg .b8 b0, b1;\nmov.b16 {b0, b1}, %2;\ncvt.rn.f16x2.e2m1x2 %0, b0;\ncvt.rn.f16x2.e2m1x2 %1, b1;\n}"
        : "=r"(e0), "=r"(e1)
        : "h"(uint16_t(codes)));
    const float2 a = f16x2_to_f32x2(e0), b = f16x2_to_f32x2(e1);
    __stcs(reinterpret_cast<float4*>(p), make_float4(__fmul_rn(__fmul_rn(a.x, scale), ckv_scale), __fmul_rn(__fmul_rn(a.y, scale), ckv_scale),
                                                     __fmul_rn(__fmul_rn(b.x, scale), ckv_scale), __fmul_rn(__fmul_rn(b.y, scale), ckv_scale)));
  }
  static __device__ __forceinline__ void put2(float* p, float a, float b) { __stcs(reinterpret_cast<float2*>(p), make_float2(a, b)); }
};
template <> struct Dequant<__nv_bfloat16> {
  static __device__ __forceinline__ void put(__nv_bfloat16* p, uint32_t codes, float scale, float ckv_scale) {  // eight channels
    uint32_t o[4], e[4];
    ptx::e2m1x8_to_f16x8(codes, e);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 v = f16x2_to_f32x2(e[i]);
      const __nv_bfloat162 h = __floats2bfloat162_rn(__fmul_rn(__fmul_rn(v.x, scale), ckv_scale), __fmul_rn(__fmul_rn(v.y, scale), ckv_scale));
      o[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    __stcs(reinterpret_cast<uint4*>(p), make_uint4(o[0], o[1], o[2], o[3]));
  }
  static __device__ __forceinline__ void put2(__nv_bfloat16* p, float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    __stcs(reinterpret_cast<uint32_t*>(p), *reinterpret_cast<const uint32_t*>(&h));
  }
};

constexpr int kDequantThreads = 256;

// Tokens a warp takes per trip: the loads of all of them are issued before the first is converted. 524288 tokens to BF16: 147.6 us
// with one token per trip and ordinary stores, 127.6 with two and streaming stores (120 at the measured copy bandwidth).
constexpr int kDequantTokens = 2;

template <typename T>
__global__ void __launch_bounds__(kDequantThreads)
mla_dequant_kernel(const uint8_t* __restrict__ ckv, const uint8_t* __restrict__ sf, const uint8_t* __restrict__ kpe,
                   float ckv_scale, float kpe_scale, T* __restrict__ ckv_out, T* __restrict__ kpe_out, long long n_tok) {
  constexpr int U = kDequantTokens, L = sizeof(T) == 2 ? 2 : 4;  // L loads of 512 / L channels per token
  const int lane = threadIdx.x & 31;
  const long long warp0 = (long long)blockIdx.x * (kDequantThreads / 32) + (threadIdx.x >> 5);
  const long long stride = (long long)gridDim.x * (kDequantThreads / 32);
  for (long long t0 = warp0 * U; t0 < n_tok; t0 += stride * U) {
    // 16-bit output: lane l owns channels 8l .. 8l+7 of each half of the row (a 4-byte load, a 16-byte store); fp32: channels
    // 4l .. 4l+3 of each quarter (a 2-byte load, a 16-byte store). Every instruction of the warp is one contiguous run. The
    // 32 block scales are loaded one per lane and handed round by shuffle (block = channel / 16).
    uint32_t w[U][L], sv[U], two[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long tok = t0 + u < n_tok ? t0 + u : n_tok - 1;
      sv[u] = __ldcs(sf + tok * (CKV / 16) + lane);
#pragma unroll
      for (int j = 0; j < L; ++j) {
        if constexpr (L == 2) w[u][j] = __ldcs(reinterpret_cast<const uint32_t*>(ckv + tok * (CKV / 2) + 128 * j) + lane);
        else w[u][j] = __ldcs(reinterpret_cast<const uint16_t*>(ckv + tok * (CKV / 2) + 64 * j) + lane);
      }
      two[u] = __ldcs(reinterpret_cast<const uint16_t*>(kpe + tok * KPE) + lane);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long tok = t0 + u;
      if (tok >= n_tok) break;
#pragma unroll
      for (int j = 0; j < L; ++j) {
        const float scale = e4m3_value(uint8_t(__shfl_sync(~0u, sv[u], (32 / L) * j + lane / L)));
        Dequant<T>::put(ckv_out + tok * CKV + (512 / L) * j + (512 / L / 32) * lane, w[u][j], scale, ckv_scale);
      }
      Dequant<T>::put2(kpe_out + tok * KPE + 2 * lane, __fmul_rn(e4m3_value(two[u] & 255), kpe_scale),
                       __fmul_rn(e4m3_value(two[u] >> 8), kpe_scale));
    }
  }
}

}  // namespace mla
