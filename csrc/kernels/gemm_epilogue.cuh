// What every GEMM kernel of this directory applies to its fp32 accumulators: the launch parameters
// and the epilogue (scale, bias, activation or its derivative, residual, accumulate) of one element.
#pragma once
#include "gemm.h"
#include "sm100_ptx.cuh"

#include <cuda_bf16.h>

namespace lt {

using namespace ptx;

struct KernelParams {
  int M, N, K;
  int tiles_m, tiles_n, batch_inner, batch_total;
  int a_mn, b_mn;
  void* C;
  long long ldc, c_stride_inner, c_stride_outer;
  float alpha;
  int c_fp32, accumulate;
  const void* bias;
  int bias_fp32;
  int act;
  const __nv_bfloat16* residual;
  long long ldr;
  __nv_bfloat16* aux_out;
  const __nv_bfloat16* aux_in;
  long long ld_aux;
  int causal_tiles;
  int k_seg;   // GemmArgs::k_seg
  int vec_ok;  // C / residual / aux rows allow 16-byte vector access
  int vec32_ok;  // ... and 32-byte (256-bit) access (bf16 output, residual, aux)
  int c32_ok;    // fp32 output rows allow 32-byte access
  // all-gather of B fused into the kernel (g_world <= 1: off)
  const uint64_t* g_b_ptrs;
  const uint64_t* g_signal_ptrs;
  uint32_t* g_flags;
  int* g_status;
  long long g_ldb;
  int g_rank, g_world, g_rows_per_shard, g_done;
  uint32_t g_epoch;
  int late_wait;   // GemmArgs::overlap_prev: wait for the previous kernel before exit, not before work
};

__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float gelu_f(float x) {
  const float k0 = 0.7978845608f, k1 = 0.044715f;
  float t = tanh_fast(k0 * (x + k1 * x * x * x));
  return 0.5f * x * (1.0f + t);
}
__device__ __forceinline__ float dgelu_f(float x) {
  const float k0 = 0.7978845608f, k1 = 0.044715f;
  float t = tanh_fast(k0 * (x + k1 * x * x * x));
  return 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * k0 * (1.0f + 3.0f * k1 * x * x);
}

// The same two functions on a pair of values with packed f32x2 arithmetic (one instruction
// per two elements; the tanh stays one MUFU each).  The epilogue of a K = 768 product is bound
// by instruction issue, so the vector path uses these.
//   gelu(x)  = h + h t,                  h = x / 2, t = tanh(x (k0 + k0 k1 x^2))
//   gelu'(x) = s + s r (1 - s) 2,        s = (1 + t) / 2, r = x (k0 + 3 k0 k1 x^2)
__device__ __forceinline__ float2 tanh_arg2(float2 x, float2 x2) {
  const float k0 = 0.7978845608f, k0k1 = 0.7978845608f * 0.044715f;
  return fmul2(x, ffma2(x2, make_float2(k0k1, k0k1), make_float2(k0, k0)));
}
__device__ __forceinline__ float2 gelu2(float2 x) {
  const float2 u = tanh_arg2(x, fmul2(x, x));
  const float2 t = make_float2(tanh_fast(u.x), tanh_fast(u.y));
  const float2 h = fmul2(x, make_float2(0.5f, 0.5f));
  return ffma2(h, t, h);
}
// returns v * gelu'(x)
__device__ __forceinline__ float2 dgelu_mul2(float2 v, float2 x) {
  const float k0 = 0.7978845608f, k0k1 = 0.7978845608f * 0.044715f;
  const float2 x2 = fmul2(x, x);
  const float2 u = tanh_arg2(x, x2);
  const float2 t = make_float2(tanh_fast(u.x), tanh_fast(u.y));
  const float2 s = ffma2(t, make_float2(0.5f, 0.5f), make_float2(0.5f, 0.5f));
  // r2 = 2 x (k0 + 3 k0 k1 x^2)
  const float2 r2 = fmul2(x, ffma2(x2, make_float2(6.0f * k0k1, 6.0f * k0k1), make_float2(2.0f * k0, 2.0f * k0)));
  const float2 z = ffma2(fmul2(r2, s), make_float2(-1.0f, -1.0f), r2);      // r2 (1 - s)
  return fmul2(v, ffma2(s, z, s));
}

// Scalar epilogue for one element, shared by the tensor-core tail path and the SIMT
// fallback kernel.
__device__ __forceinline__ void epilogue_store_scalar(const KernelParams& p, char* c_base,
                                                      long long row, int col, float acc) {
  float v = acc * p.alpha;
  if (p.bias) {
    v += p.bias_fp32 ? ((const float*)p.bias)[col]
                     : __bfloat162float(((const __nv_bfloat16*)p.bias)[col]);
  }
  if (p.act == GEMM_ACT_GELU) {
    if (p.aux_out) p.aux_out[row * p.ldc + col] = __float2bfloat16(v);
    v = gelu_f(v);
  } else if (p.act == GEMM_ACT_RELU) {
    if (p.aux_out) p.aux_out[row * p.ldc + col] = __float2bfloat16(v);
    v = fmaxf(v, 0.0f);
  } else if (p.act == GEMM_ACT_DGELU) {
    v *= dgelu_f(__bfloat162float(p.aux_in[row * p.ld_aux + col]));
  } else if (p.act == GEMM_ACT_DRELU) {
    v = __bfloat162float(p.aux_in[row * p.ld_aux + col]) > 0.0f ? v : 0.0f;
  }
  if (p.residual) v += __bfloat162float(p.residual[row * p.ldr + col]);
  if (p.c_fp32) {
    float* c = (float*)c_base + row * p.ldc + col;
    if (p.accumulate) v += *c;
    *c = v;
  } else {
    __nv_bfloat16* c = (__nv_bfloat16*)c_base + row * p.ldc + col;
    if (p.accumulate) v += __bfloat162float(*c);
    *c = __float2bfloat16(v);
  }
}

}  // namespace lt
