// Shared by the forms of vy_linear_plain (linear_plain.cu, linear_split_tc.cu).
#pragma once
#include "split_mma.cuh"
#include "vy_common.cuh"
#include "vy_ptx.cuh"   // warp_sum

namespace vy {

__device__ __forceinline__ float uact(float x, int act) {
  switch (act) {
    case VY_UACT_RELU2: { const float r = fmaxf(x, 0.f); return r * r; }
    case VY_UACT_SILU: return x / (1.f + expf(-x));
    case VY_UACT_SIGMOID: return 1.f / (1.f + expf(-x));
    case VY_UACT_GELU_TANH: return 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
    default: return x;
  }
}

struct LinDev {
  int M, N, K;
  const void* A; long long lda; int a_dt;
  const void* W; long long ldw; int w_dt;
  const void* bias; int bias_dt;
  const void* addend; long long ld_addend; int addend_dt;
  int act; float scale;
  void* out; long long ld_out; int out_dt;
  long long a_batch, w_batch, out_batch, bias_batch;   // element strides between the independent products of a batched call
};

// product b of a batched call: the same shapes at shifted base pointers
__device__ __forceinline__ void lin_select(LinDev& d, int b) {
  if (b == 0) return;
  d.A = static_cast<const char*>(d.A) + d.a_batch * b * (d.a_dt == VY_F32 ? 4 : 2);
  d.W = static_cast<const char*>(d.W) + d.w_batch * b * (d.w_dt == VY_F32 ? 4 : 2);
  d.out = static_cast<char*>(d.out) + d.out_batch * b * (d.out_dt == VY_F32 ? 4 : 2);
  if (d.bias) d.bias = static_cast<const char*>(d.bias) + d.bias_batch * b * (d.bias_dt == VY_F32 ? 4 : 2);
}

__device__ __forceinline__ void lin_store(const LinDev& d, int m, int n, float acc) {
  if (d.bias) acc += ld_as_float(d.bias, d.bias_dt, n);
  acc = uact(acc, d.act) * d.scale;
  if (d.addend) acc += ld_as_float(d.addend, d.addend_dt, static_cast<long long>(m) * d.ld_addend + n);
  st_from_float(d.out, d.out_dt, static_cast<long long>(m) * d.ld_out + n, acc);
}

// One product in fp32 FMAs by a warp (16-byte aligned rows, K a multiple of 4), the sum in every lane
static __device__ __noinline__ float lin_dot(const float* a, const float* w, int K) {
  float acc = 0.f;
  for (int k = 4 * (threadIdx.x & 31); k < K; k += 128) {
    const float4 x = *reinterpret_cast<const float4*>(a + k), y = *reinterpret_cast<const float4*>(w + k);
    acc = fmaf(x.x, y.x, acc);
    acc = fmaf(x.y, y.y, acc);
    acc = fmaf(x.z, y.z, acc);
    acc = fmaf(x.w, y.w, acc);
  }
  return warp_sum(acc);
}

// An entry's halves are off by at most 2^-49 of the largest entry under its unit (split_mma.cuh): a row's in a tile of 64 k where tiles are split, a whole row's where operands are split ahead.
// So a product is as good as an fp32 one unless it is very small beside the product of its rows' largest entries: then, as where an infinity or NaN went in (the halves of an infinity would
// all be NaN), it is computed again in FMAs. At 2^-16 of it the halves' share of a result is at most K 2^-32 and, signs being random, about sqrt(K) 2^-33: 2^-28 at K 1024, 2^-26 at 16384, where
// an fp32 sum's rounding is 2^-23. Of normal numbers' products 2 to 6 in a million are that small. One entry of 2^12 to 2^40 per row in one stretch of 64, error against 64 bits of tiles / of
// operands split ahead: K 1024 1.55 / 1.45e-7 to 1.20 / 1.20e-7, 8192 2.46 / 1.98e-7 to 2.94 / 2.94e-7, never above
constexpr float LS_SMALL = 0x1p-16f * (1 << SPLIT_TOP) * (1 << SPLIT_TOP);

// linear_split_tc.cu: scratch of the tcgen05 form (0: not for these sizes), and the form itself, two launches
long long linear_split_bytes(int M, int N, int K);
cudaError_t launch_linear_split_tc(const LinDev& d, void* ws, cudaStream_t st);

}  // namespace vy
