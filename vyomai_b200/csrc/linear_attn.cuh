// What the two tensor-core forms of linear attention over chunks share (linear_attn_mma.cu, linear_attn_tc.cu): the workspace and the decays of a state-space chunk
#pragma once
#include "seqmix.cuh"
#include "split_mma.cuh"

namespace vy {

constexpr int LM_C = 64, LT_C = 128;   // tokens per chunk; in linear_attn_tc.cu

// The chunks' states in the workspace: chunk c of sequence s is slot cu[s] / 64 + s + c (never more than rows / 64 + n_seqs in all; every other one is used of chunks of 128)
struct LaChunks {
  float* U;          // [slots][heads][dim][vdim]
  float* D;          // [slots][heads]
  unsigned* top;     // [slots][heads] largest |S| before the chunk, as bits
  int* odd;          // [slots][heads / hp][vslices] 1: not for fp16 halves
  int chunk;         // tokens per chunk
};
__device__ __forceinline__ long long la_slot(const RecDev& d, int s, int c) { return d.cu[s] / LM_C + s + c; }

// a^n, n <= 128, in eight steps of repeated squaring (double: rounded once, to the fp32 result)
__device__ __forceinline__ float power(float a, int n) {
  double x = a, r = 1.0;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    if (n >> b & 1) r *= x;
    x *= x;
  }
  return static_cast<float>(r);
}

// One warp: tokens E lane .. E lane + E - 1 of a chunk of nt (at most 32 E): log decays summed (in double: `each` gets token, sum, write strength and the sum at the
// chunk's end) as in linear_attn_chunk_kernel. Returns the chunk's whole decay
template <int E, typename Fn>
__device__ __forceinline__ float token_decays(const RecDev& d, long long r0, int nt, int h, int lane, Fn each) {
  const float rate = expf(ld_as_float(d.a_log, d.a_log_dt, h)), dt_b = ld_as_float(d.dt_bias, d.a_log_dt, h);
  double la[E], run = 0.0;
  float w[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int tt = E * lane + e;
    w[e] = tt < nt ? softplusf_(d.dt[(r0 + tt) * d.ld_dt + h] + dt_b) : 0.f;
    run += fmaxf(-rate * w[e], MIN_LOG_DECAY);
    la[e] = run;
  }
  const double own = run;
#pragma unroll
  for (int k = 1; k < 32; k <<= 1) {
    const double x = __shfl_up_sync(0xffffffffu, run, k);
    if (lane >= k) run += x;
  }
  const double end = __shfl_sync(0xffffffffu, run, 31);
#pragma unroll
  for (int e = 0; e < E; ++e) each(E * lane + e, run - own + la[e], w[e], end);
  return expf(static_cast<float>(end));
}

__device__ __forceinline__ void store_split4(unsigned char* hi, unsigned char* lo, int at, float4 x, float4 sc) {
  uint2 h, l;
  split2(x.x * sc.x, x.y * sc.y, h.x, l.x);
  split2(x.z * sc.z, x.w * sc.w, h.y, l.y);
  *reinterpret_cast<uint2*>(hi + at) = h;
  *reinterpret_cast<uint2*>(lo + at) = l;
}
// Largest and smallest (but not zero) of rows' and columns' largest entries, as bits: positive numbers order like them, NaN after infinity
constexpr unsigned RANGE_NONE = 0x7f800000u;   // infinity: no entry yet
struct Range { unsigned top, low; };
__device__ __forceinline__ void note(Range& r, unsigned m, bool few = false) {
  r.top = max(r.top, m);
  if (m) r.low = min(r.low, few ? __float_as_uint(16.f * __uint_as_float(m)) : m);
}
__device__ __forceinline__ void note_warp(Range* to, Range r) {   // to: shared memory, read after a barrier
  r.top = __reduce_max_sync(0xffffffffu, r.top);
  r.low = __reduce_min_sync(0xffffffffu, r.low);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&to->top, r.top);
    atomicMin(&to->low, r.low);
  }
}
__device__ __forceinline__ bool too_wide(Range r) { return r.top >= 0x7f800000u || __uint_as_float(r.low) < 0x1p-20f * __uint_as_float(r.top); }

// A warp's tile, a thread's N quads of it: FROM lanes share a row, 4 FROM columns. Notes the largest entry of each row and of each column (few_rows, few_columns: all
// may be small by chance) and returns the columns'
template <int N, int FROM>
__device__ __forceinline__ uint4 look(const float4 (&x)[N], bool few_rows, bool few_columns, Range& r) {
  uint4 m = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint4 a = make_uint4(abs_bits(x[i].x), abs_bits(x[i].y), abs_bits(x[i].z), abs_bits(x[i].w));
    m = make_uint4(max(m.x, a.x), max(m.y, a.y), max(m.z, a.z), max(m.w, a.w));
    unsigned most = max(max(a.x, a.y), max(a.z, a.w));
#pragma unroll
    for (int k = 1; k < FROM; k <<= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, k));
    note(r, most, few_columns);
  }
#pragma unroll
  for (int k = FROM; k < 32; k <<= 1)
    m = make_uint4(max(m.x, __shfl_xor_sync(0xffffffffu, m.x, k)), max(m.y, __shfl_xor_sync(0xffffffffu, m.y, k)), max(m.z, __shfl_xor_sync(0xffffffffu, m.z, k)),
                   max(m.w, __shfl_xor_sync(0xffffffffu, m.w, k)));
  note(r, m.x, few_rows);
  note(r, m.y, few_rows);
  note(r, m.z, few_rows);
  note(r, m.w, few_rows);
  return m;
}
__device__ __forceinline__ float4 column_units(uint4 m) {   // 2^(exponent - SPLIT_TOP) of each column
  const auto u = [](unsigned b) { return pow2i(split_exponent(__uint_as_float(b)) - SPLIT_TOP); };
  return make_float4(u(m.x), u(m.y), u(m.z), u(m.w));
}
__device__ __forceinline__ float4 column_scales(uint4 m) {
  const auto u = [](unsigned b) { return split_scale(split_exponent(__uint_as_float(b))); };
  return make_float4(u(m.x), u(m.y), u(m.z), u(m.w));
}

// linear_attn_tc.cu: states and read-outs of chunks of LT_C tokens (state space, fp32 rows in quads), at most LT_HEADS heads per CTA
constexpr int LT_HEADS = 8;
int linear_attn_tc_heads(const RecDev& d, int n_seqs, int max_new, long long rows, int vslices);   // heads per CTA; 0: not for this step
cudaError_t launch_la_states_tc(const RecDev& d, const LaChunks& w, int hp, int n_seqs, int max_new, long long rows, cudaStream_t st);
cudaError_t launch_la_outputs_tc(const RecDev& d, const LaChunks& w, int hp, int n_seqs, int max_new, long long rows, cudaStream_t st);

// linear_attn_tc_fixed.cu: the same for decays by head; has the build the registers that its kernels share out?
bool la_fixed_registers();
cudaError_t launch_la_states_fixed(const RecDev& d, const LaChunks& w, int hp, int n_seqs, int max_new, long long rows, cudaStream_t st);
cudaError_t launch_la_outputs_fixed(const RecDev& d, const LaChunks& w, int hp, int n_seqs, int max_new, long long rows, cudaStream_t st);

}  // namespace vy
