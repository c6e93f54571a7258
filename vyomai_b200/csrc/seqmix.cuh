// Shared by the sequence-mixer kernels (seqmix.cu: token-serial forms used for single tokens and short portions;
// seqmix_tiled.cu, window_attn_tc.cu, window_attn_mma.cu, linear_attn_tc.cu, linear_attn_mma.cu, delta_rule_mma.cu: forms used for prompts): activation helpers, the kernels' argument blocks and the tiled launchers.
#pragma once
#include <math.h>

#include "vy_common.cuh"
#include "vy_ptx.cuh"   // warp_sum, warp_max

namespace vy {

__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + expf(-x)); }
__device__ __forceinline__ float siluf_(float x) { return x / (1.f + expf(-x)); }
__device__ __forceinline__ float softplusf_(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float apply_uact(float x, int act) {
  switch (act) {
    case VY_UACT_RELU2: { const float r = fmaxf(x, 0.f); return r * r; }
    case VY_UACT_SILU: return siluf_(x);
    case VY_UACT_SIGMOID: return sigmoidf_(x);
    case VY_UACT_GELU_TANH: return 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
    default: return x;
  }
}
// 1 / y for y >= 1 in two Newton steps from the approximate reciprocal (1 / infinity = 0; a NaN stays one), and x / (1 + e^-x) with its quotient corrected once: rounded as a
// division but for a hair, which with its range checks is twice as many instructions. The approximate reciprocal flushes what is below 2^-126 (x below -87.3): it is taken of 2^-30 y
constexpr float RECIP_SCALE = 0x1p-30f;
__device__ __forceinline__ float recip_first(float y) { return vy_rcp_approx(y * RECIP_SCALE) * RECIP_SCALE; }
__device__ __forceinline__ float recip_near(float y) {
  const float r = recip_first(y);
  float n = fmaf(r, fmaf(-y, r, 1.f), r);
  n = fmaf(n, fmaf(-y, n, 1.f), n);
  return y < INFINITY ? n : r;
}
__device__ __forceinline__ float sigmoid_near(float x) { return recip_near(1.f + expf(-x)); }
__device__ __forceinline__ float silu_near(float x) {
  const float y = 1.f + expf(-x), r0 = recip_first(y), r = fmaf(r0, fmaf(-y, r0, 1.f), r0), q = x * r, a = fmaf(fmaf(-y, q, x), r, q);
  return a == a ? a : x * r0;   // infinities
}
__device__ __forceinline__ float uact_near(float x, int act) {
  return act == VY_UACT_SILU ? silu_near(x) : act == VY_UACT_SIGMOID ? sigmoid_near(x) : apply_uact(x, act);
}
constexpr float MIN_LOG_DECAY = -1e4f;   // exp of it is 0 in fp32; keeps sums and differences of log decays finite
// cap * tanh(s / cap) as cap * (1 - 2 / (1 + e^(2 s / cap))): expf and a fast reciprocal, absolute error a few 1e-7 * cap (the softmax
// that follows depends on score differences, i.e. on absolute error); e^x overflowing to inf gives exactly cap, underflow exactly -cap
__device__ __forceinline__ float cap_score(float s, float cap, float two_over_cap) {
  return cap > 0.f ? cap * (1.f - __fdividef(2.f, 1.f + expf(s * two_over_cap))) : s;
}

// |x| as bits, which order as numbers do: those of an infinity are 0x7f800000, a NaN's larger
__device__ __forceinline__ unsigned abs_bits(float x) { return __float_as_uint(x) & 0x7fffffffu; }
__device__ __forceinline__ float dot4(const float4 a, const float4 b, float acc) {
  acc = fmaf(a.x, b.x, acc);
  acc = fmaf(a.y, b.y, acc);
  acc = fmaf(a.z, b.z, acc);
  return fmaf(a.w, b.w, acc);
}
__device__ __forceinline__ void axpy4(float (&acc)[4], const float a, const float4 x) {
  acc[0] = fmaf(a, x.x, acc[0]);
  acc[1] = fmaf(a, x.y, acc[1]);
  acc[2] = fmaf(a, x.z, acc[2]);
  acc[3] = fmaf(a, x.w, acc[3]);
}
__device__ __forceinline__ const float4& f4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// Rows [0, rows) of a [rows, width] block of `src` into shared memory (row stride ld, zero-filled up to width4 columns, `act`
// applied): row j starts at element off(j) of src, or is all zero when off(j) < 0. Global loads go out in batches of 8 per
// thread before any of them is used, so a tile costs about one memory round trip. vec: src is fp32 and every row start and the
// width are multiples of 4 elements (16-byte loads).
template <int T, typename OffFn>
__device__ __forceinline__ void rows_to_smem(float* dst, int ld, int rows, int width, int width4, const void* src, int dt, bool vec, int act,
                                             OffFn off) {
  constexpr int U = 8;
  if (vec) {
    const int w4 = width4 >> 2, total = rows * w4;
    for (int e0 = threadIdx.x; e0 < total; e0 += T * U) {
      float4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + u * T;
        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (e < total) {
          const int j = e / w4, c = (e - j * w4) << 2;
          const long long o = off(j);
          if (o >= 0 && c < width) v[u] = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(src) + o + c);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + u * T;
        if (e < total) {
          const int j = e / w4, c = (e - j * w4) << 2;
          if (act != VY_UACT_NONE && c < width) {   // not the channels that fill up rows: act(0) may not be 0
            v[u].x = apply_uact(v[u].x, act); v[u].y = apply_uact(v[u].y, act);
            v[u].z = apply_uact(v[u].z, act); v[u].w = apply_uact(v[u].w, act);
          }
          *reinterpret_cast<float4*>(dst + j * ld + c) = v[u];
        }
      }
    }
  } else {
    const int total = rows * width4;
    for (int e0 = threadIdx.x; e0 < total; e0 += T * U) {
      float v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + u * T;
        v[u] = 0.f;
        if (e < total) {
          const int j = e / width4, c = e - j * width4;
          const long long o = off(j);
          if (o >= 0 && c < width) v[u] = ld_as_float(src, dt, o + c);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + u * T;
        if (e < total) {
          const int j = e / width4, c = e - j * width4;
          dst[j * ld + c] = act != VY_UACT_NONE && c < width ? apply_uact(v[u], act) : v[u];
        }
      }
    }
  }
}

// windowed attention with kept first tokens and a sink, over pages
struct WinDev {
  const int* cu; const int* pos0; const int* table; int tw, bs;
  const void* q; long long ldq; int q_dt;
  const void* kp; const void* vp; int pool_dt;
  long long k_row, v_row;   // row strides of the pools in elements (kv_heads * dim and kv_heads * vdim unless the caller views one pool twice)
  int heads, kv_heads, dim, vdim;
  float scale; int window, keep;
  float out_scale;   // multiplies the normalised output (fp32, before it is rounded to the output dtype)
  int chunk;   // > 0: keys of the query's own block of `chunk` positions only (window and keep are then 0)
  const void* sink; int sink_dt;
  const void* gate; long long ld_gate; int gate_dt;
  void* out; long long ld_out; int out_dt;
  int sigmoid;   // the weight of a visible key is sigmoid(score), not normalised over the keys
  const float* head_scale; const float* head_bias;   // score = (q . k) * scale * head_scale[h] + head_bias[h]; null: 1 / 0
  float softcap; const float* head_slope;   // then: cap tanh(score / cap) (cap > 0), minus head_slope[h] * distance (null: 0)
  long long rows;   // packed rows of the step (host: which prompt form)
};

__device__ __forceinline__ float head_scale_of(const WinDev& d, int h) { return d.head_scale ? d.scale * d.head_scale[h] : d.scale; }
__device__ __forceinline__ float head_bias_of(const WinDev& d, int h) { return d.head_bias ? d.head_bias[h] : 0.f; }

__device__ __forceinline__ float head_slope_of(const WinDev& d, int h) { return d.head_slope ? d.head_slope[h] : 0.f; }
// the capped score minus the distance's share; two_over_cap = 2 / softcap
__device__ __forceinline__ float shaped_score(const WinDev& d, float z, float two_over_cap, float slope, int distance) {
  return fmaf(-slope, static_cast<float>(distance), cap_score(z, d.softcap, two_over_cap));
}

// One query's visible keys at position pos: [0, nA) (kept first tokens) and [lowB, pos] (the window, or the query's chunk), disjoint
__device__ __forceinline__ void visible_keys(const WinDev& d, int pos, int& nA, int& lowB) {
  if (d.chunk > 0) { nA = 0; lowB = pos / d.chunk * d.chunk; }
  else if (d.window <= 0) { nA = pos + 1; lowB = pos + 1; }
  else { nA = min(d.keep, pos + 1); lowB = max(pos - d.window + 1, nA); }
}

// the keys a portion sees, from its first query on: slots [0, nA) are positions [0, nA) (kept first tokens), the others positions from lo on
__device__ __forceinline__ void portion_keys(const WinDev& d, int p0, int& nA, int& lo) {
  lo = d.chunk > 0 ? p0 / d.chunk * d.chunk : d.window <= 0 ? 0 : max(p0 - d.window + 1, 0);
  nA = d.window <= 0 ? 0 : min(d.keep, lo);
}

// recurrences (linear attention with a fixed decay, gated delta rule): state [slots, heads, dim, vdim] fp32
struct RecDev {
  const int* cu; const int* pos0; const int* slot;
  const void* q; long long ldq; const void* k; long long ldk; const void* v; long long ldv; int in_dt; int in_act;
  const void* a; long long ld_a; int a_dt;
  const void* b; long long ld_b; int b_dt;
  const void* a_log; int a_log_dt;
  const float* decay;
  int heads, kv_heads, dim, vdim;
  float unit_eps;
  int prepared;   // delta rule: q / k are unit vectors already (q scaled), `a` holds the decays and `b` the write strengths
  // chunked form with a decay and a write strength per head and token (state-space recurrence): strength w = softplus(dt + dt_bias[h]),
  // decay exp(-exp(a_log[h]) w), plus skip[h] v in the output, the whole times gate_act(gate); dt_bias, a_log, skip share a_log_dt
  const float* dt; long long ld_dt; const void* dt_bias; const void* skip;
  const float* gate; long long ld_gate; int gate_act;
  float q_scale;  // gated linear attention (the delta kernel without its correction term): multiplies q as it is read
  float* state;
  void* out; long long ld_out; int out_dt;
  // chunked walk behind linear_attn_mma.cu and linear_attn_tc.cu: null, or [cu / 64 + sequence + chunk][heads / odd_heads][odd_each] with a 1 where the sequence and head are left to
  // it, and their state before each chunk, [cu / 64 + sequence + chunk][heads][dim][vdim]; odd_chunk: tokens per chunk
  const int* odd; int odd_heads, odd_each, odd_chunk; const float* first;
};

// Prompt-sized steps: defined in the files named above.
cudaError_t launch_linear_attn_chunked(const RecDev& d, int n_seqs, cudaStream_t st);
cudaError_t launch_ssd_chunked(const RecDev& d, int n_seqs, cudaStream_t st);
// 16 tokens per step of the walk (delta_rule_mma.cu), given delta_rule_mma_floats(..) floats of 16-byte aligned scratch (0: not for this step); two launches
long long delta_rule_mma_floats(long long rows, int n_seqs, int max_new, int heads, int dim, int vdim);
cudaError_t launch_delta_rule_mma(const RecDev& d, int n_seqs, int max_new, long long rows, float* ws, cudaStream_t st);
// All chunks at once (linear_attn_mma.cu, linear_attn_tc.cu), given linear_attn_mma_floats(..) floats of 16-byte aligned scratch (0: not for this step); four launches
long long linear_attn_mma_floats(long long rows, int n_seqs, int max_new, int heads, int dim, int vdim);
template <bool TD>
cudaError_t launch_linear_attn_mma(const RecDev& d, int n_seqs, int max_new, long long rows, float* ws, cudaStream_t st);
// Where the split rows of (sequence s, key / value head g) lie: slot (s * kv_heads + g) * cap + i holds the i-th key, K hi | K lo | V hi | V lo, and the numbers
// that undo the scaling, 2^(exponent - SPLIT_TOP) of the key row and 2^exponent of the value row. Two layouts:
// - for mma.sync, channels filled up to 16, the two numbers in 16 bytes behind the row. The 16 bytes also make the distance between rows an odd multiple
//   of 16, as ldmatrix wants it in shared memory: a run of rows is one copy;
// - for tcgen05 (tail > 0), K hi | K lo filled up to a multiple of 64 entries together, V hi and V lo each, since a tensor map's box takes 128 bytes of a row;
//   the numbers in an array of their own, and `tail` rows of zeros behind a list's last, which the last tile's box may take in.
struct SplitKv {
  unsigned char* rows;
  long long cap;   // key slots per (sequence, key / value head)
  int row_bytes;
  int k_lo, v_at, v_lo;   // bytes from a key's hi halves to its lo ones, to its values, from those to their lo halves
  int vpad;        // channels that a value row's halves are filled up to
  float* unit;     // a slot's two numbers, `ustep` floats between slots
  int ustep, tail;
  uint4* range;    // [sequence, key / value head][blocks]: of a block of SPLIT_ROWS rows the largest key entry, the largest value entry and the smallest of its value
                   // rows' and columns' largest ones (zeros aside), as bits of floats
  int blocks;
  int* odd;        // [sequence, key / value head]: 1 where the keys or values are not for fp16 halves (split_odd) and the fp32 form has to do the work
};
constexpr int SPLIT_ROWS = 32;
// Are the values of list sg (all its visible rows) not for fp16 halves? A value row's halves are off by at most 2^-49 of its largest entry, and the weights' by as
// much of the largest row's in the tile, seen or not (they carry the rows' exponents). With every row's and every column's largest within 2^20 of the
// list's largest this stays below 2^-26 of what a column sums; rows or columns further apart, infinities and NaN are the fp32 form's. Read by a whole warp.
constexpr float SPLIT_RANGE = 0x1p-20f;
// Scores: a softmax or sigmoid takes a score's absolute error. With |q k scale| per channel up to 2^18 (units of q are 2^-13 of a row's largest or more) the
// halves' share is below 2^-30 a channel; larger ones are the fp32 form's
constexpr float SPLIT_SCORE = 0x1p5f;   // of units of q times largest entries of k
__device__ __forceinline__ bool split_odd(const SplitKv& w, int sg, int keys, float& top_k) {
  unsigned k = 0u, v = 0u, low = 0x7f800000u;
  for (int b = threadIdx.x & 31; b < (keys + SPLIT_ROWS - 1) / SPLIT_ROWS; b += 32) {
    const uint4 r = w.range[static_cast<long long>(sg) * w.blocks + b];
    k = max(k, r.x);
    v = max(v, r.y);
    low = min(low, r.z);
  }
  top_k = __uint_as_float(__reduce_max_sync(0xffffffffu, k));
  const float top = __uint_as_float(__reduce_max_sync(0xffffffffu, v));
  return !(top < INFINITY) || __uint_as_float(__reduce_min_sync(0xffffffffu, low)) < SPLIT_RANGE * top;
}
// splits the rows that some query of the step sees into ws (window_attn_split_floats(..) floats, 16-byte aligned), says where they are, sets `odd` to 0
cudaError_t launch_window_attn_split(const WinDev& d, int n_seqs, int max_new, float* ws, SplitKv* w, cudaStream_t st);
long long window_attn_split_floats(const WinDev& d, int n_seqs, int max_new);
// window_attn_tc.cu: the same rows for tcgen05, and the kernel that reads them (dim, vdim <= 128)
bool window_attn_tc_applies(const WinDev& d, int n_seqs, int max_new);
long long window_attn_tc_floats(const WinDev& d, int n_seqs, int max_new);
SplitKv window_attn_tc_layout(const WinDev& d, int n_seqs, int max_new, float* ws);   // of the second layout, in a workspace of that many floats
cudaError_t launch_window_attn_tc(const WinDev& d, int n_seqs, int max_new, float* ws, const int** odd, cudaStream_t st);
// key slots per (sequence, key / value head) that the step's queries can see at most (host-known bounds)
long long split_slots(const WinDev& d, int max_new);
cudaError_t launch_split_rows(const WinDev& d, int n_seqs, const SplitKv& w, cudaStream_t st);
// on the tensor cores, as many sequences at a time as the workspace holds; in fp32 where it holds none
cudaError_t launch_window_attn_prompt(const WinDev& d, int n_seqs, int max_new, float* ws, long long ws_floats, cudaStream_t st, int* launches);
// in fp32 (seqmix_tiled.cu); odd: null, or what the tensor-core form leaves to do
cudaError_t launch_window_attn_tiled(const WinDev& d, int n_seqs, int max_new, const int* odd, cudaStream_t st);
// Single tokens whose query heads share key / value rows in groups of 8 or more (latent rows): heads as the rows of a tile.
bool window_attn_heads_applies(const WinDev& d);
long long window_attn_heads_workspace_floats(int n_seqs, int heads, int kv_heads, int vdim);
cudaError_t launch_window_attn_heads(const WinDev& d, int n_seqs, float* ws, long long ws_floats, cudaStream_t st, int* launches);

}  // namespace vy
