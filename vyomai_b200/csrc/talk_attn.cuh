// Shared by the forms of the attention whose heads exchange scores (talking_attn.cu, talk_attn_mma.cu).
#pragma once
#include "seqmix.cuh"

namespace vy {

struct TalkDev {
  const int* cu; const int* pos0; const int* table; int tw, bs;
  const void* q; long long ldq; int q_dt;
  const void* kp; const void* vp; int pool_dt;
  int heads, kv_heads, dim, vdim;
  float scale, softcap; int window;
  const void* talk; int talk_dt;
  const void* sink; int sink_dt; int zero_sink;
  const void* gate; long long ld_gate; int gate_dt; int gate_ch;
  void* out; long long ld_out; int out_dt;
  const int* odd;   // null, or [sequence][key / value head]: sequences without a 1 are done (by talk_attn_mma_kernel)
};

// the extra softmax term of head h as (score, present)
__device__ __forceinline__ bool sink_of(const TalkDev& d, int h, float& s) {
  if (d.sink) { s = ld_as_float(d.sink, d.sink_dt, h); return true; }
  s = 0.f;
  return d.zero_sink != 0;
}

__device__ __forceinline__ float gate_of(const TalkDev& d, long long row, int h, int c) {
  if (!d.gate) return 1.f;
  return sigmoidf_(ld_as_float(d.gate, d.gate_dt, row * d.ld_gate + (d.gate_ch ? static_cast<long long>(h) * d.vdim + c : h)));
}

// Prompts on the tensor cores (talk_attn_mma.cu), given talk_attn_mma_floats(..) floats of 16-byte aligned scratch (0: not for this geometry); two launches
long long talk_attn_mma_floats(const TalkDev& d, int n_seqs, int max_new);
cudaError_t launch_talk_attn_mma(const TalkDev& d, int n_seqs, int max_new, float* ws, const int** odd, cudaStream_t st);   // odd: what the fp32 tiles have to do

// talk_attn_tc.cu: the same on tcgen05, from rows in window_attn_tc's layout. Does it pay? Never for more sequences where it does not for fewer
bool talk_attn_tc_applies(const TalkDev& d, int n_seqs, int max_new);
cudaError_t launch_talk_attn_tc(const TalkDev& d, const WinDev& keys, int n_seqs, int max_new, float* ws, const int** odd, cudaStream_t st);

}  // namespace vy
