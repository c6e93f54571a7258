// Prompt-sized linear attention with a decay per head (fixed, or per token as in the state-space recurrence), all chunks of 64 tokens at
// once, fp32 precision on the tensor cores (split_mma.cuh). Three launches:
//
//   la_states   U_c = sum_j decay(j .. end of chunk c) w_j k_j v_j^T of every chunk, and the chunk's whole decay D_c
//   la_scan     S <- D_c S + U_c chunk after chunk, element by element; the state BEFORE each chunk takes the place of U_c
//   la_outputs  O = (Q K^T . D) V + diag(decay to i) Q S_before
//
// The walk this replaces for long portions (linear_attn_chunk_kernel: one CTA per sequence, head and slice of columns goes through the chunks in
// order, on fp32 FMAs) is as long as the sequence and leaves SMs idle for few sequences; here only the scan is serial, and it is bound by the bytes
// of the states (dim x vdim x 4 per chunk and head, written twice, read twice). q and k shared by a group of heads (state space: b and c) are
// split, and their scores computed, once per group. Prompts whose rows come in quads, of a state space or with silu of q, k and v, have the
// first and the third launch on tcgen05 (linear_attn_tc.cu).
//
// The fp16 halves are off by at most 2^-49 of the largest entry under their unit, a row of q, k or v or a whole state. la_states looks at the rows (tokens) and
// columns (channels) of every chunk's q, k and v, as each warp has them, and of the state that is carried in: where the largest entry of one is below 2^-20 of the
// largest of all (rows and columns of few entries, which may all be small by chance: 2^-24; zeros aside), and where an infinity or NaN is among them, the
// heads of the CTA are left to the walk, which runs behind the three launches and starts from the state that la_scan kept as the one before the first chunk.
#include "linear_attn.cuh"
#include "seqmix.cuh"
#include "split_mma.cuh"

namespace vy {

// four entries of row `row` (element offset o of src) from column c on, zero past `width`
__device__ __forceinline__ float4 load4(const void* src, int dt, bool vec, long long o, int c, int width) {
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
  if (c >= width) return x;
  if (vec) return *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(src) + o + c);
  return load4_any(src, dt, o, c, width);
}
static __device__ __noinline__ float uact_any(float x, int act) { return apply_uact(x, act); }
// ACT: VY_UACT_NONE or VY_UACT_SILU at compile time, any other activation by a call
template <int ACT>
__device__ __forceinline__ float act_of(float x, int act) {
  if constexpr (ACT == VY_UACT_NONE) return x;
  else return act == VY_UACT_SILU ? siluf_(x) : uact_any(x, act);
}
template <int ACT>
__device__ __forceinline__ float4 act4(float4 x, int act) {
  return make_float4(act_of<ACT>(x.x, act), act_of<ACT>(x.y, act), act_of<ACT>(x.z, act), act_of<ACT>(x.w, act));
}
constexpr int LU_T = 256, LU_VB = 64 * 2 + 16;   // threads; bytes between rows of 64 value columns

// CTA: (chunk, 64 value columns) x (hp heads that share k) x sequence. Warp w owns state rows 16 w .., and it reads and splits those channels of k (eight
// tokens at a time) and value columns 8 w .. (sixteen at a time), all tokens of them: tokens are the summed index, so a channel and a column have one unit
// each, and their largest entries need no other warp. 4 x 2048 tokens, 32 heads of 128 x 64 in groups of 8: 101 us, bound by
// writing the states (134 MB) and by the latency of each chunk's few steps
// ACT: see act_of
template <bool TD, int ACT>
__global__ void __launch_bounds__(LU_T, 2) la_states_kernel(RecDev d, LaChunks w, int hp, int vslices, int dim16, bool vec) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) unsigned char lu_smem[];
  const int kb = dim16 * 2 + 16;
  unsigned char* Kh = lu_smem;
  unsigned char* Kl = Kh + LM_C * kb;
  unsigned char* Wh = Kl + LM_C * kb;
  unsigned char* Wl = Wh + LM_C * LU_VB;
  float* es = reinterpret_cast<float*>(Wl + LM_C * LU_VB);   // [64] decay to the chunk's end times write strength
  float* ku = es + LM_C;                                     // [128], [64]: units of k's channels and of w's columns
  float* wu = ku + 128;
  Range* range = reinterpret_cast<Range*>(wu + 64);          // [4]: k, q, v, state
  const int s = blockIdx.z, c = blockIdx.x / vslices, v0 = (blockIdx.x % vslices) * 64, h0 = blockIdx.y * hp;
  const int base = d.cu[s], n = d.cu[s + 1] - base, t0 = c * LM_C;
  if (t0 >= n) return;
  const int nt = min(LM_C, n - t0), t = threadIdx.x, warp = t >> 5, lane = t & 31, gq = lane >> 2, tq = lane & 3;
  const int hq = TD ? h0 / (d.heads / d.kv_heads) : h0, vw = min(64, d.vdim - v0);
  const long long r0 = base + t0, slot = la_slot(d, s, c);
  if (t < 4) range[t] = {0u, RANGE_NONE};
  __syncthreads();
  const bool few = nt < 8;
  {
    const int row = lane >> 2, ch = 16 * warp + 4 * (lane & 3);
    float4 x[LM_C / 8];
    const auto read = [&](const void* p, long long ld) {
#pragma unroll
      for (int i = 0; i < LM_C / 8; ++i) {
        const int r = row + 8 * i;
        x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < nt && ch < d.dim) x[i] = act4<ACT>(load4(p, d.in_dt, vec, (r0 + r) * ld + static_cast<long long>(hq) * d.dim, ch, d.dim), d.in_act);
      }
    };
    Range rk = {0u, RANGE_NONE}, rq = rk;
    if (v0 == 0) {
      read(d.q, d.ldq);
      look<LM_C / 8, 4>(x, few, d.dim - 16 * warp < 4, rq);
      note_warp(range + 1, rq);
    }
    read(d.k, d.ldk);
    const uint4 m = look<LM_C / 8, 4>(x, few, d.dim - 16 * warp < 4, rk);
    note_warp(range, rk);
    const float4 sc = column_scales(m);
    if (row == 0) *reinterpret_cast<float4*>(ku + ch) = column_units(m);
    if (ch < dim16) {
#pragma unroll
      for (int i = 0; i < LM_C / 8; ++i) store_split4(Kh, Kl, (row + 8 * i) * kb + ch * 2, x[i], sc);
    }
  }
  const unsigned ka = smem_addr(Kh) + lane_b(lane, kb) + 16 * warp * 2, wb = smem_addr(Wh) + lane_bt(lane, LU_VB);
  const int row = lane >> 1, vc = 8 * warp + 4 * (lane & 1);
  Range rv = {0u, RANGE_NONE}, rs = rv;   // this thread's share
  float4 next[LM_C / 16];
  const auto fetch = [&](int h) {
#pragma unroll
    for (int i = 0; i < LM_C / 16; ++i) {
      const int r = row + 16 * i;
      next[i] = r < nt ? load4(d.v, d.in_dt, vec, (r0 + r) * d.ldv + static_cast<long long>(h) * d.vdim + v0, vc, vw) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  fetch(h0);
  for (int h = h0; h < h0 + hp; ++h) {
    __syncthreads();   // the previous head's readers of es and W are done
    if constexpr (TD) {
      if (warp == 0) {
        const float whole = token_decays<LM_C / 32>(d, r0, nt, h, lane, [&](int i, double L, float strength, double end) { es[i] = expf(static_cast<float>(end - L)) * strength; });
        if (lane == 0 && v0 == 0) w.D[slot * d.heads + h] = whole;
      }
    } else if (t <= LM_C) {
      if (t < LM_C) es[t] = t < nt ? power(d.decay[h], nt - 1 - t) : 0.f;
      else if (v0 == 0) w.D[slot * d.heads + h] = power(d.decay[h], nt);
    }
    if (t == 0 && v0 == 0) w.top[slot * d.heads + h] = 0u;
    float4 y[LM_C / 16];
#pragma unroll
    for (int i = 0; i < LM_C / 16; ++i) y[i] = next[i];
    if (h + 1 < h0 + hp) fetch(h + 1);   // in flight during this head's products
    __syncthreads();
#pragma unroll
    for (int i = 0; i < LM_C / 16; ++i) {
      if (row + 16 * i < nt) y[i] = act4<ACT>(y[i], d.in_act);
    }
    uint4 m = look<LM_C / 16, 2>(y, few, vw - 8 * warp < 4, rv);
    {   // the weighted columns' units from a bound, the columns' largest times the largest weight: rows are within 2^20 of one another, and the halves good to 2^24
      unsigned top = 0u;
#pragma unroll
      for (int i = lane; i < LM_C; i += 32) top = max(top, abs_bits(es[i]));
      const float most = __uint_as_float(__reduce_max_sync(0xffffffffu, top));
      const auto times = [most](unsigned b) { return __float_as_uint(__uint_as_float(b) * most); };
      m = make_uint4(times(m.x), times(m.y), times(m.z), times(m.w));
    }
#pragma unroll
    for (int i = 0; i < LM_C / 16; ++i) {
      const float e = es[row + 16 * i];
      y[i] = make_float4(y[i].x * e, y[i].y * e, y[i].z * e, y[i].w * e);
    }
    const float4 sv = column_scales(m);
    if (row == 0) *reinterpret_cast<float4*>(wu + vc) = column_units(m);
#pragma unroll
    for (int i = 0; i < LM_C / 16; ++i) store_split4(Wh, Wl, (row + 16 * i) * LU_VB + vc * 2, y[i], sv);
    if (c == 0 && d.pos0[s] > 0) {   // the state that is carried in: a thread reads every fourth entry of a column
      const float* sp = d.state + (static_cast<long long>(d.slot[s]) * d.heads + h) * static_cast<long long>(d.dim) * d.vdim + v0 + (t & 63);
      unsigned top = 0u;
#pragma unroll 4
      for (int i = t >> 6; i < d.dim; i += 4) {
        const unsigned a = (t & 63) < vw ? abs_bits(sp[static_cast<long long>(i) * d.vdim]) : 0u, most = __reduce_max_sync(0xffffffffu, a);
        top = max(top, a);
        note(rs, most, true);
      }
      note(rs, top, true);
    }
    __syncthreads();
    if (16 * warp < dim16) {
      float a[8][4], b[8][4];   // hi hi, and the two small products
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) a[i][k] = b[i][k] = 0.f;
#pragma unroll
      for (int k = 0; k < LM_C / 16; ++k) {
        unsigned ah[4], al[4];   // k^T: stored [token][channel], read transposed (lane_b's order is what .trans turns into an A operand)
        ldsm_x4_t(ah, ka + 16 * k * kb);
        ldsm_x4_t(al, ka + LM_C * kb + 16 * k * kb);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          unsigned bh[4], bl[4];
          ldsm_x4_t(bh, wb + 16 * k * LU_VB + 32 * j);
          ldsm_x4_t(bl, wb + LM_C * LU_VB + 16 * k * LU_VB + 32 * j);
          mma_f16(b[2 * j], al, bh[0], bh[1]);
          mma_f16(b[2 * j + 1], al, bh[2], bh[3]);
          mma_f16(a[2 * j], ah, bh[0], bh[1]);
          mma_f16(a[2 * j + 1], ah, bh[2], bh[3]);
          mma_f16(b[2 * j], ah, bl[0], bl[1]);
          mma_f16(b[2 * j + 1], ah, bl[2], bl[3]);
        }
      }
      float* U = w.U + (slot * d.heads + h) * static_cast<long long>(d.dim) * d.vdim + v0;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = 16 * warp + gq + 8 * r;
        if (i >= d.dim) continue;
        const float u1 = ku[i];
        constexpr float cut = (LM_C / 16 + 1) * 0.5f * SPLIT_CUT;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int col = 8 * j + 2 * tq;
          const float2 u2 = *reinterpret_cast<const float2*>(wu + col);
          const float p = split_sum(a[j][2 * r], b[j][2 * r], cut) * u1 * u2.x, q = split_sum(a[j][2 * r + 1], b[j][2 * r + 1], cut) * u1 * u2.y;
          float* at = U + static_cast<long long>(i) * d.vdim + col;
          if (col + 1 < vw && d.vdim % 2 == 0) *reinterpret_cast<float2*>(at) = make_float2(p, q);
          else {
            if (col < vw) at[0] = p;
            if (col + 1 < vw) at[1] = q;
          }
        }
      }
    }
  }
  note_warp(range + 2, rv);
  note_warp(range + 3, rs);
  __syncthreads();
  if (t == 0) w.odd[(slot * gridDim.y + blockIdx.y) * vslices + blockIdx.x % vslices] = too_wide(range[0]) || too_wide(range[1]) || too_wide(range[2]) || too_wide(range[3]);
}

// V elements per thread. Bound by the bytes: every chunk's state read once and written once; eight chunks' worth is in flight per thread
template <int V>
__global__ void __launch_bounds__(256) la_scan_kernel(RecDev d, LaChunks w) {
  pdl_trigger();
  pdl_wait();
  constexpr int P = 8;
  const int s = blockIdx.z, h = blockIdx.y, n = d.cu[s + 1] - d.cu[s];
  if (n <= 0) return;
  const int e = (blockIdx.x * 256 + threadIdx.x) * V, each = d.dim * d.vdim, chunks = (n + w.chunk - 1) / w.chunk;
  const bool on = e < each;
  const long long first = la_slot(d, s, 0) * d.heads + h;
  float* sp = d.state + (static_cast<long long>(d.slot[s]) * d.heads + h) * each + e;
  float* U = w.U + first * each + e;
  const long long step = static_cast<long long>(d.heads) * each;
  float S[V], u[P][V], D[P];
  const auto get = [&](const float* p, float (&x)[V]) {
    if constexpr (V == 4) {
      const float4 f = *reinterpret_cast<const float4*>(p);
      x[0] = f.x; x[1] = f.y; x[2] = f.z; x[3] = f.w;
    } else x[0] = *p;
  };
  const auto put = [&](float* p, const float (&x)[V]) {
    if constexpr (V == 4) *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
    else *p = x[0];
  };
#pragma unroll
  for (int k = 0; k < V; ++k) S[k] = 0.f;
  if (on && d.pos0[s] > 0) get(sp, S);
  for (int c0 = 0; c0 < chunks; c0 += P) {
#pragma unroll
    for (int p = 0; p < P; ++p)
      if (on && c0 + p < chunks) {
        get(U + (c0 + p) * step, u[p]);
        D[p] = w.D[first + static_cast<long long>(c0 + p) * d.heads];
      }
#pragma unroll
    for (int p = 0; p < P; ++p) {
      if (c0 + p >= chunks) break;
      const long long at = first + static_cast<long long>(c0 + p) * d.heads;
      float m = 0.f;
      if (on) {
        put(U + (c0 + p) * step, S);
#pragma unroll
        for (int k = 0; k < V; ++k) m = fmaxf(m, fabsf(S[k]));
      }
      const unsigned mb = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
      if ((threadIdx.x & 31) == 0 && mb) atomicMax(w.top + at, mb);
      if (on) {
#pragma unroll
        for (int k = 0; k < V; ++k) S[k] = fmaf(D[p], S[k], u[p][k]);
      }
    }
  }
  if (on) put(sp, S);
}

constexpr int LO_T = 128, LO_W = 4;

// CTA: (chunk, 64 value columns) x (hp heads that share q and k) x sequence; warp w owns tokens 16 w .. 16 w + 15 and keeps their scores in registers
// for all its heads. 4 x 2048 tokens, 32 heads of 128 x 64 in groups of 8: 292 us (la_scan 83; the walk over the chunks was 737 us for everything). Bound by
// fixed latencies at two warps per scheduler (255 registers): the tensor pipe is 13 % active; twice the warps with half the columns: 301 us
template <bool TD, int ACT>
__global__ void __launch_bounds__(LO_T, 2) la_outputs_kernel(RecDev d, LaChunks w, int hp, int vslices, int dim16, bool vec, bool svec) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) unsigned char lo_smem[];
  const int kb = dim16 * 2 + 16, q_lo = LM_C * kb, v_lo = LM_C * LU_VB, s_lo = dim16 * LU_VB;
  unsigned char* Qh = lo_smem;
  unsigned char* Kh = Qh + 2 * q_lo;   // k until the scores are done, then V and the state of one head after the other
  unsigned char* Vh = Kh;
  unsigned char* Sh = Vh + 2 * v_lo;
  float* sc = reinterpret_cast<float*>(Kh + max(2 * q_lo, 2 * v_lo + 2 * s_lo));
  float *qu = sc, *ku = qu + LM_C, *vu = ku + LM_C, *Lh = vu + LM_C, *Ll = Lh + LM_C, *wr = Ll + LM_C, *eL = wr + LM_C;   // [64] each (eL: decay up to and with token i)
  const int s = blockIdx.z, c = blockIdx.x / vslices, v0 = (blockIdx.x % vslices) * 64, h0 = blockIdx.y * hp;
  const int base = d.cu[s], n = d.cu[s + 1] - base, t0 = c * LM_C;
  if (t0 >= n) return;
  const int nt = min(LM_C, n - t0), t = threadIdx.x, warp = t >> 5, lane = t & 31, gq = lane >> 2, tq = lane & 3;
  const int hq = TD ? h0 / (d.heads / d.kv_heads) : h0, vw = min(64, d.vdim - v0);
  const long long r0 = base + t0, slot = la_slot(d, s, c);
  const int act = d.in_act;
  const auto map = [act] {
    if constexpr (ACT == VY_UACT_NONE) return SameValue();
    else return [act](float x) { return act_of<ACT>(x, act); };
  }();
  split_rows<LO_W, 128>(Qh, Qh + q_lo, kb, qu, SPLIT_TOP, LM_C, d.dim, dim16, d.q, d.in_dt, vec,
                        [&](int r) { return r < nt ? (r0 + r) * d.ldq + static_cast<long long>(hq) * d.dim : -1LL; }, map);
  split_rows<LO_W, 128>(Kh, Kh + q_lo, kb, ku, SPLIT_TOP, LM_C, d.dim, dim16, d.k, d.in_dt, vec,
                        [&](int r) { return r < nt ? (r0 + r) * d.ldk + static_cast<long long>(hq) * d.dim : -1LL; }, map);
  __syncthreads();
  const unsigned qa = smem_addr(Qh) + 16 * warp * kb + lane_a(lane, kb), kk = smem_addr(Kh) + lane_b(lane, kb);
  const unsigned va = smem_addr(Vh) + lane_bt(lane, LU_VB), sa = smem_addr(Sh) + lane_bt(lane, LU_VB);
  const int i0 = 16 * warp + gq;   // this lane's rows: i0 and i0 + 8
  const float qunit[2] = {qu[i0], qu[i0 + 8]};
  const float cut = (dim16 / 16 + 1) * 0.5f * SPLIT_CUT, vcut = (warp + 2) * 0.5f * SPLIT_CUT;   // sums over the channels, over the tokens this warp sees
  float p[8][4];   // scores q_i . k_j; a warp's tokens only see keys j < 16 (warp + 1)
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float a[2][4], b[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) a[i][e] = b[i][e] = 0.f;
    if (j <= warp) {
      for (int k = 0; k < dim16; k += 16) {
        unsigned ah[4], al[4], bh[4], bl[4];
        ldsm_x4(ah, qa + 2 * k);
        ldsm_x4(al, qa + q_lo + 2 * k);
        ldsm_x4(bh, kk + 16 * j * kb + 2 * k);
        ldsm_x4(bl, kk + q_lo + 16 * j * kb + 2 * k);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          mma_f16(b[i], al, bh[2 * i], bh[2 * i + 1]);
          mma_f16(a[i], ah, bh[2 * i], bh[2 * i + 1]);
          mma_f16(b[i], ah, bl[2 * i], bl[2 * i + 1]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) p[2 * j + i][e] = split_sum(a[i][e], b[i][e], cut) * qunit[e >> 1] * ku[16 * j + 8 * i + 2 * tq + (e & 1)];
  }
  for (int h = h0; h < h0 + hp; ++h) {
    __syncthreads();   // the readers of k, or of the previous head's values and state, are done
    float skip = 0.f;
    if constexpr (TD) {
      skip = ld_as_float(d.skip, d.a_log_dt, h);
      if (warp == 0) {
        token_decays<LM_C / 32>(d, r0, nt, h, lane, [&](int i, double L, float strength, double) {   // two floats: the sums' differences are what counts
          Lh[i] = static_cast<float>(L);
          Ll[i] = static_cast<float>(L - static_cast<double>(Lh[i]));
          wr[i] = strength;
          eL[i] = expf(Lh[i]);
        });
      }
    } else if (t <= LM_C) {   // decay^t: wr, shifted by one: eL
      const float x = power(d.decay[h], t);
      if (t < LM_C) wr[t] = x;
      if (t > 0) eL[t - 1] = x;
    }
    const int es = split_exponent(__uint_as_float(w.top[slot * d.heads + h]));
    const float* U = w.U + (slot * d.heads + h) * static_cast<long long>(d.dim) * d.vdim + v0;
    float4 x[8];   // sixteen threads per state row, eight rows in flight (beside the values')
    const auto get = [&](int i) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int r = i + k * (LO_T / 16);
        x[k] = r < d.dim ? load4(U, VY_F32, svec, static_cast<long long>(r) * d.vdim, (t & 15) * 4, vw) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    get(t >> 4);
    split_rows<LO_W, 64>(Vh, Vh + v_lo, LU_VB, vu, 0, LM_C, vw, 64, d.v, d.in_dt, vec,
                         [&](int r) { return r < nt ? (r0 + r) * d.ldv + static_cast<long long>(h) * d.vdim + v0 : -1LL; }, map);
    for (int i = t >> 4; i < dim16; i += 8 * (LO_T / 16)) {
      if (i >= 8 * (LO_T / 16)) get(i);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int r = i + k * (LO_T / 16);
        if (r < dim16) store_split4(Sh, Sh + s_lo, r * LU_VB + (t & 15) * 8, x[k], make_float4(split_scale(es), split_scale(es), split_scale(es), split_scale(es)));
      }
    }
    __syncthreads();
    // what the earlier chunks left: Q S
    float o[8][4];
    {
      float b[8][4];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[i][e] = b[i][e] = 0.f;
      for (int k = 0; k < dim16; k += 16) {
        unsigned ah[4], al[4];
        ldsm_x4(ah, qa + 2 * k);
        ldsm_x4(al, qa + q_lo + 2 * k);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          unsigned bh[4], bl[4];
          ldsm_x4_t(bh, sa + k * LU_VB + 32 * j);
          ldsm_x4_t(bl, sa + s_lo + k * LU_VB + 32 * j);
          mma_f16(b[2 * j], al, bh[0], bh[1]);
          mma_f16(b[2 * j + 1], al, bh[2], bh[3]);
          mma_f16(o[2 * j], ah, bh[0], bh[1]);
          mma_f16(o[2 * j + 1], ah, bh[2], bh[3]);
          mma_f16(b[2 * j], ah, bl[0], bl[1]);
          mma_f16(b[2 * j + 1], ah, bl[2], bl[3]);
        }
      }
      const float su = pow2i(es - SPLIT_TOP);
      const float f[2] = {qunit[0] * eL[i0], qunit[1] * eL[i0 + 8]};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[i][e] = split_sum(o[i][e], b[i][e], cut) * su * f[e >> 1];
    }
    // the weights inside the chunk, times the exponent of each value row, then scaled row by row
    unsigned ph[4][4], pl[4][4];
    float pu[2];
    {
      float x[8][4], top[2] = {0.f, 0.f};
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = i0 + 8 * (e >> 1), k = 8 * j + 2 * tq + (e & 1);
          float y = 0.f;
          if (k <= i && j < 2 * (warp + 1)) {
            if constexpr (TD) {
              y = p[j][e] * (expf((Lh[i] - Lh[k]) + (Ll[i] - Ll[k])) * wr[k]);
              if (k == i) y += skip;
            } else y = p[j][e] * wr[i - k];
            y *= vu[k];
          }
          x[j][e] = y;
          top[e >> 1] = fmaxf(top[e >> 1], fabsf(y));
        }
      float f[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], 1));
        top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], 2));
        const int e = split_exponent(top[r]);
        f[r] = split_scale(e);
        pu[r] = pow2i(e - SPLIT_TOP);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        split2(x[j][0] * f[0], x[j][1] * f[0], ph[j >> 1][(j & 1) * 2], pl[j >> 1][(j & 1) * 2]);
        split2(x[j][2] * f[1], x[j][3] * f[1], ph[j >> 1][(j & 1) * 2 + 1], pl[j >> 1][(j & 1) * 2 + 1]);
      }
    }
    const float v_unit = pow2i(-SPLIT_TOP);
    const bool pairs = svec && d.out_dt == VY_F32 && vw % 2 == 0;   // svec: vdim, strides and bases also suit pairs
    float2 gate[2][8];   // in flight during the products below
    if constexpr (TD) {
      if (pairs && d.gate) {
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int i = i0 + 8 * r, col = 8 * j + 2 * tq;
            if (i < nt && col < vw) gate[r][j] = *reinterpret_cast<const float2*>(d.gate + (r0 + i) * d.ld_gate + static_cast<long long>(h) * d.vdim + v0 + col);
          }
      }
    }
#pragma unroll
    for (int cb = 0; cb < 2; ++cb) {
      float a[4][4], b[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) a[i][e] = b[i][e] = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (k > warp) break;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          unsigned bh[4], bl[4];
          ldsm_x4_t(bh, va + 16 * k * LU_VB + 64 * cb + 32 * j);
          ldsm_x4_t(bl, va + v_lo + 16 * k * LU_VB + 64 * cb + 32 * j);
          mma_f16(b[2 * j], pl[k], bh[0], bh[1]);
          mma_f16(b[2 * j + 1], pl[k], bh[2], bh[3]);
          mma_f16(a[2 * j], ph[k], bh[0], bh[1]);
          mma_f16(a[2 * j + 1], ph[k], bh[2], bh[3]);
          mma_f16(b[2 * j], ph[k], bl[0], bl[1]);
          mma_f16(b[2 * j + 1], ph[k], bl[2], bl[3]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[4 * cb + i][e] = fmaf(split_sum(a[i][e], b[i][e], vcut), pu[e >> 1] * v_unit, o[4 * cb + i][e]);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int i = i0 + 8 * r;
      if (i >= nt) continue;
      const long long ob = (r0 + i) * d.ld_out + static_cast<long long>(h) * d.vdim + v0, gb = (r0 + i) * d.ld_gate + static_cast<long long>(h) * d.vdim + v0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int col = 8 * j + 2 * tq;
        float y0 = o[j][2 * r], y1 = o[j][2 * r + 1];
        if (pairs) {
          if (col >= vw) continue;
          if constexpr (TD) {
            if (d.gate) {
              y0 *= act_of<VY_UACT_SILU>(gate[r][j].x, d.gate_act);
              y1 *= act_of<VY_UACT_SILU>(gate[r][j].y, d.gate_act);
            }
          }
          *reinterpret_cast<float2*>(reinterpret_cast<float*>(d.out) + ob + col) = make_float2(y0, y1);
        } else {
          if constexpr (TD) {
            if (d.gate && col < vw) y0 *= uact_any(d.gate[gb + col], d.gate_act);
            if (d.gate && col + 1 < vw) y1 *= uact_any(d.gate[gb + col + 1], d.gate_act);
          }
          store2_any(d.out, d.out_dt, ob + col, y0, y1, vw - col);
        }
      }
    }
  }
}

// From three chunks on: us, here / walk, 16 heads of 128 x 64, one portion of 70, 130, 300 tokens 27 / 24, 28 / 35, 28 / 60; 32 of 130, 300: 195 / 187, 311 / 330. Every
// sequence has a chunk at least, which here costs two passes over its state more than in the walk, while the walk takes about 10 us per chunk of the longest portion. So
// where portions are uneven these launches pay from about 2 / 3 token per chunk and head on: one of 200, 400, 512 beside 31 single tokens 88 / 62, 103 / 107, 105 / 125, one of
// 200 beside 7 41 / 53; state space, 32 heads of 128 x 64, one of 130, 400 beside 31 312 / 156, 328 / 173
long long linear_attn_mma_floats(long long rows, int n_seqs, int max_new, int heads, int dim, int vdim) {
  if (max_new <= 2 * LM_C || dim > 128 || rows <= 0) return 0;
  const long long slots = rows / LM_C + n_seqs;
  if (2 * rows < static_cast<long long>(n_seqs) * max_new && 3LL * max_new < 2 * slots * heads * ((vdim + 63) / 64) * (dim + 64) / 192) return 0;
  const long long floats = slots * heads * (static_cast<long long>(dim) * vdim + 2 + (vdim + 63) / 64) + 4;
  return floats <= (1LL << 28) ? floats : 0;   // 1 GB: past it the walk, which keeps its state on the chip
}

template <bool TD, int ACT>
static cudaError_t launch_la_mma(const RecDev& d, int n_seqs, int max_new, long long rows, float* ws, cudaStream_t st) {
  const auto al = [](const void* p, long long ld, int a) { return reinterpret_cast<uintptr_t>(p) % (4 * a) == 0 && ld % a == 0; };
  const bool vec = d.in_dt == VY_F32 && d.dim % 4 == 0 && d.vdim % 4 == 0 && al(d.q, d.ldq, 4) && al(d.k, d.ldk, 4) && al(d.v, d.ldv, 4);
  const bool svec = d.vdim % 4 == 0 && (d.out_dt != VY_F32 || al(d.out, d.ld_out, 2)) && (!d.gate || al(d.gate, d.ld_gate, 2));
  const long long slots = rows / LM_C + n_seqs;
  LaChunks w;
  w.U = ws;
  w.D = ws + slots * d.heads * static_cast<long long>(d.dim) * d.vdim;
  w.top = reinterpret_cast<unsigned*>(w.D + slots * d.heads);
  w.odd = reinterpret_cast<int*>(w.top + slots * d.heads);
  const bool quad = d.vdim % 4 == 0 && reinterpret_cast<uintptr_t>(d.state) % 16 == 0 && reinterpret_cast<uintptr_t>(ws) % 16 == 0;
  const int vslices = (d.vdim + 63) / 64, tc_hp = vec && quad ? linear_attn_tc_heads(d, n_seqs, max_new, rows, vslices) : 0;
  const bool tc = tc_hp > 0;
  const int C = w.chunk = tc ? LT_C : LM_C;
  const int dim16 = (d.dim + 15) & ~15, kb = dim16 * 2 + 16, chunks = (max_new + C - 1) / C;
  // heads per CTA: those that share q and k, fewer while that leaves less than two CTAs per SM
  int hp = TD ? d.heads / d.kv_heads : 1;
  if (tc) hp = tc_hp;
  else
    while (hp % 2 == 0 && slots * vslices * (d.heads / hp) < 2LL * num_sms()) hp /= 2;
  const dim3 grid(static_cast<unsigned>(chunks) * vslices, d.heads / hp, n_seqs);
  const size_t smem_u = 2 * LM_C * static_cast<size_t>(kb) + 2 * LM_C * LU_VB + sizeof(float) * (LM_C + 128 + 64) + 4 * sizeof(Range);
  const size_t q2 = 2 * LM_C * static_cast<size_t>(kb), vs = 2 * LM_C * LU_VB + 2 * static_cast<size_t>(dim16) * LU_VB;
  const size_t smem_o = q2 + (q2 > vs ? q2 : vs) + sizeof(float) * 7 * LM_C;
  static std::atomic<unsigned long long> allowed_u{0}, allowed_o{0};
  cudaError_t e;
  if (tc) e = launch_la_states_tc(d, w, hp, n_seqs, max_new, rows, st);
  else {
    e = allow_smem(la_states_kernel<TD, ACT>, allowed_u);
    if (e == cudaSuccess) e = launch_kernel(la_states_kernel<TD, ACT>, grid, dim3(LU_T), smem_u, st, d, w, hp, vslices, dim16, vec);
  }
  if (e != cudaSuccess) return e;
  const int each = d.dim * d.vdim;
  const int per = 256 * (quad ? 4 : 1);
  const dim3 sgrid((each + per - 1) / per, d.heads, n_seqs);
  e = quad ? launch_kernel(la_scan_kernel<4>, sgrid, dim3(256), 0, st, d, w) : launch_kernel(la_scan_kernel<1>, sgrid, dim3(256), 0, st, d, w);
  if (e != cudaSuccess) return e;
  if (tc) e = launch_la_outputs_tc(d, w, hp, n_seqs, max_new, rows, st);
  else {
    e = allow_smem(la_outputs_kernel<TD, ACT>, allowed_o);
    if (e == cudaSuccess) e = launch_kernel(la_outputs_kernel<TD, ACT>, grid, dim3(LO_T), smem_o, st, d, w, hp, vslices, dim16, vec, svec && quad);
  }
  if (e != cudaSuccess) return e;
  RecDev r = d;   // the walk, for what is left to it
  r.odd = w.odd;
  r.odd_heads = hp;
  r.odd_each = tc && !TD ? 1 : vslices;   // that form's CTAs have all columns of a head
  r.odd_chunk = C;
  r.first = w.U;
  return TD ? launch_ssd_chunked(r, n_seqs, st) : launch_linear_attn_chunked(r, n_seqs, st);
}

template <bool TD>
cudaError_t launch_linear_attn_mma(const RecDev& d, int n_seqs, int max_new, long long rows, float* ws, cudaStream_t st) {
  if constexpr (!TD) {
    if (d.in_act != VY_UACT_NONE) return launch_la_mma<TD, VY_UACT_SILU>(d, n_seqs, max_new, rows, ws, st);
  }
  return launch_la_mma<TD, VY_UACT_NONE>(d, n_seqs, max_new, rows, ws, st);
}
template cudaError_t launch_linear_attn_mma<false>(const RecDev&, int, int, long long, float*, cudaStream_t);
template cudaError_t launch_linear_attn_mma<true>(const RecDev&, int, int, long long, float*, cudaStream_t);

}  // namespace vy
