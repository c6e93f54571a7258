// Gated delta rule with a decay per channel, prompts: 16 tokens per step of the serial walk, on the tensor cores in fp32 precision
// (split_mma.cuh). Per head, with the state S [dim, vdim] before a chunk of 16 tokens, the products G_t of the chunk's decays up to token t
// and k / q the unit vectors, the 16 writes u_t and read-outs o_t solve
//   u_t + beta_t sum_{s < t} A_ts u_s = beta_t (v_t - S^T (G_t k_t)),      A_ts = k_t . (G_t / G_s k_s)
//   o_t = S^T (G_t q_t) + sum_{s <= t} B_ts u_s,                           B_ts = q_t . (G_t / G_s k_s)
//   S <- G_15 S + sum_s (G_15 / G_s k_s) u_s^T
// The quotients are products of the decays between s and t or exponentials of sums: nothing is divided, no underflow matters. Solving the triangular 16 x 16 system for
// the columns of V and of G k at once gives W v and P with u = W v - P S. Two launches:
//   delta_chunk_kernel   all chunks in parallel: A and B, then W v, P, G q, G_15 / G_s k, split into fp16 pairs and stored in the
//                        register layout of the second launch's operands
//   delta_scan_kernel    the walk. It is transposed (S^T: a warp owns 16 value columns and all channels), so that the state in accumulator
//                        registers is the next product's A operand, the writes likewise, and no warp waits for another one
//   delta_scan_split_kernel   the same with a warp for every 32 channels, whose shares of the read-outs meet in shared memory once per chunk
// The walk token by token (delta_rule_kernel) is bound by its chain of two reductions per token: 46 + 1013 us with its preparation for 4 x 2048
// tokens, 8 heads of 128 x 128; here 120 + 180 us. The first launch is bound by instructions, 85 million of them (decays, exponentials, sums over pairs of tokens; with
// W made first, a column of it per lane, and channels loaded one by one 126 million, 163 us), the second by the latency of a warp's chain: 1.4 us per chunk, 1.8 where one
// warp has all channels (236 us). Error against 64 bits at decays near 1: 2e-7 instead of 1.6e-6.
#include "seqmix.cuh"
#include "split_mma.cuh"

namespace vy {
namespace {

constexpr int DC_T = 16;            // tokens per chunk
constexpr int DC_KTOP = 15;         // the decayed unit keys are split in units of 2^-15: their entries are at most 1
constexpr int DC_NW = 2;            // warps of the walk's CTA where each has all channels: 32 value columns
constexpr int DC_NS = 3;            // chunks in flight per CTA of the walk
// What the accumulations cut off (split_mma.cuh) is added back: read-outs are off by -5.8e-8 on average without it, -0.4e-8 with it, in the serial walk +0.5e-8

// One chunk and head in the workspace. An operand entry is 16 bytes per lane: (b0, b1) of mma.m16n8k16, hi then lo
template <int DP>
struct DcBlob {
  static constexpr int q_at = 64 * DP, k_at = 128 * DP, b_at = 192 * DP, g_at = b_at + 1024, unit_at = g_at + 4 * DP, bytes = unit_at + 3 * 64;
};

struct DeltaChunks {
  unsigned char* blobs;   // [slot][head] DcBlob
  float* wv;              // [slot][head][vpad / 16][32 lanes][8]: W v as accumulator registers
  int vpad;
};

// a sequence's first chunk slot: cu[s] / 16 + s, so that sequences never overlap and rows / 16 + n_seqs slots suffice
__device__ __forceinline__ long long chunk_slot0(int base, int s) { return base / DC_T + s; }

// log(1 + e^x): with t = e^-|x| and z = t / (2 + t) <= 1/3 the logarithm of 1 + t is 2 artanh(z), whose series is cut off below 2^-29. What rounding 2 + t and z leaves over
// goes into the small term: off by 0.58 of 2^-24 in the mean square, as a logarithm of 1 + e^x rounded twice
__device__ __forceinline__ float softplus_near(float x) {
  const float t = expf(-fabsf(x)), y = 2.f + t, r0 = vy_rcp_approx(y), r = fmaf(r0, fmaf(-y, r0, 1.f), r0), z = t * r, w = z * z;
  const float left = fmaf(-z, t - (y - 2.f), fmaf(-z, y, t)) * r;
  float p = fmaf(w, 1.f / 15.f, 1.f / 13.f);
  p = fmaf(w, p, 1.f / 11.f);
  p = fmaf(w, p, 1.f / 9.f);
  p = fmaf(w, p, 1.f / 7.f);
  p = fmaf(w, p, 1.f / 5.f);
  p = fmaf(w, p, 1.f / 3.f);
  return fmaxf(x, 0.f) + (2.f * z + fmaf(2.f * z * w, p, 2.f * left));
}

template <int DP>
__global__ void __launch_bounds__(256, 4) delta_chunk_kernel(RecDev d, DeltaChunks w, bool vec) {
  pdl_trigger();
  pdl_wait();
  using Blob = DcBlob<DP>;
  constexpr int LD = DP + 4, LV = 132, LA = DC_T + 4, Q4 = DP / 4, PER = (DC_T * Q4 + 255) / 256;   // Q4 lanes hold a token, four channels each
  __shared__ __align__(16) float ks[DC_T][LD], qs[DC_T][LD], gs[DC_T][LD], xs[DC_T][LD], vs[DC_T][LV], As[DC_T][LA];   // As: [s][t] -A_ts
  __shared__ float B[DC_T][DC_T + 1], beta[DC_T], scale[3][DC_T];
  const int s = blockIdx.z, h = blockIdx.y, t0 = blockIdx.x * DC_T;
  const int base = d.cu[s], n = d.cu[s + 1] - base;
  if (t0 >= n) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nt = min(DC_T, n - t0);
  const int gq = h / (d.heads / d.kv_heads);
  const long long row0 = base + t0, at = (chunk_slot0(base, s) + blockIdx.x) * d.heads + h;
  unsigned char* blob = w.blobs + at * Blob::bytes;
  {   // unit vectors, decays and what a token reads of itself
    const int c = 4 * (tid % Q4);
    const float neg_rate = -expf(ld_as_float(d.a_log, d.a_log_dt, h)), top = 1.f / sqrtf(static_cast<float>(d.dim));
    if (tid < DC_T) beta[tid] = tid < nt ? sigmoidf_(ld_as_float(d.b, d.b_dt, (row0 + tid) * d.ld_b + h)) : 0.f;
    float4 q[PER], k[PER], a[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int t = tid / Q4 + 256 / Q4 * u;
      const long long oq = (row0 + t) * d.ldq + static_cast<long long>(gq) * d.dim, ok = (row0 + t) * d.ldk + static_cast<long long>(gq) * d.dim,
                      oa = (row0 + t) * d.ld_a + static_cast<long long>(h) * d.dim;
      q[u] = k[u] = a[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t < nt && c < d.dim) {
        if (vec) {
          q[u] = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(d.q) + oq + c);
          k[u] = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(d.k) + ok + c);
          a[u] = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(d.a) + oa + c);
        } else {
          q[u] = load4_any(d.q, d.in_dt, oq, c, d.dim);
          k[u] = load4_any(d.k, d.in_dt, ok, c, d.dim);
          a[u] = load4_any(d.a, d.a_dt, oa, c, d.dim);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int t = tid / Q4 + 256 / Q4 * u;
      float sq = dot4(q[u], q[u], 0.f), sk = dot4(k[u], k[u], 0.f);
#pragma unroll
      for (int o = 1; o < Q4; o <<= 1) {
        sq += __shfl_xor_sync(0xffffffffu, sq, o);
        sk += __shfl_xor_sync(0xffffffffu, sk, o);
      }
      const float qn = t < nt ? top / sqrtf(sq + d.unit_eps) : 0.f, kn = t < nt ? 1.f / sqrtf(sk + d.unit_eps) : 0.f;
      const float4 uq = make_float4(q[u].x * qn, q[u].y * qn, q[u].z * qn, q[u].w * qn), uk = make_float4(k[u].x * kn, k[u].y * kn, k[u].z * kn, k[u].w * kn);
      float own = dot4(uq, uk, 0.f);
#pragma unroll
      for (int o = 1; o < Q4; o <<= 1) own += __shfl_xor_sync(0xffffffffu, own, o);
      if (DC_T * Q4 < 256 && t >= DC_T) continue;
      if (c == 0) B[t][t] = own;
      const auto x_of = [&](float v, int i) { return t < nt && c + i < d.dim ? neg_rate * softplus_near(v) : 0.f; };
      const float4 x = make_float4(x_of(a[u].x, 0), x_of(a[u].y, 1), x_of(a[u].z, 2), x_of(a[u].w, 3));
      *reinterpret_cast<float4*>(&qs[t][c]) = uq;
      *reinterpret_cast<float4*>(&ks[t][c]) = uk;
      *reinterpret_cast<float4*>(&xs[t][c]) = x;
      *reinterpret_cast<float4*>(&gs[t][c]) = make_float4(expf(x.x), expf(x.y), expf(x.z), expf(x.w));
    }
  }
  __syncthreads();
  {   // A and B: sixteen lanes carry G_t / G_s k_s through the tokens t after s, for s = warp and s = 15 - warp
    constexpr int RP = (DP + 63) / 64;
    const int l16 = lane & 15, sl = lane & 16 ? 15 - warp : warp, c = DP < 64 ? 4 * (l16 & 7) : 4 * l16;
    const bool idle = DP < 64 && l16 >= 8;
    f32x2 D[RP][2];
#pragma unroll
    for (int m = 0; m < RP; ++m) {
      const float4 v = f4(&ks[sl][c + 64 * m]);
      D[m][0] = idle ? pair(0.f) : pair(v.x, v.y);
      D[m][1] = idle ? pair(0.f) : pair(v.z, v.w);
    }
#pragma unroll 1
    for (int t = warp + 1; t < DC_T; ++t) {
      float a = 0.f, b = 0.f;
      if (t > sl) {
        f32x2 sa = pair(0.f), sb = pair(0.f);
#pragma unroll
        for (int m = 0; m < RP; ++m) {
          const float4 gt = f4(&gs[t][c + 64 * m]), kt = f4(&ks[t][c + 64 * m]), qt = f4(&qs[t][c + 64 * m]);
          D[m][0] = mul2(D[m][0], pair(gt.x, gt.y));
          D[m][1] = mul2(D[m][1], pair(gt.z, gt.w));
          sa = fma2(D[m][0], pair(kt.x, kt.y), sa);
          sb = fma2(D[m][0], pair(qt.x, qt.y), sb);
          sa = fma2(D[m][1], pair(kt.z, kt.w), sa);
          sb = fma2(D[m][1], pair(qt.z, qt.w), sb);
        }
        const float2 ya = unpair(sa), yb = unpair(sb);
        a = ya.x + ya.y;
        b = yb.x + yb.y;
        if (idle) a = b = 0.f;
      }
      __syncwarp();
      const float other = __shfl_xor_sync(0xffffffffu, lane & 8 ? a : b, 8);   // the first eight lanes of sixteen go on with a, the others with b
      float y = (lane & 8 ? b : a) + other;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
      if (t > sl && (lane & 7) == 0) (lane & 8 ? B[t][sl] : As[sl][t]) = lane & 8 ? y : -y;
    }
  }
  __syncthreads();
  // The triangular system, a column per thread: those of G k by the first half of the threads, those of V by the other. A later token never enters an earlier one's
  // sum, not even times zero
  const auto solve = [&](float (&r)[DC_T]) {   // what the earlier tokens take away is summed by itself: it is small beside most entries, whose rounding would be that of every term
    float less[DC_T];
#pragma unroll
    for (int t = 0; t < DC_T; ++t) less[t] = 0.f;
#pragma unroll
    for (int i = 0; i < DC_T; ++i) {
      const float x = r[i] = fmaf(beta[i], r[i], beta[i] * less[i]);
#pragma unroll
      for (int t = i & ~3; t < DC_T; t += 4) {
        if (t + 3 == i) continue;
        const float4 m = f4(&As[i][t]);
        if (t > i) less[t] = fmaf(m.x, x, less[t]);
        if (t + 1 > i) less[t + 1] = fmaf(m.y, x, less[t + 1]);
        if (t + 2 > i) less[t + 2] = fmaf(m.z, x, less[t + 2]);
        less[t + 3] = fmaf(m.w, x, less[t + 3]);
      }
    }
  };
  // G_t and G_15 / G_s are exponentials of sums of the decays' logarithms: an fp32 decay near 1 is off by a share of its distance from 1 that a product over a long
  // memory multiplies
  const int ch = tid & 127;
  const auto value_column = [&](int c) {   // W v of column c, into vs
    float r[DC_T];
#pragma unroll
    for (int t = 0; t < DC_T; ++t) r[t] = t < nt && c < d.vdim ? ld_as_float(d.v, d.in_dt, (row0 + t) * d.ldv + static_cast<long long>(h) * d.vdim + c) : 0.f;
    solve(r);
#pragma unroll
    for (int t = 0; t < DC_T; ++t) vs[t][c & 127] = r[t];
  };
  float r[DC_T];
  if (tid >= 128) {
    if (ch < DP) {
      float x = 0.f;
#pragma unroll
      for (int t = DC_T - 1; t >= 0; --t) {
        gs[t][ch] = ks[t][ch] * expf(x);
        x += xs[t][ch];
      }
    }
    value_column(ch);
  } else if (ch < DP) {
    float x = 0.f;
#pragma unroll
    for (int t = 0; t < DC_T; ++t) {
      const float G = expf(x += xs[t][ch]);
      qs[t][ch] *= G;
      r[t] = ks[t][ch] * G;
      if (t == DC_T - 1) reinterpret_cast<float*>(blob + Blob::g_at)[ch] = G;
    }
    solve(r);
  }
  __syncthreads();
  if (tid < DP)
#pragma unroll
    for (int t = 0; t < DC_T; ++t) xs[t][ch] = r[t];   // P
  const int l4 = lane >> 2, tq = 2 * (lane & 3);
  const auto store_values = [&](int c0) {   // entry lane of 16 columns holds columns l4, l4 + 8 of tokens tq, tq + 1, tq + 8, tq + 9
    const int b16 = (c0 >> 4) + warp;
    if (16 * b16 >= w.vpad) return;
    float x[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = vs[tq + 8 * (e >> 2) + (e & 1)][16 * warp + l4 + 8 * ((e >> 1) & 1)];
    float4* o = reinterpret_cast<float4*>(w.wv + (at * (w.vpad / 16) + b16) * 256 + lane * 8);
    o[0] = make_float4(x[0], x[1], x[2], x[3]);
    o[1] = make_float4(x[4], x[5], x[6], x[7]);
  };
  store_values(0);
#pragma unroll 1
  for (int c0 = 128; c0 < w.vpad; c0 += 128) {
    __syncthreads();
    if (tid < 128) value_column(c0 + ch);
    __syncthreads();
    store_values(c0);
  }
  __syncthreads();
#pragma unroll
  for (int e = 0; e < 2; ++e) {   // a scale per token for each of P, G q and B
    const int tt = 2 * warp + e;
    float mp = 0.f, mq = 0.f, mb = lane <= tt ? fabsf(B[tt][min(lane, DC_T - 1)]) : 0.f;
#pragma unroll
    for (int m = 0; m < DP / 32; ++m) {
      mp = fmaxf(mp, fabsf(xs[tt][lane + 32 * m]));
      mq = fmaxf(mq, fabsf(qs[tt][lane + 32 * m]));
    }
    const int ep = split_exponent(warp_max(mp)), eq = split_exponent(warp_max(mq)), eb = split_exponent(warp_max(mb));
    if (lane == 0) {
      scale[0][tt] = split_scale(ep);
      scale[1][tt] = split_scale(eq);
      scale[2][tt] = split_scale(eb);
      float* unit = reinterpret_cast<float*>(blob + Blob::unit_at);
      unit[tt] = pow2i(ep - SPLIT_TOP);
      unit[DC_T + tt] = pow2i(eq - SPLIT_TOP);
      unit[2 * DC_T + tt] = pow2i(eb - SPLIT_TOP);
    }
  }
  __syncthreads();
  uint4* out = reinterpret_cast<uint4*>(blob);
#pragma unroll
  for (int u = 0; u < DP / 64 + (DP < 64); ++u) {
    const int e = tid + 256 * u;
    if (e < 4 * DP) {   // P and G q: 16 channels (k) x 8 tokens (n) per 32 entries
      const int t = 8 * ((e >> 5) & 1) + l4, i = 16 * (e >> 6) + tq;
      uint4 x;
      const float sp = scale[0][t], sq = scale[1][t];
      const float2 p0 = *reinterpret_cast<const float2*>(&xs[t][i]), p1 = *reinterpret_cast<const float2*>(&xs[t][i + 8]);
      split2(p0.x * sp, p0.y * sp, x.x, x.z);
      split2(p1.x * sp, p1.y * sp, x.y, x.w);
      out[e] = x;
      const float2 q0 = *reinterpret_cast<const float2*>(&qs[t][i]), q1 = *reinterpret_cast<const float2*>(&qs[t][i + 8]);
      split2(q0.x * sq, q0.y * sq, x.x, x.z);
      split2(q1.x * sq, q1.y * sq, x.y, x.w);
      out[Blob::q_at / 16 + e] = x;
      const int j = 8 * (e >> 5) + l4;   // G_15 / G_s k_s: 16 tokens (k) x 8 channels (n)
      constexpr float one = 1 << DC_KTOP;
      split2(gs[tq][j] * one, gs[tq + 1][j] * one, x.x, x.z);
      split2(gs[tq + 8][j] * one, gs[tq + 9][j] * one, x.y, x.w);
      out[Blob::k_at / 16 + e] = x;
    }
  }
  if (tid < 64) {   // B: tokens s (k) x tokens t (n)
    const int t = 8 * warp + l4;
    const float sb = scale[2][t];
    const auto b = [&](int c) { return c <= t ? B[t][c] * sb : 0.f; };
    uint4 x;
    split2(b(tq), b(tq + 1), x.x, x.z);
    split2(b(tq + 8), b(tq + 9), x.y, x.w);
    out[Blob::b_at / 16 + tid] = x;
  }
}

// The writes' share of the read-outs in FMAs, a token at a time: where a write is infinite or NaN, the product's zeros would carry it to the tokens before it, and
// where the writes of a column lie far apart, the larger ones' unit would cost the smaller ones, which earlier tokens read, their bits
constexpr float DC_APART = 0x1p-20f;   // the halves are off by at most 2^-49 of the column's largest write; 3 in 10000 chunks of normal numbers come here, and a
                                       // sequence's last chunk where it has fewer than 16 tokens (writes of zero beside others: the test has no instruction for them)
static __device__ __noinline__ void dc_read_serial(float (&o)[2][4], const float (&u)[2][4], const unsigned char* b, const float* unit, int lane) {
  const int tq = 2 * (lane & 3);
#pragma unroll
  for (int s = 0; s < DC_T; ++s) {
    const int src = (lane & ~3) | ((s & 7) >> 1);
    const float u0 = __shfl_sync(0xffffffffu, u[s >> 3][s & 1], src), u1 = __shfl_sync(0xffffffffu, u[s >> 3][2 + (s & 1)], src);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int t = 8 * (r >> 1) + tq + (r & 1);
      if (s > t) continue;
      const __half* e = reinterpret_cast<const __half*>(b + 16 * (32 * (t >> 3) + 4 * (t & 7) + ((s & 7) >> 1))) + 2 * (s >> 3) + (s & 1);
      const float x = fmaf(__half2float(e[4]), LO_UNIT, __half2float(e[0])) * unit[t];
      o[r >> 1][r & 1] = fmaf(x, u0, o[r >> 1][r & 1]);
      o[r >> 1][2 + (r & 1)] = fmaf(x, u1, o[r >> 1][2 + (r & 1)]);
    }
  }
}

// One chunk's writes as accumulators, from what the state gives (read-outs of P by `KW` warps, [warp][4][32 lanes] in `part`), and as A operand; m, w: each column's largest write, its unit
struct DcWrites {
  float u[2][4], m[2], w[2];
  unsigned hi[4], lo[4];
};
template <int KW>
__device__ __forceinline__ void dc_writes(DcWrites& x, const float4* part, const float4* wv, const float* unit, int lane) {
  const int tq = 2 * (lane & 3);
  x.m[0] = x.m[1] = 0.f;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    float4 z[KW];
#pragma unroll
    for (int k = 0; k < KW; ++k) z[k] = part[(4 * k + j) * 32 + lane];
#pragma unroll
    for (int k = 1; k < KW; k <<= 1)
#pragma unroll
      for (int i = 0; i + k < KW; i += 2 * k) {
        z[i].x += z[i + k].x; z[i].y += z[i + k].y; z[i].z += z[i + k].z; z[i].w += z[i + k].w;
      }
    const float4 y = wv[j];
    const float2 p = *reinterpret_cast<const float2*>(unit + 8 * j + tq);
    x.u[j][0] = fmaf(-z[0].x, p.x, y.x);
    x.u[j][1] = fmaf(-z[0].y, p.y, y.y);
    x.u[j][2] = fmaf(-z[0].z, p.x, y.z);
    x.u[j][3] = fmaf(-z[0].w, p.y, y.w);
    x.m[0] = fmaxf(x.m[0], fmaxf(fabsf(x.u[j][0]), fabsf(x.u[j][1])));
    x.m[1] = fmaxf(x.m[1], fmaxf(fabsf(x.u[j][2]), fabsf(x.u[j][3])));
  }
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    x.m[0] = fmaxf(x.m[0], __shfl_xor_sync(0xffffffffu, x.m[0], o));
    x.m[1] = fmaxf(x.m[1], __shfl_xor_sync(0xffffffffu, x.m[1], o));
  }
  const int f0 = split_exponent(x.m[0]), f1 = split_exponent(x.m[1]);
  const float t0 = split_scale(f0), t1 = split_scale(f1);
  x.w[0] = pow2i(f0 - SPLIT_TOP);
  x.w[1] = pow2i(f1 - SPLIT_TOP);
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    split2(x.u[j][0] * t0, x.u[j][1] * t0, x.hi[2 * j], x.lo[2 * j]);
    split2(x.u[j][2] * t1, x.u[j][3] * t1, x.hi[2 * j + 1], x.lo[2 * j + 1]);
  }
}

// A CTA has 16 value columns, KW warps with 32 channels of the state apiece and one warp for the read-outs. Every warp works out the writes for itself: less of a chain, more
// instructions, and a barrier per chunk
template <int DP>
__global__ void __launch_bounds__(32 * (DP / 32 + 1)) delta_scan_split_kernel(RecDev d, DeltaChunks w, PoisonRef poison) {
  pdl_trigger();
  pdl_wait();
  using Blob = DcBlob<DP>;
  constexpr int KW = DP / 32, STAGE = Blob::bytes + 1024;
  extern __shared__ __align__(128) unsigned char dc_smem[];
  __shared__ __align__(8) uint64_t full[DC_NS];
  __shared__ int issued[DC_NS];   // chunks sent for into a stage
  const int s = blockIdx.z, h = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l4 = lane >> 2, tq = 2 * (lane & 3);
  const int base = d.cu[s], n = d.cu[s + 1] - base;
  if (n <= 0) return;
  const int chunks = (n + DC_T - 1) / DC_T;
  const long long slot0 = chunk_slot0(base, s);
  const auto fetch = [&](int c, int b) {
    const long long at = (slot0 + c) * d.heads + h;
    unsigned char* st = dc_smem + b * STAGE;
    ++issued[b];
    mbar_arrive_expect_tx(&full[b], STAGE);
    bulk_load(st, w.blobs + at * Blob::bytes, Blob::bytes, &full[b]);
    bulk_load(st + Blob::bytes, w.wv + (at * (w.vpad / 16) + blockIdx.x) * 256, 1024, &full[b]);
  };
  const bool sender = threadIdx.x == 32 * KW;   // a lane of the read-out warp
  if (sender) {
    for (int b = 0; b < DC_NS; ++b) {
      mbar_init(&full[b], 1);
      issued[b] = 0;
    }
    fence_mbar_init();
    for (int b = 0; b < min(DC_NS, chunks); ++b) fetch(b, b);
  }
  float4* exchange = reinterpret_cast<float4*>(dc_smem + DC_NS * STAGE);   // [chunk parity][warp][P, P, G q, G q][lane]
  constexpr int TURN = KW * 128;
  const int col = 16 * blockIdx.x + l4;
  const bool ok0 = col < d.vdim, ok1 = col + 8 < d.vdim;
  bool alive = true;   // no wait of this thread has timed out
  // a stage is free once every warp has come to the barrier of the chunk after it
  const auto refill = [&](int c) {
    if (c > 0 && alive && c - 1 + DC_NS < chunks) {
      fence_proxy_async_smem();
      fetch(c - 1 + DC_NS, (c - 1) % DC_NS);
    }
  };
  if (warp < KW) {
    // S^T as accumulators: S[j][e] is column l4 + 8 (e / 2), channel 32 warp + 8 j + tq + e % 2
    float* sp = d.state + ((static_cast<long long>(d.slot[s]) * d.heads + h) * d.dim) * d.vdim + col;
    const bool carried = d.pos0[s] > 0;
    float S[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = 32 * warp + 8 * j + tq + (e & 1);
        S[j][e] = carried && i < d.dim && (e < 2 ? ok0 : ok1) ? sp[static_cast<long long>(i) * d.vdim + 8 * (e >> 1)] : 0.f;
      }
    __syncthreads();
    for (int c = 0; c < chunks; ++c) {
      const int b = c % DC_NS;
      const unsigned char* st = dc_smem + b * STAGE;
      float4* part = exchange + (c & 1) * TURN;
      float m0 = 0.f, m1 = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        m0 = fmaxf(m0, fmaxf(fabsf(S[j][0]), fabsf(S[j][1])));
        m1 = fmaxf(m1, fmaxf(fabsf(S[j][2]), fabsf(S[j][3])));
      }
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, o));
        m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
      }
      const int e0 = split_exponent(m0), e1 = split_exponent(m1);
      const float s0 = split_scale(e0), s1 = split_scale(e1), n0 = pow2i(e0 - SPLIT_TOP), n1 = pow2i(e1 - SPLIT_TOP);
      alive = mbar_wait_soft(&full[b], (c / DC_NS) & 1, poison) && alive;
      const uint4* ops = reinterpret_cast<const uint4*>(st) + lane;
      const float* unit = reinterpret_cast<const float*>(st + Blob::unit_at);
      float r[4][4], x[4][4];   // S^T P and S^T G q over this warp's channels: 8 tokens each
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) r[j][e] = x[j][e] = 0.f;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        unsigned ah[4], al[4];
        split2(S[2 * k][0] * s0, S[2 * k][1] * s0, ah[0], al[0]);
        split2(S[2 * k][2] * s1, S[2 * k][3] * s1, ah[1], al[1]);
        split2(S[2 * k + 1][0] * s0, S[2 * k + 1][1] * s0, ah[2], al[2]);
        split2(S[2 * k + 1][2] * s1, S[2 * k + 1][3] * s1, ah[3], al[3]);
        uint4 f[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) f[j] = ops[(j >= 2 ? Blob::q_at / 16 : 0) + 32 * (2 * (2 * warp + k) + (j & 1))];
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_f16(x[j], al, f[j].x, f[j].y);
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_f16(r[j], ah, f[j].x, f[j].y);
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_f16(x[j], ah, f[j].z, f[j].w);
      }
      constexpr float cut = 1.5f * SPLIT_CUT;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        part[(4 * warp + j) * 32 + lane] = make_float4(split_sum(r[j][0], x[j][0], cut) * n0, split_sum(r[j][1], x[j][1], cut) * n0,
                                                     split_sum(r[j][2], x[j][2], cut) * n1, split_sum(r[j][3], x[j][3], cut) * n1);
        const float2 q = *reinterpret_cast<const float2*>(unit + DC_T + 8 * j + tq);
        part[(4 * warp + 2 + j) * 32 + lane] = make_float4(split_sum(r[2 + j][0], x[2 + j][0], cut) * (n0 * q.x), split_sum(r[2 + j][1], x[2 + j][1], cut) * (n0 * q.y),
                                                         split_sum(r[2 + j][2], x[2 + j][2], cut) * (n1 * q.x), split_sum(r[2 + j][3], x[2 + j][3], cut) * (n1 * q.y));
      }
      __syncthreads();
      DcWrites u;
      dc_writes<KW>(u, part, reinterpret_cast<const float4*>(st + Blob::bytes + 32 * lane), unit, lane);
      // the state
      const float k0 = u.w[0] * (1.f / (1 << DC_KTOP)), k1 = u.w[1] * (1.f / (1 << DC_KTOP));
      const float* G = reinterpret_cast<const float*>(st + Blob::g_at) + 32 * warp + tq;
      float y[4][4], z[4][4];
      uint4 f[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) y[j][e] = z[j][e] = 0.f;
        f[j] = ops[Blob::k_at / 16 + 32 * (4 * warp + j)];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) mma_f16(z[j], u.lo, f[j].x, f[j].y);
#pragma unroll
      for (int j = 0; j < 4; ++j) mma_f16(y[j], u.hi, f[j].x, f[j].y);
#pragma unroll
      for (int j = 0; j < 4; ++j) mma_f16(z[j], u.hi, f[j].z, f[j].w);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 g = *reinterpret_cast<const float2*>(G + 8 * j);
#pragma unroll
        for (int e = 0; e < 4; ++e) S[j][e] = fmaf(S[j][e], e & 1 ? g.y : g.x, split_sum(y[j][e], z[j][e], SPLIT_CUT) * (e < 2 ? k0 : k1));
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = 32 * warp + 8 * j + tq + (e & 1);
        if (i < d.dim && (e < 2 ? ok0 : ok1)) sp[static_cast<long long>(i) * d.vdim + 8 * (e >> 1)] = S[j][e];
      }
  } else {
    __syncthreads();
    for (int c = 0; c < chunks; ++c) {
      const int b = c % DC_NS;
      const unsigned char* st = dc_smem + b * STAGE;
      const float4* part = exchange + (c & 1) * TURN;
      alive = mbar_wait_soft(&full[b], (c / DC_NS) & 1, poison) && alive;
      __syncthreads();
      if (sender) refill(c);
      const float* unit = reinterpret_cast<const float*>(st + Blob::unit_at);
      DcWrites u;
      dc_writes<KW>(u, part, reinterpret_cast<const float4*>(st + Blob::bytes + 32 * lane), unit, lane);
      float o[2][4];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        float4 x = part[(2 + j) * 32 + lane];
#pragma unroll
        for (int k = 1; k < KW; ++k) {
          const float4 y = part[(4 * k + 2 + j) * 32 + lane];
          x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
        }
        o[j][0] = x.x; o[j][1] = x.y; o[j][2] = x.z; o[j][3] = x.w;
      }
      const float a0 = DC_APART * u.m[0], a1 = DC_APART * u.m[1];
      bool together = u.m[0] < INFINITY && u.m[1] < INFINITY;
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) together = together && fabsf(u.u[j][e]) >= (e < 2 ? a0 : a1);   // false for NaN
      if (__all_sync(0xffffffffu, together)) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float y[4] = {0.f, 0.f, 0.f, 0.f}, z[4] = {0.f, 0.f, 0.f, 0.f};
          const uint4 f = (reinterpret_cast<const uint4*>(st) + lane)[Blob::b_at / 16 + 32 * j];
          const float2 p = *reinterpret_cast<const float2*>(unit + 2 * DC_T + 8 * j + tq);
          mma_f16(z, u.lo, f.x, f.y);
          mma_f16(y, u.hi, f.x, f.y);
          mma_f16(z, u.hi, f.z, f.w);
#pragma unroll
          for (int e = 0; e < 4; ++e) o[j][e] = fmaf(split_sum(y[e], z[e], SPLIT_CUT) * u.w[e >> 1], e & 1 ? p.y : p.x, o[j][e]);
        }
      } else {
        dc_read_serial(o, u.u, st + Blob::b_at, unit + 2 * DC_T, lane);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = DC_T * c + 8 * j + tq + (e & 1);
          if (t < n && (e < 2 ? ok0 : ok1))
            st_from_float(d.out, d.out_dt, static_cast<long long>(base + t) * d.ld_out + static_cast<long long>(h) * d.vdim + col + 8 * (e >> 1), o[j][e]);
        }
    }
  }
  if (__syncthreads_or(!alive)) mbar_drain(full, issued, DC_NS);
}

template <int DP>
__global__ void __launch_bounds__(32 * DC_NW) delta_scan_kernel(RecDev d, DeltaChunks w, PoisonRef poison) {
  pdl_trigger();
  pdl_wait();
  using Blob = DcBlob<DP>;
  constexpr int KS = DP / 16, NT = DP / 8, STAGE = Blob::bytes + DC_NW * 1024;
  extern __shared__ __align__(128) unsigned char dc_smem[];
  __shared__ __align__(8) uint64_t full[DC_NS];
  __shared__ int done[DC_NS], issued[DC_NS];   // warps that are through with a stage, counted up for ever; chunks sent for into it
  const int s = blockIdx.z, h = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l4 = lane >> 2, tq = 2 * (lane & 3);
  const int base = d.cu[s], n = d.cu[s + 1] - base;
  if (n <= 0) return;
  const int chunks = (n + DC_T - 1) / DC_T;
  const long long slot0 = chunk_slot0(base, s);
  const auto fetch = [&](int c, int b) {
    const long long at = (slot0 + c) * d.heads + h;
    unsigned char* st = dc_smem + b * STAGE;
    ++issued[b];
    mbar_arrive_expect_tx(&full[b], STAGE);
    bulk_load(st, w.blobs + at * Blob::bytes, Blob::bytes, &full[b]);
    bulk_load(st + Blob::bytes, w.wv + (at * (w.vpad / 16) + blockIdx.x * DC_NW) * 256, DC_NW * 1024, &full[b]);
  };
  if (threadIdx.x == 0) {
    for (int b = 0; b < DC_NS; ++b) {
      mbar_init(&full[b], 1);
      done[b] = issued[b] = 0;
    }
    fence_mbar_init();
    for (int b = 0; b < min(DC_NS, chunks); ++b) fetch(b, b);
  }
  // S^T as accumulators: S[j][e] is column l4 + 8 (e / 2), channel 8 j + tq + e % 2
  const int col = 32 * blockIdx.x + 16 * warp + l4;
  const bool ok0 = col < d.vdim, ok1 = col + 8 < d.vdim;
  float* sp = d.state + ((static_cast<long long>(d.slot[s]) * d.heads + h) * d.dim) * d.vdim + col;
  const bool carried = d.pos0[s] > 0;
  float S[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = 8 * j + tq + (e & 1);
      S[j][e] = carried && i < d.dim && (e < 2 ? ok0 : ok1) ? sp[static_cast<long long>(i) * d.vdim + 8 * (e >> 1)] : 0.f;
    }
  __syncthreads();
  bool alive = true;   // no wait of this thread has timed out; lane 0 sends for chunks
  for (int c = 0; c < chunks; ++c) {
    const int b = c % DC_NS;
    const unsigned char* st = dc_smem + b * STAGE;
    float m0 = 0.f, m1 = 0.f;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      m0 = fmaxf(m0, fmaxf(fabsf(S[j][0]), fabsf(S[j][1])));
      m1 = fmaxf(m1, fmaxf(fabsf(S[j][2]), fabsf(S[j][3])));
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, o));
      m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
    }
    const int e0 = split_exponent(m0), e1 = split_exponent(m1);
    const float s0 = split_scale(e0), s1 = split_scale(e1), n0 = pow2i(e0 - SPLIT_TOP), n1 = pow2i(e1 - SPLIT_TOP);
    alive = mbar_wait_soft(&full[b], (c / DC_NS) & 1, poison) && alive;
    const uint4* ops = reinterpret_cast<const uint4*>(st) + lane;
    float r[4][4], x[4][4], half[4][4];   // S^T P and S^T G q: 8 tokens each
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) r[j][e] = x[j][e] = half[j][e] = 0.f;
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      unsigned ah[4], al[4];
      split2(S[2 * k][0] * s0, S[2 * k][1] * s0, ah[0], al[0]);
      split2(S[2 * k][2] * s1, S[2 * k][3] * s1, ah[1], al[1]);
      split2(S[2 * k + 1][0] * s0, S[2 * k + 1][1] * s0, ah[2], al[2]);
      split2(S[2 * k + 1][2] * s1, S[2 * k + 1][3] * s1, ah[3], al[3]);
      uint4 f[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) f[j] = ops[(j >= 2 ? Blob::q_at / 16 : 0) + 32 * (2 * k + (j & 1))];
#pragma unroll
      for (int j = 0; j < 4; ++j) mma_f16(x[j], al, f[j].x, f[j].y);
#pragma unroll
      for (int j = 0; j < 4; ++j) mma_f16(r[j], ah, f[j].x, f[j].y);
#pragma unroll
      for (int j = 0; j < 4; ++j) mma_f16(x[j], ah, f[j].z, f[j].w);
      if (KS >= 4 && k == KS / 2 - 1) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            half[j][e] = r[j][e];
            r[j][e] = 0.f;
          }
      }
    }
    // the writes, then as A operand
    constexpr float cut = ((KS >= 4 ? KS / 2 : KS) + 1) * 0.5f * SPLIT_CUT;
    const float* unit = reinterpret_cast<const float*>(st + Blob::unit_at);
    const float4* wv = reinterpret_cast<const float4*>(st + Blob::bytes + 1024 * warp + 32 * lane);
    float u[2][4];
    m0 = m1 = 0.f;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float4 y = wv[j];
      const float2 p = *reinterpret_cast<const float2*>(unit + 8 * j + tq);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float y0 = r[j][e] + half[j][e], z = split_sum(y0, x[j][e], cut) * (e < 2 ? n0 : n1);
        u[j][e] = fmaf(-z, e & 1 ? p.y : p.x, e == 0 ? y.x : e == 1 ? y.y : e == 2 ? y.z : y.w);
      }
      m0 = fmaxf(m0, fmaxf(fabsf(u[j][0]), fabsf(u[j][1])));
      m1 = fmaxf(m1, fmaxf(fabsf(u[j][2]), fabsf(u[j][3])));
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, o));
      m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
    }
    const int f0 = split_exponent(m0), f1 = split_exponent(m1);
    const float t0 = split_scale(f0), t1 = split_scale(f1), w0 = pow2i(f0 - SPLIT_TOP), w1 = pow2i(f1 - SPLIT_TOP);
    unsigned uh[4], ul[4];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      split2(u[j][0] * t0, u[j][1] * t0, uh[2 * j], ul[2 * j]);
      split2(u[j][2] * t1, u[j][3] * t1, uh[2 * j + 1], ul[2 * j + 1]);
    }
    // the state
    const float k0 = w0 * (1.f / (1 << DC_KTOP)), k1 = w1 * (1.f / (1 << DC_KTOP));
    const float* G = reinterpret_cast<const float*>(st + Blob::g_at) + tq;
#pragma unroll
    for (int j = 0; j < NT; j += 2) {
      float y[2][4], z[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) y[i][e] = z[i][e] = 0.f;
      const uint4 f[2] = {ops[Blob::k_at / 16 + 32 * j], ops[Blob::k_at / 16 + 32 * j + 32]};
#pragma unroll
      for (int i = 0; i < 2; ++i) mma_f16(z[i], ul, f[i].x, f[i].y);
#pragma unroll
      for (int i = 0; i < 2; ++i) mma_f16(y[i], uh, f[i].x, f[i].y);
#pragma unroll
      for (int i = 0; i < 2; ++i) mma_f16(z[i], uh, f[i].z, f[i].w);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float2 g = *reinterpret_cast<const float2*>(G + 8 * (j + i));
#pragma unroll
        for (int e = 0; e < 4; ++e) S[j + i][e] = fmaf(S[j + i][e], e & 1 ? g.y : g.x, split_sum(y[i][e], z[i][e], SPLIT_CUT) * (e < 2 ? k0 : k1));
      }
    }
    // the read-outs
    float o[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float2 q = *reinterpret_cast<const float2*>(unit + DC_T + 8 * j + tq);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float y0 = r[2 + j][e] + half[2 + j][e];
        o[j][e] = split_sum(y0, x[2 + j][e], cut) * ((e < 2 ? n0 : n1) * (e & 1 ? q.y : q.x));
      }
    }
    const float a0 = DC_APART * m0, a1 = DC_APART * m1;
    bool together = m0 < INFINITY && m1 < INFINITY;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) together = together && fabsf(u[j][e]) >= (e < 2 ? a0 : a1);   // false for NaN
    if (__all_sync(0xffffffffu, together)) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        float y[4] = {0.f, 0.f, 0.f, 0.f}, z[4] = {0.f, 0.f, 0.f, 0.f};
        const uint4 f = ops[Blob::b_at / 16 + 32 * j];
        const float2 p = *reinterpret_cast<const float2*>(unit + 2 * DC_T + 8 * j + tq);
        mma_f16(z, ul, f.x, f.y);
        mma_f16(y, uh, f.x, f.y);
        mma_f16(z, uh, f.z, f.w);
#pragma unroll
        for (int e = 0; e < 4; ++e) o[j][e] = fmaf(split_sum(y[e], z[e], SPLIT_CUT) * (e < 2 ? w0 : w1), e & 1 ? p.y : p.x, o[j][e]);
      }
    } else {
      dc_read_serial(o, u, st + Blob::b_at, unit + 2 * DC_T, lane);
    }
    // through with the stage: the last warp refills it
    __syncwarp();
    if (lane == 0 && alive && c + DC_NS < chunks) {
      __threadfence_block();
      if (atomicAdd(&done[b], 1) % DC_NW == DC_NW - 1) {
        __threadfence_block();
        fence_proxy_async_smem();
        fetch(c + DC_NS, b);
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = DC_T * c + 8 * j + tq + (e & 1);
        if (t < n && (e < 2 ? ok0 : ok1))
          st_from_float(d.out, d.out_dt, static_cast<long long>(base + t) * d.ld_out + static_cast<long long>(h) * d.vdim + col + 8 * (e >> 1), o[j][e]);
      }
  }
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = 8 * j + tq + (e & 1);
      if (i < d.dim && (e < 2 ? ok0 : ok1)) sp[static_cast<long long>(i) * d.vdim + 8 * (e >> 1)] = S[j][e];
    }
  if (__syncthreads_or(!alive)) mbar_drain(full, issued, DC_NS);
}

int blob_bytes(int dim) { return dim <= 32 ? DcBlob<32>::bytes : dim <= 64 ? DcBlob<64>::bytes : DcBlob<128>::bytes; }
int round32(int x) { return (x + 31) / 32 * 32; }

template <int DP>
cudaError_t launch(const RecDev& d, int n_seqs, int max_new, const DeltaChunks& w, cudaStream_t st) {
  constexpr int split_smem = DC_NS * (DcBlob<DP>::bytes + 1024) + 2 * (DP / 32) * 2048, smem = DC_NS * (DcBlob<DP>::bytes + DC_NW * 1024);
  // While all CTAs run at once, two per SM, the split walk's shorter chain counts; where they queue up, its instructions. All channels per warp / split, us, heads of 128 x 128:
  // 8 over 4 x 2048 tokens (256 CTAs) 236 / 180, over one of 500 63 / 40; 16 over one of 2000 231 / 142; 8 over 8 x 1024 (512 CTAs) 125 / 182; 16 over 8 x 1000 243 / 340;
  // 4 of 64 x 64 over 4 x 300 30 / 22, over 32 x 300 (512 CTAs) 32 / 35
  const bool split = static_cast<long long>(n_seqs) * d.heads * (w.vpad / 16) <= 2 * num_sms();
  static std::atomic<unsigned long long> allowed_split{0}, allowed{0};
  cudaError_t e = split ? allow_smem(delta_scan_split_kernel<DP>, allowed_split) : allow_smem(delta_scan_kernel<DP>, allowed);
  if (e != cudaSuccess) return e;
  PoisonRef poison = {};
  if (!poison_ref(&poison)) return cudaErrorMemoryAllocation;
  const auto quads = [](const void* p, long long ld) { return reinterpret_cast<uintptr_t>(p) % 16 == 0 && ld % 4 == 0; };
  const bool vec = d.in_dt == VY_F32 && d.a_dt == VY_F32 && d.dim % 4 == 0 && quads(d.q, d.ldq) && quads(d.k, d.ldk) && quads(d.a, d.ld_a);
  e = launch_kernel(delta_chunk_kernel<DP>, dim3((max_new + DC_T - 1) / DC_T, d.heads, n_seqs), dim3(256), 0, st, d, w, vec);
  if (e != cudaSuccess) return e;
  count_launch();
  if (split) return launch_kernel(delta_scan_split_kernel<DP>, dim3(w.vpad / 16, d.heads, n_seqs), dim3(32 * (DP / 32 + 1)), split_smem, st, d, w, poison);
  return launch_kernel(delta_scan_kernel<DP>, dim3(w.vpad / 32, d.heads, n_seqs), dim3(32 * DC_NW), smem, st, d, w, poison);
}

}  // namespace

// From 32 tokens on (64 for heads of up to 32 channels): two launches and a chunk's preparation cost more than a short walk. In us, chunks / tokens:
// 1 sequence, 8 heads of 128 x 128: 20.3 / 19.9 at 24 tokens, 20.5 / 23.2 at 32, 30 / 71 at 128; 32 sequences, 4 heads of 64 x 64: 19.2 / 18.4,
// 19.3 / 22.0, 44 / 72; 4 sequences, 4 heads of 16 x 16: 16.2 / 15.4 at 48, 17.3 / 18.6 at 64. Where a long portion stands beside many short ones the walk is
// through with those at once, but here each of their CTAs fills its buffers: 8 heads of 128 x 128, 31 single tokens and one portion of 32, 64, 100: 46 / 27, 47 / 43,
// 48 / 62; 63 single tokens and 70, 200: 71 / 51, 83 / 115; 4 heads of 64 x 64, 31 and 48: 21 / 24. So 20 tokens per round of CTAs (two per SM).
// Past 128 channels a warp's share of the state (16 columns) does not fit its registers.
long long delta_rule_mma_floats(long long rows, int n_seqs, int max_new, int heads, int dim, int vdim) {
  if (max_new < (dim > 32 ? 32 : 64) || dim > 128 || rows <= 0) return 0;
  const long long ctas = static_cast<long long>(n_seqs) * heads * (round32(vdim) / 32);
  if (4 * rows < static_cast<long long>(n_seqs) * max_new && max_new < 20 * ctas / (2 * num_sms())) return 0;
  const long long f = (rows / DC_T + n_seqs) * heads * (blob_bytes(dim) / 4 + 16LL * round32(vdim));
  return f <= (1LL << 28) ? f : 0;
}

cudaError_t launch_delta_rule_mma(const RecDev& d, int n_seqs, int max_new, long long rows, float* ws, cudaStream_t st) {
  DeltaChunks w;
  w.blobs = reinterpret_cast<unsigned char*>(ws);
  w.wv = ws + (rows / DC_T + n_seqs) * d.heads * (blob_bytes(d.dim) / 4);
  w.vpad = round32(d.vdim);
  if (d.dim <= 32) return launch<32>(d, n_seqs, max_new, w, st);
  if (d.dim <= 64) return launch<64>(d, n_seqs, max_new, w, st);
  return launch<128>(d, n_seqs, max_new, w, st);
}

}  // namespace vy
