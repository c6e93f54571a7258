// Prompt-sized form of the attention whose heads exchange scores (vy_talk_attn; see talking_attn.cu), in fp32 precision on the tensor cores
// (split_mma.cuh), for 8, 16 or 32 heads of at most 64 channels.
//
// One CTA owns all H heads of TQ = 256 / H queries: 256 (head, query) rows, 16 per warp, on 16 warps. Keys go by in tiles of N. Per tile a
// warp computes its rows' scores, the CTA lays them out as a [head][query, key] matrix in shared memory, multiplies that by `talk` (another
// split product: M = K = heads, columns = pairs), and every warp takes its own rows of the result back into registers for the softmax and the
// weighted values. Key and value rows come split from the workspace that window_attn_mma.cu's first launch fills (cp.async: the next tile's keys
// arrive during the exchange, its values during the scores).
//
// What bounds it: per tile and SM about as many cycles of the tensor pipe as of softmax instructions, and three barriers. The fp32-FMA tiles
// (talk_attn_tiled_kernel, which stays for other head counts and sizes) spend 62 % of their issue slots on operand reads and the exchange.
// 2 x 1437 tokens, 16 heads of 64: 805 us by those, 325 us here, 5 for the splitting. Up to four key / value heads and few or long enough prompts go to talk_attn_tc_kernel, which takes
// 150 there (talk_attn_tc_applies says which); the others stay here.
#include "seqmix.cuh"
#include "split_mma.cuh"
#include "talk_attn.cuh"

namespace vy {

constexpr int TM_T = 512, TM_W = 16, TM_R = 256;
// As SPLIT_SCORE (seqmix.cuh), for scores that are mixed: |q k scale| per channel, and an exchange weight times the largest score. A tile's scores share one scale,
// so a mixed score is off by 2^-48 of TM_MIXED per head at most
constexpr float TM_SCORE = 0x1p14f, TM_MIXED = 0x1p20f;

// sizes in bytes or elements that the kernel and its launcher share
template <int HL, int N>
struct TalkMma {
  static constexpr int H = 1 << HL, TQ = TM_R >> HL;
  static constexpr int PQ = N + 8;                               // fp16 pairs of a query in a score plane's row: stores of 8 queries fall into distinct banks
  static constexpr int PB = TQ * PQ * 2 + 16;                    // bytes of a head's row in a score plane: an odd multiple of 16
  static constexpr int XQ = N + 4;                               // floats of a query in a head's row of exchanged scores
  static constexpr int XH = (TQ * XQ + 31) / 32 * 32 + 8;
  static constexpr int MT = H < 16 ? 1 : H / 16;                 // 16-head blocks of the exchange
  static constexpr int TB = MT * 32 + 16;                        // bytes of a row of `talk`
};

template <int HL, int N>
__global__ void __launch_bounds__(TM_T, 1) talk_attn_mma_kernel(TalkDev d, SplitKv w, int dim16, int vdim16, bool qvec, bool ovec) {
  pdl_trigger();
  pdl_wait();
  using C = TalkMma<HL, N>;
  constexpr int H = C::H, TQ = C::TQ, NT = N / 8, KT = N / 16, MT = C::MT;
  extern __shared__ __align__(16) unsigned char tm_smem[];
  const int G = d.kv_heads, per = H / G, kb = dim16 * 2 + 16, vb = vdim16 * 2 + 16, q_lo = TM_R * kb, k_lo = G * N * kb, v_lo = G * N * vb;
  unsigned char* Qh = tm_smem;
  unsigned char* Kh = Qh + 2 * q_lo;
  unsigned char* Vh = Kh + 2 * k_lo;
  unsigned char* Sh = Vh + 2 * v_lo;             // raw scores, [H][TQ][PQ] hi and lo
  unsigned char* Th = Sh + 2 * H * C::PB;        // talk, [16 MT][16 MT] hi and lo
  unsigned char* zero = Th + 2 * 16 * MT * C::TB;   // 16 bytes of zeros: the head rows a block of 16 lacks
  float* X = reinterpret_cast<float*>(zero + 16);   // exchanged scores, [H][XH]
  float* qu = X + H * C::XH;                     // powers of two that undo the scaling: query rows, talk rows, key and value rows [G][N]
  float* tu = qu + TM_R;
  float* ku = tu + 16 * MT;
  float* vu = ku + G * N;
  unsigned* top_s = reinterpret_cast<unsigned*>(vu + G * N);
  const int s = blockIdx.y, t = threadIdx.x, warp = t >> 5, lane = t & 31, gq = lane >> 2, tq = lane & 3;
  const int base = d.cu[s], n = d.cu[s + 1] - base;
  const int blk = (n + TQ - 1) / TQ - 1 - static_cast<int>(blockIdx.x);   // the last queries see the most keys: they go first
  if (blk < 0) return;
  const int i0 = blk * TQ, nq = min(TQ, n - i0);
  const int p0 = d.pos0[s], p_lo = p0 + i0, p_hi = p_lo + nq - 1;
  const int lo = d.window > 0 ? max(p_lo - d.window + 1, 0) : 0, lo0 = d.window > 0 ? max(p0 - d.window + 1, 0) : 0;
  const int count = p_hi - lo + 1;
  // one tile's K (part 0) or V (part 1) rows of every key / value head; past the end: zeros
  const auto fetch = [&](int c0, int part) {
    const int w16 = (part ? vdim16 : dim16) >> 3, each = 2 * w16, rb = part ? vb : kb, pl = part ? v_lo : k_lo;
    const unsigned dst = smem_addr(part ? Vh : Kh);
    float* un = part ? vu : ku;
    for (int x = t; x < G * N; x += TM_T) {
      const int g = x / N, j = x & (N - 1);
      const long long at = (static_cast<long long>(s) * G + g) * w.cap + (lo - lo0) + min(c0 + j, count - 1);
      un[x] = c0 + j < count ? reinterpret_cast<const float*>(w.rows + at * w.row_bytes + 4 * (dim16 + vdim16))[part] : pow2i(SPLIT_MIN_E);
    }
    for (int x = t; x < G * N * each; x += TM_T) {
      const int r = x / each, c = x - r * each, g = r / N, j = r & (N - 1);
      const long long at = (static_cast<long long>(s) * G + g) * w.cap + (lo - lo0) + min(c0 + j, count - 1);
      cp_async16(dst + (c < w16 ? r * rb + 16 * c : pl + r * rb + 16 * (c - w16)), w.rows + at * w.row_bytes + (part ? 4 * dim16 : 0) + 16 * c, c0 + j < count);
    }
    cp_async_commit();
  };
  fetch(0, 0);
  split_rows<TM_W, 64>(Qh, Qh + q_lo, kb, qu, SPLIT_TOP, TM_R, d.dim, dim16, d.q, d.q_dt, qvec, [&](int r) {
    const int h = r / TQ, i = r & (TQ - 1);
    return i < nq ? static_cast<long long>(base + i0 + i) * d.ldq + static_cast<long long>(h) * d.dim : -1LL;
  });
  // talk: two lanes' worth of loads per row would not pay: a thread scales and splits a row
  bool odd = false;   // numbers that are not for fp16 halves (seqmix.cuh): the fp32 tiles' sequence
  if (t < 16 * MT) {
    float x[16 * MT], m = 0.f;
#pragma unroll
    for (int b = 0; b < 16 * MT; ++b) {
      x[b] = t < H && b < H ? (d.talk ? ld_as_float(d.talk, d.talk_dt, t * H + b) : (t == b ? 1.f : 0.f)) : 0.f;
      m = fmaxf(m, fabsf(x[b]));
    }
    const int e = split_exponent(m);
    tu[t] = pow2i(e - SPLIT_TOP);
    odd = !(m * (d.softcap > 0.f ? fminf(d.softcap, TM_SCORE) : TM_SCORE) <= TM_MIXED);
#pragma unroll
    for (int b = 0; b < 16 * MT; b += 2) {
      unsigned h, l;
      split2(x[b] * split_scale(e), x[b + 1] * split_scale(e), h, l);
      *reinterpret_cast<unsigned*>(Th + t * C::TB + 2 * b) = h;
      *reinterpret_cast<unsigned*>(Th + (16 * MT + t) * C::TB + 2 * b) = l;
    }
  }
  if (t < 4) reinterpret_cast<unsigned*>(zero)[t] = 0u;
  const int rw = 16 * warp, hw = rw / TQ, g = hw / per;   // this warp's rows; they all read key / value head g
  float top_k;
  odd = split_odd(w, s * G + g, p0 + n - lo0, top_k) || odd;
  __syncthreads();   // qu
#pragma unroll
  for (int e = 0; e < 2; ++e) odd = odd || !(fabsf(qu[rw + gq + 8 * e] * d.scale) * top_k <= TM_SCORE * 0x1p-13f);
  if (__syncthreads_or(odd)) {
    cp_async_wait<0>();
    if (t == 0) w.odd[s * G] = 1;
    return;
  }
  const float two_over_cap = d.softcap > 0.f ? 2.f / d.softcap : 0.f;
  float m[2], l[2];
  int pos[2], hr[2], qr[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int r = rw + gq + 8 * e;
    hr[e] = r / TQ;
    qr[e] = r & (TQ - 1);
    pos[e] = p_lo + qr[e];
    float sk;
    const bool has = sink_of(d, hr[e], sk);
    m[e] = has ? sk : -INFINITY;
    l[e] = has && tq == 0 ? 1.f : 0.f;
  }
  float o[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[i][e] = 0.f;
  int E = SPLIT_MIN_E;
  const unsigned qa = smem_addr(Qh) + rw * kb + lane_a(lane, kb), ka = smem_addr(Kh) + g * N * kb + lane_b(lane, kb);
  const unsigned va = smem_addr(Vh) + g * N * vb + lane_bt(lane, vb), ta = smem_addr(Th) + lane_a(lane, C::TB);
  for (int c0 = 0; c0 < count; c0 += N) {
    cp_async_wait<0>();
    if (t == 0) *top_s = 0u;
    __syncthreads();   // this tile's keys are here; the previous tile's values and exchanged scores have been read
    fetch(c0, 1);
    // ---- raw scores ----
    float sc[NT][4], x[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) sc[i][e] = x[i][e] = 0.f;
    for (int k = 0; k < dim16; k += 16) {
      unsigned ah[4], al[4];
      ldsm_x4(ah, qa + 2 * k);
      ldsm_x4(al, qa + q_lo + 2 * k);
#pragma unroll
      for (int j = 0; j < NT / 2; ++j) {
        unsigned bh[4], bl[4];
        ldsm_x4(bh, ka + 16 * j * kb + 2 * k);
        ldsm_x4(bl, ka + k_lo + 16 * j * kb + 2 * k);
        mma_f16(x[2 * j], al, bh[0], bh[1]);
        mma_f16(x[2 * j + 1], al, bh[2], bh[3]);
        mma_f16(sc[2 * j], ah, bh[0], bh[1]);
        mma_f16(sc[2 * j + 1], ah, bh[2], bh[3]);
        mma_f16(x[2 * j], ah, bl[0], bl[1]);
        mma_f16(x[2 * j + 1], ah, bl[2], bl[3]);
      }
    }
    float largest = 0.f;
    const float qm[2] = {qu[rw + gq] * d.scale, qu[rw + gq + 8] * d.scale};
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const float2 k2 = *reinterpret_cast<const float2*>(ku + g * N + 8 * i + 2 * tq);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        sc[i][e] = cap_score(fmaf(x[i][e], LO_UNIT, sc[i][e]) * (e & 1 ? k2.y : k2.x) * qm[e >> 1], d.softcap, two_over_cap);
        largest = fmaxf(largest, fabsf(sc[i][e]));
      }
    }
    int es;   // one power of two for the tile's scores: the cap bounds them, without one their largest is found
    if (d.softcap > 0.f) es = split_exponent(d.softcap);
    else {
      const unsigned b = __reduce_max_sync(0xffffffffu, __float_as_uint(largest));
      if (lane == 0) atomicMax(top_s, b);
      __syncthreads();
      es = split_exponent(__uint_as_float(*top_s));
    }
    {
      const float f = split_scale(es);
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          unsigned hi, lo2;
          split2(sc[i][2 * r] * f, sc[i][2 * r + 1] * f, hi, lo2);
          unsigned char* at = Sh + hr[r] * C::PB + (qr[r] * C::PQ + 8 * i + 2 * tq) * 2;
          *reinterpret_cast<unsigned*>(at) = hi;
          *reinterpret_cast<unsigned*>(at + H * C::PB) = lo2;
        }
    }
    __syncthreads();   // the scores are laid out; the keys have been read
    if (c0 + N < count) fetch(c0 + N, 0);
    else cp_async_commit();
    // ---- exchange: 16 pairs (one query, 16 keys) at a time ----
    const float su = pow2i(es - SPLIT_TOP);
    for (int u = warp; u < TQ * (N / 16); u += TM_W) {
      const int q = u / (N / 16), j = u % (N / 16);
      const int krow = (lane & 7) + (((lane >> 3) & 1) << 3), col = (q * C::PQ + 16 * j) * 2 + ((lane >> 4) << 4);
      float y[MT][2][4], z[MT][2][4];
#pragma unroll
      for (int a = 0; a < MT; ++a)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) y[a][i][e] = z[a][i][e] = 0.f;
#pragma unroll
      for (int k = 0; k < MT; ++k) {
        unsigned bh[4], bl[4];
        const int row = 16 * k + krow;
        const unsigned at = row < H ? smem_addr(Sh) + row * C::PB + col : smem_addr(zero);
        ldsm_x4_t(bh, at);
        ldsm_x4_t(bl, row < H ? at + H * C::PB : at);
#pragma unroll
        for (int a = 0; a < MT; ++a) {
          unsigned ah[4], al[4];
          ldsm_x4(ah, ta + 16 * a * C::TB + 32 * k);
          ldsm_x4(al, ta + 16 * (MT + a) * C::TB + 32 * k);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            mma_f16(z[a][i], al, bh[2 * i], bh[2 * i + 1]);
            mma_f16(y[a][i], ah, bh[2 * i], bh[2 * i + 1]);
            mma_f16(z[a][i], ah, bl[2 * i], bl[2 * i + 1]);
          }
        }
      }
#pragma unroll
      for (int a = 0; a < MT; ++a)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int h = 16 * a + gq + 8 * r;
          if (h < H) {
            const float f = tu[h] * su;
#pragma unroll
            for (int i = 0; i < 2; ++i)
              *reinterpret_cast<float2*>(X + h * C::XH + q * C::XQ + 16 * j + 8 * i + 2 * tq) =
                  make_float2(fmaf(z[a][i][2 * r], LO_UNIT, y[a][i][2 * r]) * f, fmaf(z[a][i][2 * r + 1], LO_UNIT, y[a][i][2 * r + 1]) * f);
          }
        }
    }
    cp_async_wait<1>();
    __syncthreads();   // the exchanged scores and this tile's values are here
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float2 v = *reinterpret_cast<const float2*>(X + hr[r] * C::XH + qr[r] * C::XQ + 8 * i + 2 * tq);
        sc[i][2 * r] = v.x;
        sc[i][2 * r + 1] = v.y;
      }
    const int f0 = lo + c0, f1 = f0 + N - 1;
    if (!(c0 + N <= count && f1 <= p_lo && (d.window <= 0 || p_hi - f0 < d.window))) {
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int c = c0 + 8 * i + 2 * tq + (e & 1), kp = lo + c, p = pos[e >> 1];
          if (!(c < count && kp <= p && (d.window <= 0 || p - kp < d.window))) sc[i][e] = -INFINITY;
        }
    }
    // ---- softmax and values, as in window_attn_mma_kernel ----
    const unsigned ev = __float_as_uint(vu[g * N + (lane & (N - 1))]);
    const int e_new = max(E, static_cast<int>(__reduce_max_sync(0xffffffffu, ev) >> 23) - 127);
    float keep_o[2] = {pow2i(E - e_new), pow2i(E - e_new)};
    E = e_new;
    const float v_unit = pow2i(SPLIT_TOP - E);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float top = -INFINITY;
#pragma unroll
      for (int i = 0; i < NT; ++i) top = fmaxf(top, fmaxf(sc[i][2 * r], sc[i][2 * r + 1]));
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
      const float mn = fmaxf(m[r], top);
      const float cr = mn == -INFINITY ? 1.f : expf(m[r] - mn);
      m[r] = mn;
      l[r] *= cr;
      keep_o[r] *= cr;
    }
    const float mm[2] = {m[0] == -INFINITY ? 0.f : m[0], m[1] == -INFINITY ? 0.f : m[1]};
    unsigned ph[KT][4], pl[KT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const float2 v2 = *reinterpret_cast<const float2*>(vu + g * N + 8 * i + 2 * tq);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        sc[i][e] = expf(sc[i][e] - mm[e >> 1]);
        l[e >> 1] += sc[i][e];
        sc[i][e] *= (e & 1 ? v2.y : v2.x) * v_unit;
      }
      split2(sc[i][0], sc[i][1], ph[i >> 1][(i & 1) * 2], pl[i >> 1][(i & 1) * 2]);
      split2(sc[i][2], sc[i][3], ph[i >> 1][(i & 1) * 2 + 1], pl[i >> 1][(i & 1) * 2 + 1]);
    }
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
      if (16 * cc >= vdim16) break;
      float y[2][4], z[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) y[i][e] = z[i][e] = 0.f;
#pragma unroll
      for (int k = 0; k < KT; ++k) {
        unsigned bh[4], bl[4];
        ldsm_x4_t(bh, va + 16 * k * vb + 32 * cc);
        ldsm_x4_t(bl, va + v_lo + 16 * k * vb + 32 * cc);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          mma_f16(z[i], pl[k], bh[2 * i], bh[2 * i + 1]);
          mma_f16(y[i], ph[k], bh[2 * i], bh[2 * i + 1]);
          mma_f16(z[i], ph[k], bl[2 * i], bl[2 * i + 1]);
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[2 * cc + i][e] = fmaf(o[2 * cc + i][e], keep_o[e >> 1], fmaf(z[i][e], LO_UNIT, y[i][e]));
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
    l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
    if (qr[r] >= nq) continue;
    const long long row = base + i0 + qr[r], ob = row * d.ld_out + static_cast<long long>(hr[r]) * d.vdim;
    const float unit = pow2i(E - 2 * SPLIT_TOP), inv = l[r] > 0.f ? 1.f / l[r] : 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int col = 8 * j + 2 * tq;
      if (col >= d.vdim) continue;
      const float y0 = o[j][2 * r] * unit * inv * gate_of(d, row, hr[r], col);
      const float y1 = col + 1 < d.vdim ? o[j][2 * r + 1] * unit * inv * gate_of(d, row, hr[r], col + 1) : 0.f;
      if (ovec) {
        if (d.out_dt == VY_BF16) *reinterpret_cast<__nv_bfloat162*>(reinterpret_cast<__nv_bfloat16*>(d.out) + ob + col) = __floats2bfloat162_rn(y0, y1);
        else *reinterpret_cast<float2*>(reinterpret_cast<float*>(d.out) + ob + col) = make_float2(y0, y1);
      } else store2_any(d.out, d.out_dt, ob + col, y0, y1, d.vdim - col);
    }
  }
}

template <int HL, int N>
static size_t talk_mma_smem(const TalkDev& d) {
  using C = TalkMma<HL, N>;
  const size_t kb = ((d.dim + 15) & ~15) * 2 + 16, vb = ((d.vdim + 15) & ~15) * 2 + 16, G = d.kv_heads;
  return 2 * TM_R * kb + 2 * G * N * (kb + vb) + 2 * C::H * C::PB + 2 * 16 * C::MT * C::TB + 16 + sizeof(float) * (C::H * C::XH + TM_R + 16 * C::MT + 2 * G * N) + 16;
}

// keys per tile: 32, or 16 where the key / value heads of 32 do not fit; 0: this geometry is not for the kernel
static int talk_mma_keys(const TalkDev& d) {
  const int per = d.heads / d.kv_heads;
  if (d.dim > 64 || d.vdim > 64) return 0;
  constexpr size_t most = 227 * 1024;
  if (d.heads == 8) return talk_mma_smem<3, 32>(d) <= most ? 32 : 0;
  if (d.heads == 16) return talk_mma_smem<4, 32>(d) <= most ? 32 : talk_mma_smem<4, 16>(d) <= most ? 16 : 0;
  if (d.heads == 32 && per % 2 == 0) return talk_mma_smem<5, 32>(d) <= most ? 32 : talk_mma_smem<5, 16>(d) <= most ? 16 : 0;   // two heads share a warp's keys
  return 0;
}

static WinDev talk_keys(const TalkDev& d) {   // the rows a step sees, in the words of the splitting launch
  WinDev v = {};
  v.cu = d.cu; v.pos0 = d.pos0; v.table = d.table; v.tw = d.tw; v.bs = d.bs;
  v.kp = d.kp; v.vp = d.vp; v.pool_dt = d.pool_dt;
  v.k_row = static_cast<long long>(d.kv_heads) * d.dim; v.v_row = static_cast<long long>(d.kv_heads) * d.vdim;
  v.heads = d.heads; v.kv_heads = d.kv_heads; v.dim = d.dim; v.vdim = d.vdim;
  v.window = d.window;
  return v;
}

long long talk_attn_mma_floats(const TalkDev& d, int n_seqs, int max_new) {
  if (!talk_mma_keys(d)) return 0;
  const long long a = window_attn_split_floats(talk_keys(d), n_seqs, max_new), b = talk_attn_tc_applies(d, 1, max_new) ? window_attn_tc_floats(talk_keys(d), n_seqs, max_new) : 0;
  return a > b ? a : b;   // of either layout; as many times one sequence's as there are, by which vy_talk_attn reckons how many fit
}

template <int HL, int N>
static cudaError_t launch_talk_mma(const TalkDev& d, const SplitKv& w, int n_seqs, int max_new, cudaStream_t st) {
  const size_t smem = talk_mma_smem<HL, N>(d);
  static std::atomic<unsigned long long> allowed{0};
  if (smem > 48 * 1024) {
    cudaError_t e = allow_smem(talk_attn_mma_kernel<HL, N>, allowed);
    if (e != cudaSuccess) return e;
  }
  const auto al = [](const void* p, int a) { return reinterpret_cast<uintptr_t>(p) % a == 0; };
  const bool qvec = d.q_dt == VY_F32 && d.dim % 4 == 0 && d.ldq % 4 == 0 && al(d.q, 16);
  const bool ovec = d.vdim % 2 == 0 && d.ld_out % 2 == 0 && al(d.out, d.out_dt == VY_BF16 ? 4 : 8);
  constexpr int TQ = TalkMma<HL, N>::TQ;
  return launch_kernel(talk_attn_mma_kernel<HL, N>, dim3((max_new + TQ - 1) / TQ, n_seqs), dim3(TM_T), smem, st, d, w, (d.dim + 15) & ~15, (d.vdim + 15) & ~15,
                       qvec, ovec);
}

cudaError_t launch_talk_attn_mma(const TalkDev& d, int n_seqs, int max_new, float* ws, const int** odd, cudaStream_t st) {
  if (talk_attn_tc_applies(d, n_seqs, max_new)) return launch_talk_attn_tc(d, talk_keys(d), n_seqs, max_new, ws, odd, st);
  SplitKv w;
  cudaError_t e = launch_window_attn_split(talk_keys(d), n_seqs, max_new, ws, &w, st);
  if (e != cudaSuccess) return e;
  *odd = w.odd;
  const int N = talk_mma_keys(d);
  if (d.heads == 8) return launch_talk_mma<3, 32>(d, w, n_seqs, max_new, st);
  if (d.heads == 16) return N == 32 ? launch_talk_mma<4, 32>(d, w, n_seqs, max_new, st) : launch_talk_mma<4, 16>(d, w, n_seqs, max_new, st);
  return N == 32 ? launch_talk_mma<5, 32>(d, w, n_seqs, max_new, st) : launch_talk_mma<5, 16>(d, w, n_seqs, max_new, st);
}

}  // namespace vy
