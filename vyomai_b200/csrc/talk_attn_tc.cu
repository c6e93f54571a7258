// Prompts of the attention whose heads exchange scores on tcgen05 (vy_talk_attn; see talking_attn.cu), in fp32 precision from fp16 halves (split_mma.cuh): 8, 16 or 32 heads of at most 64
// channels over 1, 2 or 4 key / value heads.
//
// A CTA owns all H heads of 128 / H queries: 128 rows (head, query), a lane of tensor memory each, so that the 32 rows of a warp share a key / value head. Per tile of 64 keys
//   scores:    all rows times the keys of each key / value head, whose rows alone are kept (the others' lanes are masked out of the product);
//   exchange:  the capped scores go to shared memory as halves, [query, head][key]; the rows of `talk` spread over the queries' diagonal (128 x 128, made once) times that are the mixed scores;
//   values:    the weights, written over the mixed scores, times the values of each key / value head, masked in the same way.
// Queries and the spread `talk` lie in tensor memory too, so that shared memory holds a whole tile's keys and values of four heads ahead. One warp sends off exchanges and
// values, one the next tile's scores, two bring keys and values, sixteen hold the rows, four threads a row with 16 keys and 16 channels each. A tile's values are added while the next one's
// exchange is under way.
//
// What bounds it: 6700 cycles a tile. Products are under way in 5600: 120 of 128 x 64 x 16 at 45 to 60 cycles (the pipe's own counter: active 47 % of the time), where those of a key / value head keep a quarter of their
// rows when there are four. The rows' own chain - 2000 for caps and halves, 1000 until the exchange is back, 1600 for the softmax - hides behind them or hides them. A CTA's start
// takes 13000 (queries, `talk` and 64 keys from memory, instructions not yet in the cache). Eight warps of rows with two tiles' scores in tensor memory, products of all scores against all
// rows: 218 us; masked products by one warp: 193; by two: 150.
// 2 x 1437 tokens, 16 heads of 64 over 4: 326 us by talk_attn_mma_kernel, 150 here; one of 700, 8 heads: 175 / 58; one of 64: 32 / 17. Errors are 0.73 to 0.96 of that kernel's (14 shapes, with caps and
// without, scores of standard deviation 0.3 to 8): the cap's tanh divides as exactly as fp32 can, which its cancellation needs, the weights' exponents are of differences of scores, and a
// query's heads meet in one accumulation or two. With the exponents multiplied out before the difference and the contraction in the rows' order they were up to 1.09 of it, at the same time.
#include "seqmix.cuh"
#include "split_mma.cuh"
#include "talk_attn.cuh"
#include "vy_ptx.cuh"

namespace vy {

constexpr int TT_ROWS = 128, TT_KEYS = 64, TT_ATOM2 = TT_ROWS * 128, TT_ATOM = TT_KEYS * 128;
constexpr int TT_PARTS = 4, TT_PER = TT_KEYS / TT_PARTS;   // threads of a row, keys and channels of each
constexpr int TT_KS = 3, TT_VS = 2, TT_MAXG = 4;
constexpr int TT_WARPS = 4 * TT_PARTS, TT_THREADS = 32 * (TT_WARPS + 4);   // rows; then copies, products, tensor memory, one that only looks at the ranges
constexpr float TT_SCORE = 0x1p14f, TT_MIXED = 0x1p20f;   // as TM_SCORE, TM_MIXED (talk_attn_mma.cu)

struct TalkGeo {
  int dim16, nks, k_atoms, per, heads, n_seqs, qvec, ovec;   // heads: key / value heads of a stage of the rings
  unsigned short khi[4], klo[4];   // where the halves of channels 16 k .. lie in a tile of keys, in 16 bytes
};

__device__ __forceinline__ void tt_split(f32x2 v, uint32_t& hi, uint32_t& lo) {
  const float2 x = unpair(v);
  const __half2 h = __floats2half2_rn(x.x, x.y);
  const float2 b = __half22float2(h), y = unpair(fma2(pair(b.x, b.y), pair(-1.f / LO_UNIT), mul2(v, pair(1.f / LO_UNIT))));
  hi = pack_h2(h);
  lo = pack_h2(__floats2half2_rn(y.x, y.y));
}

__device__ __forceinline__ float at_most_100(float a) {   // NaN stays, as in cap_score; fminf would give the 100, and the score the cap
  float r;
  asm("min.NaN.f32 %0, %1, 0f42C80000;" : "=f"(r) : "f"(a));
  return r;
}

__global__ void __launch_bounds__(TT_THREADS, 1)
talk_attn_tc_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ TalkDev d, const __grid_constant__ SplitKv w, const __grid_constant__ TalkGeo geo,
                    const __grid_constant__ PoisonRef poison) {
  pdl_trigger();
  extern __shared__ __align__(1024) unsigned char tt_smem[];
  const int H = d.heads, G = d.kv_heads, TQ = TT_ROWS / H, HS = geo.heads, k_bytes = geo.k_atoms * TT_ATOM;
  constexpr int v_bytes = 2 * TT_ATOM;
  unsigned char* Ss = tt_smem;                          // queries, then capped scores as halves, hi | lo, then results
  unsigned char* Ks = Ss + 2 * TT_ATOM2;                // [stages]
  unsigned char* Vs = Ks + TT_KS * HS * k_bytes;             // [stages]
  float* units = reinterpret_cast<float*>(Vs + TT_VS * HS * v_bytes);   // [tile parity][key / value head][K | V][key]
  float* qe = units + 2 * TT_MAXG * 2 * TT_KEYS;        // units of the queries' rows
  float* te = qe + TT_ROWS;                             // of the rows of talk
  float* share = te + 32;                               // [part][row]: maxima, then sums
  float* about = share + TT_PARTS * TT_ROWS;                   // [key / value head][largest key entry, not for halves, largest value entry]
  uint32_t* talk = reinterpret_cast<uint32_t*>(about + 4 * TT_MAXG);   // [head][head], hi | lo halves
  uint64_t* bars = reinterpret_cast<uint64_t*>(talk + 32 * 32);
  uint64_t *kfull = bars, *kempty = kfull + TT_KS, *vfull = kempty + TT_KS, *vempty = vfull + TT_VS, *sfull = vempty + TT_VS, *xready = sfull + 1, *xfull = xready + 1, *pready = xfull + 1,
           *ofull = pready + 1, *done = ofull + 1;
  int* kissued = reinterpret_cast<int*>(done + 1);
  int* vissued = kissued + TT_KS;
  uint32_t* tmem_at = reinterpret_cast<uint32_t*>(vissued + TT_VS);
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  if (warp == TT_WARPS + 1 && lane == 0) {
    for (int i = 0; i < TT_KS; ++i) {
      mbar_init(&kfull[i], 1);
      mbar_init(&kempty[i], 1);
      kissued[i] = 0;
    }
    for (int i = 0; i < TT_VS; ++i) {
      mbar_init(&vfull[i], 1);
      mbar_init(&vempty[i], 1);
      vissued[i] = 0;
    }
    for (uint64_t* b : {sfull, xfull, ofull}) mbar_init(b, 1);
    mbar_init(done, 2);
    for (uint64_t* b : {xready, pready}) mbar_init(b, TT_WARPS);
    fence_mbar_init();
  }
  __syncthreads();
  pdl_wait();
  const int turn = blockIdx.x / geo.n_seqs, s = blockIdx.x - turn * geo.n_seqs, base = d.cu[s], n = d.cu[s + 1] - base;
  const int blk = (n + TQ - 1) / TQ - 1 - turn;   // the last queries see the most keys: they go first, of all sequences
  if (blk < 0) return;
  if (warp == TT_WARPS + 2) {
    tmem_alloc(tmem_at, 512);
    tmem_relinquish();
  }
  const int i0 = blk * TQ, nq = min(TQ, n - i0), p0 = d.pos0[s], p_lo = p0 + i0, p_hi = p_lo + nq - 1;
  const int lo = d.window > 0 ? max(p_lo - d.window + 1, 0) : 0, lo0 = d.window > 0 ? max(p0 - d.window + 1, 0) : 0;
  const int tiles = (p_hi - lo + TT_KEYS) / TT_KEYS, slot0 = lo - lo0;
  const auto list = [&](int g) { return (static_cast<long long>(s) * G + g) * w.cap + slot0; };
  const int loads = tiles * G / HS;
  const auto load_k = [&](int i) {   // HS key / value heads' keys, by one lane
    const int b = i % TT_KS;
    ++kissued[b];
    mbar_arrive_expect_tx(&kfull[b], HS * k_bytes);
    for (int k = 0; k < HS; ++k)
      for (int a = 0; a < geo.k_atoms; ++a)
        tma_load_2d(Ks + (b * HS + k) * k_bytes + a * TT_ATOM, &map, &kfull[b], 64 * a, static_cast<int>(list((i * HS + k) % G)) + i * HS / G * TT_KEYS);
  };
  const auto load_v = [&](int i) {
    const int b = i % TT_VS;
    ++vissued[b];
    mbar_arrive_expect_tx(&vfull[b], HS * v_bytes);
    for (int k = 0; k < HS; ++k)
      for (int a = 0; a < 2; ++a)
        tma_load_2d(Vs + (b * HS + k) * v_bytes + a * TT_ATOM, &map, &vfull[b], (w.v_at >> 1) + 64 * a, static_cast<int>(list((i * HS + k) % G)) + i * HS / G * TT_KEYS);
  };
  if (warp == TT_WARPS) {
    if (elect_one_sync()) {
      for (int i = 0; i < min(TT_KS, loads); ++i) load_k(i);
      for (int i = 0; i < min(TT_VS, loads); ++i) load_v(i);
    }
    __syncwarp();
  }
  bool odd = false;
  if (warp >= TT_WARPS && warp - TT_WARPS < G) {
    const int k = warp - TT_WARPS, sg = s * G + k, keys = p0 + n - lo0;
    float top_k;
    const bool no = split_odd(w, sg, keys, top_k);
    unsigned tv = 0u;
    for (int x = lane; x < (keys + SPLIT_ROWS - 1) / SPLIT_ROWS; x += 32) tv = max(tv, w.range[static_cast<long long>(sg) * w.blocks + x].y);
    tv = __reduce_max_sync(0xffffffffu, tv);
    if (lane == 0) {
      about[3 * k] = top_k;
      about[3 * k + 1] = no ? 1.f : 0.f;
      about[3 * k + 2] = __uint_as_float(tv);
    }
  }
  // `talk` as halves, a warp per row; queries as numbers, 16 bytes of row r at place (its channels / 4) ^ (r & 15): sixteen lanes share a row
#pragma unroll 1
  for (int k = warp; k < H; k += TT_WARPS + 4) {
    float x = 0.f;
    if (lane < H) x = d.talk ? ld_as_float(d.talk, d.talk_dt, k * H + lane) : (lane == k ? 1.f : 0.f);
    const float m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(x))));   // a NaN's bits are the largest
    odd = odd || !(m < INFINITY) || !(m * (d.softcap > 0.f ? fminf(d.softcap, TT_SCORE) : TT_SCORE) <= TT_MIXED);
    const int e = split_exponent(m);
    const float y = x * split_scale(e);
    const __half hi = __float2half_rn(y), lo_ = __float2half_rn((y - __half2float(hi)) * (1.f / LO_UNIT));
    if (lane < H) talk[k * H + lane] = __half_as_ushort(hi) | static_cast<uint32_t>(__half_as_ushort(lo_)) << 16;
    if (lane == 0) te[k] = pow2i(e - SPLIT_TOP);
  }
  const int tqs = 31 - __clz(TQ);
  if (warp < TT_WARPS) {
    const int l16 = lane & 15;
    const auto fetch = [&](const auto& from) {
#pragma unroll 4
      for (int r = warp * 2 + (lane >> 4); r < TT_ROWS; r += 2 * TT_WARPS) {
        const int i = r & (TQ - 1);
        const long long at = static_cast<long long>(base + i0 + i) * d.ldq + static_cast<long long>(r >> tqs) * d.dim;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < nq && l16 * 4 < d.dim) x = from(at, l16 * 4);
        *reinterpret_cast<float4*>(Ss + r * 256 + ((l16 ^ (r & 15)) << 4)) = x;
        unsigned top = max(max(abs_bits(x.x), abs_bits(x.y)), max(abs_bits(x.z), abs_bits(x.w)));   // bits: a NaN's are the largest
#pragma unroll
        for (int k = 1; k < 16; k <<= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, k));
        if (l16 == 0) qe[r] = __uint_as_float(top);
        odd = odd || top >= 0x7f800000u;   // the exchange takes all queries' rows: times zero such a score would still be a NaN in the others'
      }
    };
    if (geo.qvec) fetch([&](long long at, int c) { return *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(d.q) + at + c); });
    else fetch([&](long long at, int c) { return load4_any(d.q, d.q_dt, at, c, d.dim); });
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_at, S0 = tmem, X0 = tmem + 64, O0 = tmem + 128, Q0 = tmem + 192, T0 = tmem + 256;   // scores; mixed scores, then weights; weighted values; queries, hi | lo; spread talk, hi | lo
  const int quarter = warp & 3, part = warp >> 2, row = quarter * 32 + lane, h = row >> tqs, q = row & (TQ - 1), g = ((quarter * 32) >> tqs) / geo.per;   // of row warps
  const uint32_t at = static_cast<uint32_t>(quarter * 32) << 16;
  // The exchange's contraction goes through the scores by query, so that a query's heads come in one step of 16 or two, and steps of others add zeros: an accumulation cuts off. Heads
  // are turned by the query, for lanes next to one another to write to different banks
  const int turned = q << (tqs < 3 ? 1 : 0), xrow = q * H + ((h + turned) & (H - 1));
  float qunit = 0.f;
  if (warp < TT_WARPS) {   // the row as halves, and the weights of its query's rows
    {
      const int e = split_exponent(qe[row]);
      const float sc = split_scale(e);
      qunit = pow2i(e - SPLIT_TOP);
#pragma unroll 1
      for (int c = part * TT_PER; c < (part + 1) * TT_PER; c += 16) {
        uint32_t hi[8], lo_[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 x = *reinterpret_cast<const float4*>(Ss + row * 256 + (((c / 4 + i) ^ (row & 15)) << 4));
          split2(x.x * sc, x.y * sc, hi[2 * i], lo_[2 * i]);
          split2(x.z * sc, x.w * sc, hi[2 * i + 1], lo_[2 * i + 1]);
        }
        tmem_st_x8(Q0 + at + c / 2, hi);
        tmem_st_x8(Q0 + 32 + at + c / 2, lo_);
      }
    }
#pragma unroll 1
    for (int c0 = part * (128 / TT_PARTS); c0 < (part + 1) * (128 / TT_PARTS); c0 += 16) {   // columns of hi | lo: column c holds rows 2 c and 2 c + 1
      uint32_t w16[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int k = 2 * ((c0 + i) & 63), b = k - turned;
        const uint32_t x = __byte_perm(talk[h * H + (b & (H - 1))], talk[h * H + ((b + 1) & (H - 1))], c0 < 64 ? 0x5410u : 0x7632u);
        w16[i] = k >> (7 - tqs) == q ? x : 0u;
      }
      tmem_st_x16(T0 + at + c0, w16);
    }
    tmem_st_wait();
  }
  const float qmul = qunit * d.scale;
  float bound = 0.f;   // of a channel's share of any score
  for (int k = 0; k < G; ++k) {
    odd = odd || about[3 * k + 1] != 0.f;
    bound = fmaxf(bound, about[3 * k]);
  }
  odd = odd || (warp < TT_WARPS && !(fabsf(qmul) * about[3 * g] <= TT_SCORE * 0x1p-13f));
  tc_fence_before();
  if (__syncthreads_or(odd)) {   // not for fp16 halves: the fp32 form's
    if (warp == TT_WARPS) {
      mbar_drain(kfull, kissued, TT_KS);   // the copies in flight write to this CTA's memory
      mbar_drain(vfull, vissued, TT_VS);
      if (lane == 0) w.odd[s * G] = 1;
    }
    __syncthreads();
    if (warp == TT_WARPS + 2) tmem_dealloc(tmem, 512);
    return;
  }
  tc_fence_after();
  bool alive = true;
  if (warp == TT_WARPS || warp == TT_WARPS + 3) {
    // ---- copies: keys by one warp, values by another ----
    const bool keys = warp == TT_WARPS;
    const int stages = keys ? TT_KS : TT_VS;
    uint64_t* empty = keys ? kempty : vempty;
#pragma unroll 1
    for (int i = stages; i < loads && alive; ++i) {
      alive = mbar_wait_soft(&empty[i % stages], (i / stages - 1) & 1, poison);
      if (alive && elect_one_sync()) {
        if (keys) load_k(i);
        else load_v(i);
      }
      __syncwarp();
    }
  } else if (warp == TT_WARPS + 1 || warp == TT_WARPS + 2) {
    // ---- products, by a lane each: exchange and values by one warp, scores by another, behind the exchange, which the rows are waiting for ----
    constexpr uint32_t id_s = make_idesc(0, TT_ROWS, TT_KEYS, 0, 0), id_x = make_idesc(0, TT_ROWS, TT_KEYS, 0, 1), id_o = make_idesc(0, TT_ROWS, 64, 0, 1);
    const int of1 = (32 >> tqs) / geo.per, of2 = (64 >> tqs) / geo.per, of3 = (96 >> tqs) / geo.per;   // key / value heads of the quarters
    const auto other = [](int k2, int of) { return k2 == of ? 0u : 0xffffffffu; };                     // masks out other heads' rows
    if (elect_one_sync()) {
      if (warp == TT_WARPS + 2) {
        const uint64_t k_at0 = make_smem_desc_sw128(0, 16, 1024) + (smem_u32(Ks) >> 4);
        int stage = 0, parity = 0;
#pragma unroll 1
        for (int t = 0; t < tiles; ++t) {
          if (t > 0) alive = mbar_wait_soft(xfull, (t - 1) & 1, poison) && alive;   // the last scores have been read
#pragma unroll 1
          for (int k2 = 0; k2 < G && alive;) {
            alive = mbar_wait_soft(&kfull[stage], parity, poison);
            tc_fence_after();
            if (!alive) break;
            uint64_t k_at = k_at0 + (stage * HS * k_bytes >> 4);
#pragma unroll 1
            for (int k = 0; k < HS; ++k, ++k2, k_at += k_bytes >> 4) {
              const uint32_t m0 = other(k2, 0), m1 = other(k2, of1), m2 = other(k2, of2), m3 = other(k2, of3);
#pragma unroll
              for (int c = 0; c < 4; ++c)
                if (c < geo.nks) umma_f16_ta_lanes(S0, Q0 + 32 + 8 * c, k_at + geo.khi[c], id_s, c != 0, m0, m1, m2, m3);
#pragma unroll
              for (int c = 0; c < 4; ++c)
                if (c < geo.nks) umma_f16_ta_lanes(S0, Q0 + 8 * c, k_at + geo.klo[c], id_s, 1, m0, m1, m2, m3);
              umma_f16_ta_lanes_shift11(S0, Q0, k_at, id_s, m0, m1, m2, m3);
#pragma unroll
              for (int c = 1; c < 4; ++c)
                if (c < geo.nks) umma_f16_ta_lanes(S0, Q0 + 8 * c, k_at + geo.khi[c], id_s, 1, m0, m1, m2, m3);
            }
            umma_commit(&kempty[stage]);
            if (++stage == TT_KS) {
              stage = 0;
              parity ^= 1;
            }
          }
          if (!alive) break;
          umma_commit(sfull);
        }
      } else {
        const uint64_t vd = make_smem_desc_sw128(0, TT_ATOM, 1024), x_at = vd + (smem_u32(Ss) >> 4), v_at0 = vd + (smem_u32(Vs) >> 4);
        int stage = 0, parity = 0;
#pragma unroll 1
        for (int t = 0; t < tiles; ++t) {
          alive = mbar_wait_soft(xready, t & 1, poison) && alive;
          tc_fence_after();
          if (!alive) break;
#pragma unroll
          for (int k = 0; k < 8; ++k) umma_f16_ta(X0, T0 + 64 + 8 * k, x_at + k * 128, id_x, k != 0);
#pragma unroll
          for (int k = 0; k < 8; ++k) umma_f16_ta(X0, T0 + 8 * k, x_at + (TT_ATOM2 >> 4) + k * 128, id_x, 1);
          umma_f16_ta_shift11(X0, T0, x_at, id_x);
#pragma unroll
          for (int k = 1; k < 8; ++k) umma_f16_ta(X0, T0 + 8 * k, x_at + k * 128, id_x, 1);
          umma_commit(xfull);
          alive = mbar_wait_soft(pready, t & 1, poison);
          tc_fence_after();
#pragma unroll 1
          for (int k2 = 0; k2 < G && alive;) {
            alive = mbar_wait_soft(&vfull[stage], parity, poison);
            tc_fence_after();
            if (!alive) break;
            uint64_t v_at = v_at0 + (stage * HS * v_bytes >> 4);
#pragma unroll 1
            for (int k = 0; k < HS; ++k, ++k2, v_at += v_bytes >> 4) {
              const uint32_t m0 = other(k2, 0), m1 = other(k2, of1), m2 = other(k2, of2), m3 = other(k2, of3);
#pragma unroll
              for (int c = 0; c < 4; ++c) umma_f16_ta_lanes(O0, X0 + 32 + 8 * c, v_at + c * 128, id_o, c != 0, m0, m1, m2, m3);
#pragma unroll
              for (int c = 0; c < 4; ++c) umma_f16_ta_lanes(O0, X0 + 8 * c, v_at + (TT_ATOM >> 4) + c * 128, id_o, 1, m0, m1, m2, m3);
              umma_f16_ta_lanes_shift11(O0, X0, v_at, id_o, m0, m1, m2, m3);
#pragma unroll
              for (int c = 1; c < 4; ++c) umma_f16_ta_lanes(O0, X0 + 8 * c, v_at + c * 128, id_o, 1, m0, m1, m2, m3);
            }
            umma_commit(&vempty[stage]);
            if (++stage == TT_VS) {
              stage = 0;
              parity ^= 1;
            }
          }
          if (!alive) break;
          umma_commit(ofull);
        }
      }
    }
    __syncwarp();
  } else if (warp < TT_WARPS) {
    // ---- rows ----
    const int p = p_lo + q;
    constexpr float L2E = 1.4426950408889634f, L2E_LO = static_cast<float>(1.4426950408889634 - static_cast<double>(L2E));
    // the score or, under a cap, the exponent of 2 of e^(2 s / cap), its factor in two parts so that it is as good as fp32 arithmetic
    const bool capped = d.softcap > 0.f;
    const float to2 = capped ? 2.f * L2E / d.softcap : 1.f, q1 = qmul * to2;
    const f32x2 qhi = pair(q1), qlo = pair(capped ? fmaf(qmul, to2, -q1) : 0.f), cap = pair(d.softcap), cap2 = pair(-2.f * d.softcap);
    // one power of two for all scores: what bounds them
    float largest = bound * 0x1p13f * d.dim;
    {
      const float4 v = reinterpret_cast<const float4*>(qe)[lane];
      const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w))));
      largest *= pow2i(split_exponent(__uint_as_float(top)) - SPLIT_TOP) * fabsf(d.scale);
    }
    if (capped) largest = fmaxf(fminf(largest, d.softcap), d.softcap * 0x1p-20f);   // cap - 2 cap r is off by about 2^-23 cap, whatever the score
    const int es = split_exponent(largest);
    const f32x2 sf = pair(split_scale(es));
    // a power of two for the mixed scores, and what makes a difference of them an exponent of 2: of differences, which are small where they matter, the product's rounding is too. Scores
    // that are this small are all alike
    const float mf = fmaxf(te[h] * pow2i(es - SPLIT_TOP), 0x1p-80f), f1 = mf * L2E, f2 = mf * L2E_LO;
    const f32x2 fhi = pair(f1), flo = pair(f2);
    float sink;
    const bool has = sink_of(d, h, sink);
    float m = has ? sink / mf : -INFINITY, l = has && part == 0 ? 1.f : 0.f;
    const int E = split_exponent(about[3 * g + 2]);
    const float v_unit = pow2i(SPLIT_TOP - E);
    f32x2 o[TT_PER / 2];
#pragma unroll
    for (int i = 0; i < TT_PER / 2; ++i) o[i] = pair(0.f);
    const auto take_o = [&]() {
      uint32_t raw[TT_PER];
      tmem_ld_x16(O0 + at + TT_PER * part, raw);
      const f32x2 cut = pair(0.5f * (TT_KEYS / 16 + 1) * 0x1p-25f);   // SPLIT_CUT, of a sum of TT_KEYS / 16 accumulations
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < TT_PER; i += 2) {
        const f32x2 v = pair_bits(raw[i], raw[i + 1]);
        o[i / 2] = add2(o[i / 2], fma2(v, cut, v));
      }
    };
    const f32x2 cut_s = pair(0.5f * (geo.nks + 1) * 0x1p-25f), cut_x = pair(0.5f * ((H + 15) / 16 + 1) * 0x1p-25f);
    // units: thread i brings those of key i % 64 of key / value head i / 64, a tile ahead
    const bool brings = threadIdx.x < TT_KEYS * G;
    const float2* unit_at = reinterpret_cast<const float2*>(w.unit) + list(brings ? threadIdx.x / TT_KEYS : 0) + threadIdx.x % TT_KEYS;
    float2 unit = brings ? unit_at[0] : make_float2(0.f, 0.f);
#pragma unroll 1
    for (int t = 0; t < tiles; ++t) {
      float* un = units + (t & 1) * TT_MAXG * 2 * TT_KEYS;
      if (brings) {
        float* to = un + threadIdx.x / TT_KEYS * 2 * TT_KEYS + threadIdx.x % TT_KEYS;
        to[0] = unit.x;
        to[TT_KEYS] = unit.y;
        if (t + 1 < tiles) unit = unit_at[(t + 1) * TT_KEYS];
      }
      named_bar_sync(1, 32 * TT_WARPS);
      const float* ku = un + g * 2 * TT_KEYS + TT_PER * part;
      const float* vu = ku + TT_KEYS;
      alive = mbar_wait_soft(sfull, t & 1, poison) && alive;
      tc_fence_after();
      uint32_t raw[TT_PER];
      tmem_ld_x16(S0 + at + TT_PER * part, raw);
      tmem_ld_wait();
      {
        uint32_t hi[TT_PER / 2], lo_[TT_PER / 2];
#pragma unroll
        for (int i = 0; i < TT_PER / 2; i += 2) {
          const float4 k4 = *reinterpret_cast<const float4*>(ku + 2 * i);
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const f32x2 v = pair_bits(raw[2 * (i + k)], raw[2 * (i + k) + 1]), y = mul2(fma2(v, cut_s, v), k ? pair(k4.z, k4.w) : pair(k4.x, k4.y));
            f32x2 x = fma2(y, qhi, mul2(y, qlo));
            if (capped) {   // cap tanh(s / cap) = cap - 2 cap / (1 + e^(2 s / cap)); far out that is cap or -cap
              const float2 e = unpair(x);
              const f32x2 z = add2(pair(vy_ex2_approx(at_most_100(e.x)), vy_ex2_approx(at_most_100(e.y))), pair(1.f));
              const float2 z2 = unpair(z);
              f32x2 r = pair(vy_rcp_approx(z2.x), vy_rcp_approx(z2.y));
              r = fma2(r, fma2(mul2(z, pair(-1.f)), r, pair(1.f)), r);   // as good as a division: the difference below cancels
              x = fma2(cap2, r, cap);
            }
            tt_split(mul2(x, sf), hi[i + k], lo_[i + k]);
          }
        }
        unsigned char* to = Ss + xrow * 128;
#pragma unroll
        for (int i = 0; i < TT_PER / 2; i += 4) {
          const int c = (2 * TT_PER * part + 4 * i) ^ ((xrow & 7) << 4);
          *reinterpret_cast<uint4*>(to + c) = make_uint4(hi[i], hi[i + 1], hi[i + 2], hi[i + 3]);
          *reinterpret_cast<uint4*>(to + TT_ATOM2 + c) = make_uint4(lo_[i], lo_[i + 1], lo_[i + 2], lo_[i + 3]);
        }
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(xready);
      if (t > 0) {   // the last tile's values
        alive = mbar_wait_soft(ofull, (t - 1) & 1, poison) && alive;
        tc_fence_after();
        take_o();
      }
      alive = mbar_wait_soft(xfull, t & 1, poison) && alive;
      tc_fence_after();
      tmem_ld_x16(X0 + at + TT_PER * part, raw);
      tmem_ld_wait();
      f32x2 x[TT_PER / 2];
#pragma unroll
      for (int i = 0; i < TT_PER / 2; ++i) {
        const f32x2 v = pair_bits(raw[2 * i], raw[2 * i + 1]);
        x[i] = fma2(v, cut_x, v);
      }
      const int f = lo + t * TT_KEYS + TT_PER * part;   // position of this thread's first key
      if (!(f + TT_PER - 1 <= p_lo && (d.window <= 0 || p_hi - f < d.window))) {
        const int jhi = p - f + 1, jlo = d.window > 0 ? p - d.window + 1 - f : 0;   // visible: [jlo, jhi)
        const auto below = [](int j) { return j <= 0 ? 0u : j >= 32 ? 0xffffffffu : (1u << j) - 1u; };
        const unsigned vis = below(jhi) & ~below(jlo);
#pragma unroll
        for (int i = 0; i < TT_PER / 2; ++i) {
          const float2 e = unpair(x[i]);
          x[i] = pair(vis >> (2 * i) & 1u ? e.x : -INFINITY, vis >> (2 * i + 1) & 1u ? e.y : -INFINITY);
        }
      }
      float tops[2] = {m, -INFINITY};
#pragma unroll
      for (int i = 0; i < TT_PER / 2; ++i) {
        const float2 e = unpair(x[i]);
        tops[i & 1] = fmaxf(tops[i & 1], fmaxf(e.x, e.y));
      }
      share[part * TT_ROWS + row] = fmaxf(tops[0], tops[1]);
      named_bar_sync(2 + quarter, 32 * TT_PARTS);   // the row's other threads: their maxima; all have read the mixed scores
      float mn = share[row];
#pragma unroll
      for (int k = 1; k < TT_PARTS; ++k) mn = fmaxf(mn, share[k * TT_ROWS + row]);
      const float cr = mn == -INFINITY ? 1.f : vy_ex2_approx(fmaf(m - mn, f1, (m - mn) * f2));
      m = mn;
      const f32x2 mm = pair(m == -INFINITY ? 0.f : -m);
      f32x2 sum = pair(0.f);
      {
        uint32_t hi[TT_PER / 2], lo_[TT_PER / 2];
        const f32x2 vs = pair(v_unit);
#pragma unroll
        for (int i = 0; i < TT_PER / 2; i += 2) {
          const float4 v4 = *reinterpret_cast<const float4*>(vu + 2 * i);
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const f32x2 less = add2(x[i + k], mm);
            const float2 z = unpair(fma2(less, fhi, mul2(less, flo)));
            const f32x2 e = pair(vy_ex2_approx(z.x), vy_ex2_approx(z.y));
            sum = add2(sum, e);
            tt_split(mul2(e, mul2(k ? pair(v4.z, v4.w) : pair(v4.x, v4.y), vs)), hi[i + k], lo_[i + k]);
          }
        }
        tmem_st_x8(X0 + at + TT_PER / 2 * part, hi);
        tmem_st_x8(X0 + 32 + at + TT_PER / 2 * part, lo_);
      }
      const float2 a = unpair(sum);
      l = fmaf(l, cr, a.x + a.y);
      if (__any_sync(0xffffffffu, cr != 1.f)) {
#pragma unroll
        for (int i = 0; i < TT_PER / 2; ++i) o[i] = mul2(o[i], pair(cr));
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(pready);
    }
    alive = mbar_wait_soft(ofull, (tiles - 1) & 1, poison) && alive;
    tc_fence_after();
    take_o();
    named_bar_sync(2 + quarter, 32 * TT_PARTS);   // all have read the maxima
    share[part * TT_ROWS + row] = l;
    named_bar_sync(2 + quarter, 32 * TT_PARTS);
    l = share[row];
#pragma unroll
    for (int k = 1; k < TT_PARTS; ++k) l += share[k * TT_ROWS + row];
    // through shared memory, where the queries were, to lanes that share rows, eight a row
    const bool shared_gate = d.gate && !d.gate_ch;
    float whole = pow2i(E - 2 * SPLIT_TOP) * (l > 0.f ? 1.f / l : 0.f);
    if (shared_gate && q < nq) whole *= gate_of(d, base + i0 + q, h, 0);
#pragma unroll
    for (int i = 0; i < TT_PER / 4; ++i) {
      const float2 a = unpair(mul2(o[2 * i], pair(whole))), b = unpair(mul2(o[2 * i + 1], pair(whole)));
      *reinterpret_cast<float4*>(Ss + row * 256 + (((part * (TT_PER / 4) + i) ^ (row & 15)) << 4)) = make_float4(a.x, a.y, b.x, b.y);
    }
    named_bar_sync(2 + quarter, 32 * TT_PARTS);
#pragma unroll 1
    for (int r = quarter * 32 + part * 4 + (lane >> 3); r < quarter * 32 + 32; r += 4 * TT_PARTS) {
      const int i = r & (TQ - 1), hr = r >> tqs, c = (lane & 7) * 8;
      if (i >= nq || c >= d.vdim) continue;
      const long long qrow = base + i0 + i, ob = qrow * d.ld_out + static_cast<long long>(hr) * d.vdim;
      float y[8];
#pragma unroll
      for (int k = 0; k < 2; ++k) *reinterpret_cast<float4*>(y + 4 * k) = *reinterpret_cast<const float4*>(Ss + r * 256 + (((c / 4 + k) ^ (r & 15)) << 4));
      if (d.gate && d.gate_ch) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (c + k < d.vdim) y[k] *= gate_of(d, qrow, hr, c + k);
      }
      if (geo.ovec) st8_from_float(d.out, d.out_dt, ob + c, y);
      else {
#pragma unroll
        for (int k = 0; k < 8; k += 2) store2_any(d.out, d.out_dt, ob + c + k, y[k], y[k + 1], d.vdim - c - k);
      }
    }
  }
  tc_fence_before();
  if (__syncthreads_or(!alive)) {   // a wait has timed out: what is still in flight ends before the memory is given back
    if (warp == TT_WARPS) {
      mbar_drain(kfull, kissued, TT_KS);
      mbar_drain(vfull, vissued, TT_VS);
    } else if (warp == TT_WARPS + 1 || warp == TT_WARPS + 2) {
      if (elect_one_sync()) umma_commit(done);
      __syncwarp();
      for (uint32_t spins = 0; spins < (1u << 20) && !mbar_try_wait(done, 0); ++spins) {}
    }
  }
  __syncthreads();
  if (warp == TT_WARPS + 2) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

static int tt_round(int n, int m) { return (n + m - 1) / m * m; }

bool talk_attn_tc_applies(const TalkDev& d, int n_seqs, int max_new) {
  const int per = d.heads / d.kv_heads, tq = TT_ROWS / d.heads;
  const long long whole = static_cast<long long>(d.tw) * d.bs - max_new / 2, sees = d.window > 0 && d.window < whole ? d.window : whole;   // keys a query of the longest sequence sees on average
  const long long ctas = static_cast<long long>(n_seqs) * ((max_new + tq - 1) / tq);
  // What a CTA costs before its first tile (7 us) is more than that of talk_attn_mma_kernel, several of which share an SM's time better; a tile costs less than half. It pays where all CTAs
  // run at once (64 x 16 tokens, 8 heads: 30 against 38 us) and where a query sees 256 keys on average (2 x 1437: 150 / 326;
  // 6 x 520 tokens, 32 heads: 1.06 to 2 times as fast). Past that: 148 x 16 tokens, 16 heads: 56 / 40; one of 2000 behind a window of 64: 58 / 54; behind one of 128: equal; 32 heads of 32 and
  // 300 x 100 tokens: 1058 / 853. What is cached counts: mma.sync / here, 16 heads of 64, 40 x 64 tokens
  // on 2000 cached ones 1008 / 466, on 500 304 / 157, behind a window of 256 163 / 107; 100 x 32 on 1000 596 / 324; 50 x 100 from position 0 beside one token on 4000 951 / 269. Beside one long prompt the CTAs of short ones find nothing to do, at 0.7 us each: 1500 and 20 of 3 tokens, 32 heads, 7900 CTAs: 175 / 136.
  if (ctas > num_sms() && (ctas > 8 * num_sms() || sees < 256 || d.dim + d.vdim < 64)) return false;   // 8 x 600, 8 heads of 16: 64 / 60
  // the rows of a warp (H / 4 heads) share a key / value head
  return (d.heads == 8 || d.heads == 16 || d.heads == 32) && (d.kv_heads == 1 || d.kv_heads == 2 || d.kv_heads == 4) && per % (d.heads / 4) == 0 && d.dim <= 64 && d.vdim <= 64;
}

cudaError_t launch_talk_attn_tc(const TalkDev& d, const WinDev& keys, int n_seqs, int max_new, float* ws, const int** odd, cudaStream_t st) {
  const SplitKv w = window_attn_tc_layout(keys, n_seqs, max_new, ws);
  *odd = w.odd;
  cudaError_t e = launch_split_rows(keys, n_seqs, w, st);
  if (e != cudaSuccess) return e;
  const uint64_t dims[2] = {static_cast<uint64_t>(w.row_bytes / 2), static_cast<uint64_t>(n_seqs) * d.kv_heads * w.cap}, strides[2] = {0, static_cast<uint64_t>(w.row_bytes)};
  const uint32_t box[2] = {64, TT_KEYS};
  CUtensorMap map;
  if (get_tensor_map_cached(&map, VY_BF16, 2, ws, dims, strides, box, 1) != VY_OK) return cudaErrorInvalidValue;   // 16-bit entries of either kind
  const auto al = [](const void* p, int a) { return reinterpret_cast<uintptr_t>(p) % a == 0; };
  TalkGeo geo = {};
  geo.dim16 = tt_round(d.dim, 16);
  geo.nks = geo.dim16 / 16;
  geo.k_atoms = tt_round(2 * geo.dim16, 64) / 64;
  geo.per = d.heads / d.kv_heads;
  geo.heads = min(d.kv_heads, 2);
  geo.n_seqs = n_seqs;
  for (int k = 0; k < geo.nks; ++k) {
    const auto at = [](int x, int atom) { return static_cast<unsigned short>((x / 64 * atom + x % 64 * 2) / 16); };
    geo.khi[k] = at(16 * k, TT_ATOM);
    geo.klo[k] = at(geo.dim16 + 16 * k, TT_ATOM);
  }
  geo.qvec = d.q_dt == VY_F32 && d.dim % 4 == 0 && d.ldq % 4 == 0 && al(d.q, 16);
  geo.ovec = d.vdim % 8 == 0 && d.ld_out % 8 == 0 && al(d.out, 16);
  const size_t smem = 2 * TT_ATOM2 + static_cast<size_t>(geo.heads) * (TT_KS * geo.k_atoms + TT_VS * 2) * TT_ATOM +
                      sizeof(float) * (2 * TT_MAXG * 2 * TT_KEYS + TT_ROWS + 32 + TT_PARTS * TT_ROWS + 4 * TT_MAXG + 32 * 32) + 256;
  static std::atomic<unsigned long long> allowed{0};
  e = allow_smem(talk_attn_tc_kernel, allowed);
  if (e != cudaSuccess) return e;
  PoisonRef poison = {};
  if (!poison_ref(&poison)) return cudaErrorMemoryAllocation;
  const int tq = TT_ROWS / d.heads;
  return launch_kernel(talk_attn_tc_kernel, dim3(static_cast<unsigned>((max_new + tq - 1) / tq) * n_seqs), dim3(TT_THREADS), smem, st, map, d, w, geo, poison);
}

}  // namespace vy
