// State-space and linear-attention prompts on tcgen05, chunks of 128 tokens: linear_attn_mma.cu's first and third launch, with fp32 precision from fp16 halves (split_mma.cuh).
//
// Read-outs, O = (Q K^T . D) V + diag(decay to i) Q S_before. A CTA owns a chunk, 64 value columns and heads that share q and k. Its scores are made once and stay in
// tensor memory. Per head eight warps split the values and the state, a head ahead of the sixteen others, which turn scores into weights (by row as fp16
// halves, into tensor memory; four threads per row, 32 keys each) and bring out the head before: its two products have an accumulator each, since a row's weights have a
// unit of their own. Small products go first, then hi hi onto 2^-11 of them (scale-input-d). Gates come and outputs leave by bulk copies of 32 columns.
// A decay from a key to a row further on than the key's run of 32 is a product of two, at the end of the run: one exponential per row and run.
// Without steps of time (TD false: a fixed decay per head, q, k and v activated as they are read) a head has q and k of its own, and a CTA takes its value columns 64 at a time where it
// otherwise takes heads; decays come from a table of powers.
// Loops are kept short: a CTA's code beyond the instruction cache costs as much as its arithmetic.
//
// What bounds it: chains of short steps with twenty-four warps to hide them (9,500 cycles per head: 2,500 weights, 1,800 splitting them, 3,500 bringing out) and
// 17,000 cycles before the first head. 4 x 2048 tokens, 32 heads of 128 x 64 in groups of 8: 115 us (mma.sync, chunks of 64: 299). Tried: eight warps for the rows, scores in
// registers 180; outputs and gates through L1 rather than bulk copies 124; four warps that split, 129; a full division in the gate 138.
// 4 x 2048 tokens, 8 heads of 128 x 128 with decays by head and silu: 114 here, 93 for the states, 17 for the scan (mma.sync: 332, 140, 39); with divisions in silu 141 and 101.
#include "linear_attn.cuh"
#include "split_mma.cuh"
#include "vy_ptx.cuh"

namespace vy {

constexpr int LT_SPLIT = 8, LT_WARPS = LT_SPLIT + 16, LT_THREADS = 32 * LT_WARPS;   // warps that split, then sixteen for weights and outputs
constexpr int LT_REGS = 80, LT_REGS_SPLIT = 64, LT_REGS_ROWS = 88;   // a thread: at launch, and as six groups of four warps share them out: 2 x 64 + 4 x 88 = 6 x 80
constexpr int LT_ATOM = LT_C * 128;   // 64 fp16 entries of each of 128 rows, 128-byte swizzle
constexpr int LT_HALF = LT_C * 128;   // 32 fp32 columns of the 128 rows of a head's gate or outputs, 128-byte swizzle

__device__ __forceinline__ f32x2 two_of(float4 v) { return pair(v.x, v.y); }
__device__ __forceinline__ f32x2 other_two_of(float4 v) { return pair(v.z, v.w); }
// split2 of both entries times f
__device__ __forceinline__ void split_pair(f32x2 v, f32x2 f, f32x2 f_lo, unsigned& hi, unsigned& lo) {   // f_lo: f / LO_UNIT
  const float2 x = unpair(mul2(v, f));
  const __half2 h = __floats2half2_rn(x.x, x.y);
  const float2 b = __half22float2(h);
  const float2 y = unpair(fma2(pair(b.x, b.y), pair(-1.f / LO_UNIT), mul2(v, f_lo)));
  hi = pack_h2(h);
  lo = pack_h2(__floats2half2_rn(y.x, y.y));
}
// x / (1 + e^-x) of both entries, in a third of the instructions of two exponentials and two divisions: e^-x as 2^t with what rounding t left over brought back, then a reciprocal with
// a Newton step, whose quotient is corrected once (without it the outputs' error grows by a hundredth); see silu_near. Infinities and NaN give what the division gives
__device__ __forceinline__ float within_100(float a) {   // NaN stays
  float r;
  asm("min.NaN.f32 %0, %1, 0f42C80000;\n\tmax.NaN.f32 %0, %0, 0fC2C80000;" : "=f"(r) : "f"(a));
  return r;
}
// EXP: of expf, as good as the division's to the last bit but for rare ones (of q, k and v themselves: by 2^t the outputs' error is a seventh larger)
template <bool EXP = false>
__device__ __forceinline__ f32x2 silu_pair(f32x2 x) {
  constexpr float L2E = 1.4426950408889634f, L2E_LO = static_cast<float>(1.4426950408889634 - static_cast<double>(L2E));
  const float2 g = unpair(x);
  const f32x2 c = pair(within_100(g.x), within_100(g.y)), t = mul2(c, pair(-L2E));   // e^100 is infinite
  const f32x2 left = fma2(c, pair(-L2E_LO), fma2(c, pair(-L2E), mul2(t, pair(-1.f))));
  const float2 tt = unpair(t), cc = unpair(c);
  const f32x2 y = add2(EXP ? pair(expf(-cc.x), expf(-cc.y)) : mul2(pair(vy_ex2_approx(tt.x), vy_ex2_approx(tt.y)), fma2(left, pair(0.6931471805599453f), pair(1.f))), pair(1.f));
  const float2 ys = unpair(mul2(y, pair(RECIP_SCALE)));
  const f32x2 minus = mul2(y, pair(-1.f)), r0 = mul2(pair(vy_rcp_approx(ys.x), vy_rcp_approx(ys.y)), pair(RECIP_SCALE)), r = fma2(r0, fma2(minus, r0, pair(1.f)), r0), q = mul2(x, r);
  const float2 a = unpair(fma2(fma2(minus, q, x), r, q)), b = unpair(mul2(x, r0));
  return pair(a.x == a.x ? a.x : b.x, a.y == a.y ? a.y : b.y);   // infinities
}
template <int ACT>
__device__ __forceinline__ float4 act_quad(float4 x) {
  if constexpr (ACT == VY_UACT_SILU) {
    const float2 a = unpair(silu_pair<true>(two_of(x))), b = unpair(silu_pair<true>(other_two_of(x)));
    x = make_float4(a.x, a.y, b.x, b.y);
  }
  return x;
}
static __device__ __noinline__ float gate_any(float x, int act) { return apply_uact(x, act); }

// The states that the chunks leave, U = sum_j decay(j .. end of the chunk) w_j k_j v_j^T. A CTA as below: k (as A operand, channels by tokens) is split once, the values by
// eight warps that each own eight columns - tokens are the summed index, so that a channel and a column have one unit each, and a column's largest entry needs no other warp -
// and the outputs are brought out by eight others. Raw values come by bulk copies, two heads ahead, and the states leave by such. Tokens are summed in two accumulators
// of 64: one of 128 loses more (see SPLIT_CUT; error of the final states 1.55e-7, 1.30e-7 in two). As in la_states_kernel, the largest entries of the rows and columns of q,
// k, v and of a carried state are looked at, and where they lie too far apart the CTA's heads are left to the walk.
// What bounds it: 12,000 cycles before the first head, then the splitting's instructions. 4 x 2048 tokens, 32 heads of 128 x 64 in groups of 8: 60 us (mma.sync, chunks of 64: 102;
// the scan between, of half as many states, 33 for 85).
constexpr int LTS_THREADS = 544;   // eight warps that split, eight that bring out, one for copies and products
template <bool TD, int ACT>
__global__ void __launch_bounds__(LTS_THREADS, 1)
la_states_tc_kernel(const __grid_constant__ CUtensorMap v_map, const __grid_constant__ CUtensorMap u_map, const __grid_constant__ RecDev d, const __grid_constant__ LaChunks w, int hp, int vslices,
                    const __grid_constant__ PoisonRef poison) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(1024) unsigned char lts_smem[];
  unsigned char* Ks = lts_smem;                  // [token][64 channels] hi, hi, lo, lo
  unsigned char* Ws = Ks + 4 * LT_ATOM;          // [token][64 columns] hi, lo
  unsigned char* Rs = Ws + 2 * LT_ATOM;          // [2][2] raw values, 32 columns each
  unsigned char* Os = Rs + 4 * LT_HALF;          // [2] states, 32 columns each
  float* es = reinterpret_cast<float*>(Os + 2 * LT_HALF);   // [head][128] decay to the chunk's end times write strength
  float* ku = es + LT_HEADS * LT_C;              // [128], [4][64]: units of k's channels and of the heads' columns
  float* wu = ku + LT_C;
  Range* range = reinterpret_cast<Range*>(wu + 4 * 64);   // [4]: k, q, v, state
  uint64_t* bars = reinterpret_cast<uint64_t*>(range + 4);
  uint64_t *vfull = bars, *wready = bars + 2, *wfree = bars + 3, *dfull = bars + 4, *dfree = bars + 6, *done = bars + 8;
  uint32_t* tmem_at = reinterpret_cast<uint32_t*>(bars + 9);
  int* issued = reinterpret_cast<int*>(tmem_at + 1);   // [2] copies of values sent for
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31, t = threadIdx.x;
  const int s = blockIdx.z, c = TD ? blockIdx.x / vslices : blockIdx.x, v0 = TD ? (blockIdx.x % vslices) * 64 : 0, h0 = blockIdx.y * hp;
  const int base = d.cu[s], n = d.cu[s + 1] - base, t0 = c * LT_C;
  if (t0 >= n) return;
  const int nt = min(LT_C, n - t0), hq = TD ? h0 / (d.heads / d.kv_heads) : h0;
  const int items = TD ? hp : vslices;   // heads, or 64 columns each of the one head, which then share q and k
  const auto head_of = [&](int hh) { return TD ? h0 + hh : h0; };
  const auto col_of = [&](int hh) { return TD ? v0 : 64 * hh; };
  const long long r0 = base + t0, slot = la_slot(d, s, c);
  const bool few = nt < 8;
  bool alive = true;
  const auto load_v = [&](int hh) {   // by one elected lane
    const int b = hh & 1;
    ++issued[b];
    mbar_arrive_expect_tx(&vfull[b], 2 * LT_HALF);
    for (int i = 0; i < 2; ++i) tma_load_2d(Rs + (2 * b + i) * LT_HALF, &v_map, &vfull[b], head_of(hh) * d.vdim + col_of(hh) + 32 * i, static_cast<int>(r0));
  };
  if (t < 4) range[t] = {0u, RANGE_NONE};
  __syncthreads();
  if (warp == 16) {
    if (lane == 0) {
      for (int i = 0; i < 2; ++i) {
        mbar_init(&vfull[i], 1);
        mbar_init(&dfull[i], 1);
        mbar_init(&dfree[i], 8);
        issued[i] = 0;
      }
      mbar_init(wready, 256);
      mbar_init(wfree, 1);
      mbar_init(done, 1);
      fence_mbar_init();
    }
    __syncwarp();
    if (elect_one_sync()) {
      load_v(0);
      if (items > 1) load_v(1);
    }
    __syncwarp();
    tmem_alloc(tmem_at, 256);
    tmem_relinquish();
  } else {
    if (!TD && warp == 8) {
      const float decay = d.decay[h0];
#pragma unroll 1
      for (int i = lane; i < LT_C; i += 32) es[i] = i < nt ? power(decay, nt - 1 - i) : 0.f;
      if (lane == 0) {
        w.D[slot * d.heads + h0] = power(decay, nt);
        w.top[slot * d.heads + h0] = 0u;
      }
    }
    if (TD && warp >= 8)
#pragma unroll 1
      for (int hh = warp - 8; hh < hp; hh += 8) {   // as token_decays, in short loops: code that a CTA runs once comes cold
        const int h = h0 + hh;
        float* mine = es + hh * LT_C;
        double* sums = reinterpret_cast<double*>(Os) + hh * LT_C;
        const float rate = expf(ld_as_float(d.a_log, d.a_log_dt, h)), dt_b = ld_as_float(d.dt_bias, d.a_log_dt, h);
        double end = 0.0;
        float dt = lane < nt ? d.dt[(r0 + lane) * d.ld_dt + h] : 0.f;
#pragma unroll 1
        for (int i = lane; i < LT_C; i += 32) {
          const float strength = i < nt ? softplusf_(dt + dt_b) : 0.f;
          if (i + 32 < nt) dt = d.dt[(r0 + i + 32) * d.ld_dt + h];
          double L = fmaxf(-rate * strength, MIN_LOG_DECAY);
#pragma unroll
          for (int k = 1; k < 32; k <<= 1) {
            const double x = __shfl_up_sync(0xffffffffu, L, k);
            if (lane >= k) L += x;
          }
          L += end;
          end = __shfl_sync(0xffffffffu, L, 31);
          sums[i] = L;
          mine[i] = strength;
        }
#pragma unroll 1
        for (int i = lane; i < LT_C; i += 32) mine[i] *= expf(static_cast<float>(end - sums[i]));
        if (lane == 0 && v0 == 0) {
          w.D[slot * d.heads + h] = expf(static_cast<float>(end));
          w.top[slot * d.heads + h] = 0u;
        }
      }
    // k by the first eight warps, 16 channels each; the others only look at q
    const bool isq = warp >= 8;
    if (!isq || v0 == 0) {
      const int row = lane >> 2, ch = 16 * (warp & 7) + 4 * (lane & 3);
      const float* p = reinterpret_cast<const float*>(isq ? d.q : d.k) + static_cast<long long>(hq) * d.dim + ch;
      const long long ld = isq ? d.ldq : d.ldk;
      float4 x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) x[i] = row + 8 * i < nt && ch < d.dim ? *reinterpret_cast<const float4*>(p + (r0 + row + 8 * i) * ld) : make_float4(0.f, 0.f, 0.f, 0.f);
      if constexpr (ACT != VY_UACT_NONE) {
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = act_quad<ACT>(x[i]);
      }
      Range rk = {0u, RANGE_NONE};
      const uint4 m = look<16, 4>(x, few, d.dim - 16 * (warp & 7) < 4, rk);
      note_warp(range + isq, rk);
      if (!isq) {
        const float4 sc = column_scales(m);
        if (row == 0) *reinterpret_cast<float4*>(ku + ch) = column_units(m);
        unsigned char* to = Ks + (ch >> 6) * LT_ATOM;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int r = row + 8 * i;
          store_split4(to, to + 2 * LT_ATOM, r * 128 + (((ch & 63) * 2) ^ ((r & 7) << 4)), x[i], sc);
        }
      }
    }
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_at;   // [2 heads][tokens 0 .. 63, 64 .. 127][64 columns]
  if (warp < 8) {
    // ---- split: columns 8 warp + 4 (lane & 1) .., tokens row + 16 i; the order of the rows keeps their pieces of the swizzled raw values apart ----
    const int rr = lane >> 1, row = (rr & 8) + 2 * (rr & 3) + (rr >> 2 & 1), vc = 8 * warp + 4 * (lane & 1);
    Range rv = {0u, RANGE_NONE}, rs = rv;   // this thread's share
#pragma unroll 1
    for (int hh = 0; hh < items; ++hh) {
      const int h = head_of(hh), b = hh & 1, vw = min(64, d.vdim - col_of(hh));
      const float* weight = es + (TD ? hh : 0) * LT_C;
      unsigned most_b = 0u;
#pragma unroll
      for (int i = lane; i < LT_C; i += 32) most_b = max(most_b, abs_bits(weight[i]));
      const float most = __uint_as_float(__reduce_max_sync(0xffffffffu, most_b));
      if (c == 0 && d.pos0[s] > 0) {   // the state that is carried in: a thread reads every fourth entry of a column
        const float* sp = d.state + (static_cast<long long>(d.slot[s]) * d.heads + h) * static_cast<long long>(d.dim) * d.vdim + col_of(hh) + (t & 63);
        unsigned top = 0u;
#pragma unroll 1
        for (int i0 = t >> 6; i0 < d.dim; i0 += 64) {   // sixteen rows in flight: four at a time took 15 us a head
          unsigned a[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) a[k] = (t & 63) < vw && i0 + 4 * k < d.dim ? abs_bits(sp[static_cast<long long>(i0 + 4 * k) * d.vdim]) : 0u;
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            top = max(top, a[k]);
            note(rs, __reduce_max_sync(0xffffffffu, a[k]), true);   // a row past the last one notes nothing
          }
        }
        note(rs, top, true);
      }
      alive = mbar_wait_soft(&vfull[b], (hh >> 1) & 1, poison) && alive;
      float4 y[8];
      const unsigned char* from = Rs + (2 * b + (vc >> 5)) * LT_HALF;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = row + 16 * i;
        const float4 x = *reinterpret_cast<const float4*>(from + r * 128 + (((vc & 31) * 4) ^ ((r & 7) << 4)));
        y[i] = r < nt && vc < vw ? act_quad<ACT>(x) : make_float4(0.f, 0.f, 0.f, 0.f);   // other sequences' rows, other heads' columns
      }
      uint4 m = look<8, 2>(y, few, vw - 8 * warp < 4, rv);
      {   // the weighted columns' units from a bound, the columns' largest times the largest weight: rows are within 2^20 of one another, and the halves good to 2^24
        const auto times = [most](unsigned k) { return __float_as_uint(__uint_as_float(k) * most); };
        m = make_uint4(times(m.x), times(m.y), times(m.z), times(m.w));
      }
      const float4 sv = column_scales(m);
      if (hh > 0) alive = mbar_wait_soft(wfree, (hh - 1) & 1, poison) && alive;   // the products of the head before are done
      if (lane < 2) *reinterpret_cast<float4*>(wu + (hh & 3) * 64 + vc) = column_units(m);   // two heads ahead of the slowest reader at most
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = row + 16 * i;
        const float e = weight[r];
        store_split4(Ws, Ws + LT_ATOM, r * 128 + ((vc * 2) ^ ((r & 7) << 4)), make_float4(y[i].x * e, y[i].y * e, y[i].z * e, y[i].w * e), sv);
      }
      fence_proxy_async_smem();
      mbar_arrive(wready);
    }
    note_warp(range + 2, rv);
    note_warp(range + 3, rs);
  } else if (warp == 16) {
    // ---- products ----
    const uint64_t ka = make_smem_desc_sw128(smem_u32(Ks), LT_ATOM, 1024), wb = make_smem_desc_sw128(smem_u32(Ws), 1024, 1024);
    constexpr uint32_t id = make_idesc(0, LT_C, 64, 1, 1);
#pragma unroll 1
    for (int hh = 0; hh < items; ++hh) {
      const int b = hh & 1;
      alive = mbar_wait_soft(wready, hh & 1, poison) && alive;
      if (hh > 1) alive = mbar_wait_soft(&dfree[b], ((hh >> 1) - 1) & 1, poison) && alive;
      tc_fence_after();
      if (alive && elect_one_sync()) {
#pragma unroll 1
        for (int part = 0; part < 2; ++part) {   // 64 tokens each: four steps of 16, 2048 bytes of either operand
          const uint32_t D = tmem + b * 128 + part * 64;
          const uint64_t kh = ka + part * 512, wh = wb + part * 512, kl = kh + (2 * LT_ATOM >> 4), wl = wh + (LT_ATOM >> 4);
#pragma unroll 1
          for (int k = 0; k < 4; ++k) umma_f16(D, kl + k * 128, wh + k * 128, id, k != 0);
#pragma unroll 1
          for (int k = 0; k < 4; ++k) umma_f16(D, kh + k * 128, wl + k * 128, id, 1);
          umma_f16_shift11(D, kh, wh, id);
#pragma unroll 1
          for (int k = 1; k < 4; ++k) umma_f16(D, kh + k * 128, wh + k * 128, id, 1);
        }
        umma_commit(wfree);
        umma_commit(&dfull[b]);
        if (hh + 2 < items) load_v(hh + 2);   // this head's raw values have been read
      }
      __syncwarp();
    }
  } else {
    // ---- the states: channel = row of tensor memory, 32 columns per thread ----
    const int quarter = warp & 3, half = (warp >> 2) & 1, row = quarter * 32 + lane;
    const uint32_t at = static_cast<uint32_t>(quarter * 32) << 16;
    const f32x2 cut = pair(0.5f * (64 / 16 + 1) * 0x1p-25f);   // SPLIT_CUT, of a sum of four accumulations
    const float unit = row < d.dim ? ku[row] : 0.f;
    unsigned char* to = Os + half * LT_HALF + row * 128;
#pragma unroll 1
    for (int hh = 0; hh < items; ++hh) {
      const int b = hh & 1;
      alive = mbar_wait_soft(&dfull[b], (hh >> 1) & 1, poison) && alive;
      tc_fence_after();
      uint32_t x[32], z[32];
      tmem_ld_x32(tmem + b * 128 + at + 32 * half, x);
      tmem_ld_x32(tmem + b * 128 + 64 + at + 32 * half, z);
      if (warp == 8) tma_store_wait_read<0>();   // the states of the head before have left (of the lane that sent them off)
      named_bar_sync(1, 256);
      tmem_ld_wait();
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float4 u = *reinterpret_cast<const float4*>(wu + (hh & 3) * 64 + 32 * half + 4 * k);
        const auto sum = [&](int i) {
          const f32x2 a = pair_bits(x[i], x[i + 1]), p = pair_bits(z[i], z[i + 1]);
          return mul2(add2(fma2(a, cut, a), fma2(p, cut, p)), pair(unit));
        };
        const float2 ya = unpair(mul2(sum(4 * k), two_of(u))), yb = unpair(mul2(sum(4 * k + 2), other_two_of(u)));
        *reinterpret_cast<float4*>(to + ((k ^ (row & 7)) << 4)) = make_float4(ya.x, ya.y, yb.x, yb.y);
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&dfree[b]);
      named_bar_sync(1, 256);
      if (warp == 8) {
        if (alive && elect_one_sync()) {
          for (int i = 0; i < 2; ++i)
            if (col_of(hh) + 32 * i < d.vdim) tma_store_2d(&u_map, Os + i * LT_HALF, col_of(hh) + 32 * i, static_cast<int>((slot * d.heads + head_of(hh)) * d.dim));
          tma_store_commit();
        }
        __syncwarp();
      }
    }
    if (warp == 8) tma_store_wait_read<0>();
  }
  tc_fence_before();
  if (__syncthreads_or(!alive) && warp == 16) {   // a wait has timed out: what is in flight ends before the memory is given back
    if (elect_one_sync()) umma_commit(done);
    __syncwarp();
    for (uint32_t spins = 0; spins < (1u << 20) && !mbar_try_wait(done, 0); ++spins) {}
    mbar_drain(vfull, issued, 2);
  }
  __syncthreads();
  if (t == 0) w.odd[TD ? (slot * gridDim.y + blockIdx.y) * vslices + blockIdx.x % vslices : slot * gridDim.y + blockIdx.y] = too_wide(range[0]) || too_wide(range[1]) || too_wide(range[2]) || too_wide(range[3]);
  if (warp == 16) {
    tc_fence_after();
    tmem_dealloc(tmem, 256);
  }
}

template <bool TD, int ACT>
__global__ void __launch_bounds__(LT_THREADS, 1)
la_outputs_tc_kernel(const __grid_constant__ CUtensorMap gate_map, const __grid_constant__ CUtensorMap out_map, const __grid_constant__ RecDev d, const __grid_constant__ LaChunks w, int hp, int vslices,
                     int dim16, const __grid_constant__ PoisonRef poison) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(1024) unsigned char lt_smem[];
  const int atoms = (dim16 + 63) / 64, q_lo = atoms * LT_ATOM, s_lo = dim16 * 128;
  unsigned char* Qs = lt_smem;                    // hi | lo
  unsigned char* Vs = Qs + 2 * q_lo;              // [2] hi | lo; the keys, until the scores are made
  unsigned char* Ss = Vs + 4 * LT_ATOM;           // hi | lo
  unsigned char* Os = Ss + 2 * s_lo;              // [2] halves of a head's gate, then of its outputs
  float* qu = reinterpret_cast<float*>(Os + 2 * LT_HALF);   // units of the queries' and keys' rows
  float* ku = qu + LT_C;
  float* vu = ku + LT_C;                          // [2] units of a head's value rows
  float* tops = vu + 2 * LT_C;                    // [2][4][128]
  float* decays = tops + 8 * LT_C;                // [head][-Lh, -Ll, strength of a key, decay up to and with a token, strength times decay to the end of the key's run of 32][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(decays + 5 * LT_HEADS * LT_C);
  uint64_t *sfull = bars, *filled = bars + 1, *pfull = bars + 3, *ofull = bars + 5, *ofree = bars + 7, *sready = bars + 9, *sdone = bars + 10, *gfull = bars + 11, *odone = bars + 12, *done = bars + 13;
  uint32_t* tmem_at = reinterpret_cast<uint32_t*>(bars + 14);
  int* issued = reinterpret_cast<int*>(tmem_at + 1);   // copies of gates sent for
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int s = blockIdx.z, c = TD ? blockIdx.x / vslices : blockIdx.x, v0 = TD ? (blockIdx.x % vslices) * 64 : 0, h0 = blockIdx.y * hp;
  const int base = d.cu[s], n = d.cu[s + 1] - base, t0 = c * LT_C;
  if (t0 >= n) return;
  const int nt = min(LT_C, n - t0), hq = TD ? h0 / (d.heads / d.kv_heads) : h0;
  const int items = TD ? hp : vslices;   // heads, or 64 columns each of the one head, which then share q and k
  const auto head_of = [&](int hh) { return TD ? h0 + hh : h0; };
  const auto col_of = [&](int hh) { return TD ? v0 : 64 * hh; };
  const long long r0 = base + t0, slot = la_slot(d, s, c);
  if (warp == 0) {
    if (lane == 0) {
      mbar_init(sfull, 1);
      for (int i = 0; i < 2; ++i) {
        mbar_init(&filled[i], 32 * LT_SPLIT);
        mbar_init(&pfull[i], 16);
        mbar_init(&ofull[i], 1);
        mbar_init(&ofree[i], 16);
      }
      mbar_init(gfull, 1);
      mbar_init(odone, 16);
      *issued = 0;
      mbar_init(sready, 32 * LT_SPLIT);
      mbar_init(sdone, 1);
      mbar_init(done, 1);
      fence_mbar_init();
    }
    __syncwarp();
    tmem_alloc(tmem_at, 512);
    tmem_relinquish();
  }
  if (warp >= LT_WARPS - hp) {
    const int hh = warp - (LT_WARPS - hp);
    float* mine = decays + hh * 5 * LT_C;
    const int h = h0 + hh;
    if constexpr (!TD) {
      const float decay = d.decay[h];   // its powers; up to and with a token
#pragma unroll 1
      for (int i = lane; i < LT_C; i += 32) {
        mine[2 * LT_C + i] = power(decay, i);
        mine[3 * LT_C + i] = power(decay, i + 1);
      }
    } else {
    const float rate = expf(ld_as_float(d.a_log, d.a_log_dt, h)), dt_b = ld_as_float(d.dt_bias, d.a_log_dt, h);
    double before = 0.0;   // log decays summed, as in token_decays; a short loop: code that a CTA runs once comes cold
    float dt = lane < nt ? d.dt[(r0 + lane) * d.ld_dt + h] : 0.f;
#pragma unroll 1
    for (int i = lane; i < LT_C; i += 32) {
      const float strength = i < nt ? softplusf_(dt + dt_b) : 0.f;
      if (i + 32 < nt) dt = d.dt[(r0 + i + 32) * d.ld_dt + h];
      double L = fmaxf(-rate * strength, MIN_LOG_DECAY);
#pragma unroll
      for (int k = 1; k < 32; k <<= 1) {
        const double x = __shfl_up_sync(0xffffffffu, L, k);
        if (lane >= k) L += x;
      }
      L += before;
      before = __shfl_sync(0xffffffffu, L, 31);
      const float hi = static_cast<float>(L);   // two floats: the sums' differences are what counts
      mine[i] = -hi;
      mine[LT_C + i] = -static_cast<float>(L - static_cast<double>(hi));
      mine[2 * LT_C + i] = strength;
      mine[3 * LT_C + i] = expf(hi);
      mine[4 * LT_C + i] = strength * expf(static_cast<float>(before - L));
    }
    }
  } else {   // queries, then keys: eight lanes share a row; the next rows are on their way while two are split
    const int l8 = lane & 7, warps = LT_WARPS - hp, first = warp * 4 + (lane >> 3);
    float4 next[2][4];
    const auto get = [&](int r_0) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int r = r_0 + 4 * warps * u, i = r & (LT_C - 1);
        const bool q = r < LT_C;
        const float* p = reinterpret_cast<const float*>(q ? d.q : d.k) + (r0 + i) * (q ? d.ldq : d.ldk) + static_cast<long long>(hq) * d.dim;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int col = l8 * 4 + 32 * k;
          next[u][k] = r < 2 * LT_C && i < nt && col < d.dim ? *reinterpret_cast<const float4*>(p + col) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
    };
    get(first);
#pragma unroll 1
    for (int r_0 = first; r_0 - (lane >> 3) < 2 * LT_C; r_0 += 8 * warps) {
      float4 x[2][4];
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int k = 0; k < 4; ++k) x[u][k] = act_quad<ACT>(next[u][k]);
      get(r_0 + 8 * warps);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int r = r_0 + 4 * warps * u, i = r & (LT_C - 1);
        float top = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) top = fmaxf(top, fmaxf(fmaxf(fabsf(x[u][k].x), fabsf(x[u][k].y)), fmaxf(fabsf(x[u][k].z), fabsf(x[u][k].w))));
#pragma unroll
        for (int k = 1; k < 8; k <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, k));
        if (r >= 2 * LT_C) continue;
        const int e = split_exponent(top);
        const float sc = split_scale(e);
        if (l8 == 0) qu[r] = pow2i(e - SPLIT_TOP);   // the keys' behind the queries'
        unsigned char* to = (r < LT_C ? Qs : Vs) + i * 128;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int col = l8 * 4 + 32 * k;
          if (col < dim16) {
            uint2 hi, lo;
            split2(x[u][k].x * sc, x[u][k].y * sc, hi.x, lo.x);
            split2(x[u][k].z * sc, x[u][k].w * sc, hi.y, lo.y);
            unsigned char* at = to + (col >> 6) * LT_ATOM + (((col & 63) * 2) ^ ((i & 7) << 4));
            *reinterpret_cast<uint2*>(at) = hi;
            *reinterpret_cast<uint2*>(at + q_lo) = lo;
          }
        }
      }
    }
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_at, P0 = tmem, S0 = tmem + 128, O0 = tmem + 256;   // weights (hi | lo, 64 columns each), scores, [2][Q S | weights V]
  bool alive = true;

  if (warp < LT_SPLIT) {
    // ---- values and states, one after the other, each sent for as soon as the one before is split ----
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(LT_REGS_SPLIT));
    const int t = threadIdx.x, row = t >> 3, col = (t & 7) * 4;   // rows row + 32 i, columns col .. and col + 32 ..
    float4 x[4][2];
    unsigned next_top = 0u;
    const auto get = [&](int turn) {
      const int item = turn >> 1, h = head_of(item), v0 = col_of(item), vw = min(64, d.vdim - v0);
      if (item >= items) return;
      const bool state = turn & 1;
      const float* p = state ? w.U + (slot * d.heads + h) * static_cast<long long>(d.dim) * d.vdim + v0 : reinterpret_cast<const float*>(d.v) + r0 * d.ldv + static_cast<long long>(h) * d.vdim + v0;
      const long long ld = state ? d.vdim : d.ldv;
      const int rows = state ? d.dim : nt;
      if (state) next_top = w.top[slot * d.heads + h];
      // the next head's on its way to L2: from memory they take longer than half a turn
      const float* ahead = p + (!TD ? 64 : state ? d.dim * d.vdim : d.vdim);
      const int ahead_vw = TD ? vw : min(64, d.vdim - v0 - 64);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int r = row + 32 * i;
          x[i][k] = r < rows && col + 32 * k < vw ? *reinterpret_cast<const float4*>(p + r * ld + col + 32 * k) : make_float4(0.f, 0.f, 0.f, 0.f);
          if ((t & 7) == 0 && item + 1 < items && r < rows && 32 * k < ahead_vw) asm volatile("prefetch.global.L2 [%0];" ::"l"(ahead + r * ld + 32 * k));
        }
    };
    get(0);
#pragma unroll 1
    for (int turn = 0; turn < 2 * items; ++turn) {
      const int hh = turn >> 1, b = hh & 1;
      const bool state = turn & 1;
      float* units = vu + b * LT_C;
      unsigned char* to = state ? Ss : Vs + b * 2 * LT_ATOM;
      const int lo_at = state ? s_lo : LT_ATOM, until = state ? dim16 : LT_C;
      const float whole = split_scale(split_exponent(__uint_as_float(next_top)));
      // the buffer's last readers: the scores' product (keys), the products of two heads ago, or that with the state of the head before
      if (state) alive = (hh == 0 || mbar_wait_soft(sdone, (hh - 1) & 1, poison)) && alive;
      else alive = (hh < 2 ? mbar_wait_soft(sfull, 0, poison) : mbar_wait_soft(&ofull[b], ((hh >> 1) - 1) & 1, poison)) && alive;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = row + 32 * i;
        const float4 u = state ? x[i][0] : act_quad<ACT>(x[i][0]), v = state ? x[i][1] : act_quad<ACT>(x[i][1]);
        float f = whole;
        if (!state) {
          float top = fmaxf(fmaxf(fmaxf(fabsf(u.x), fabsf(u.y)), fmaxf(fabsf(u.z), fabsf(u.w))), fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
#pragma unroll
          for (int k = 1; k < 8; k <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, k));
          const int e = split_exponent(top);
          if ((t & 7) == 0) units[r] = pow2i(e);
          f = split_scale(e);
        }
        const f32x2 f2 = pair(f), f_lo = pair(f * (1.f / LO_UNIT));
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          uint2 hi, lo;
          split_pair(two_of(k ? v : u), f2, f_lo, hi.x, lo.x);
          split_pair(other_two_of(k ? v : u), f2, f_lo, hi.y, lo.y);
          unsigned char* at = to + r * 128 + (((col + 32 * k) * 2) ^ ((r & 7) << 4));
          if (r < until) {
            *reinterpret_cast<uint2*>(at) = hi;
            *reinterpret_cast<uint2*>(at + lo_at) = lo;
          }
        }
      }
      get(turn + 1);
      fence_proxy_async_smem();
      mbar_arrive(state ? sready : &filled[b]);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(LT_REGS_ROWS));
    const int j = (warp - LT_SPLIT) >> 2, quarter = warp & 3, row = quarter * 32 + lane;   // j: this warp's run of 32 keys, and of 16 outputs
    const uint32_t at = static_cast<uint32_t>(quarter * 32) << 16;
    const float qunit = qu[row];
    const f32x2 cut_s = pair(0.5f * (dim16 / 16 + 1) * 0x1p-25f), cut_v = pair(0.5f * (2 * quarter + 3) * 0x1p-25f);   // SPLIT_CUT: over the channels; over the tokens that these rows see
    const bool products = quarter == 0 && j == 2;   // a warp whose rows see none of its keys sends off the products
    const uint64_t kmaj = make_smem_desc_sw128(0, 16, 1024), mnmaj = make_smem_desc_sw128(0, 1024, 1024);
    const auto desc = [](uint64_t kind, uint32_t at) { return kind + (at >> 4); };
    const uint32_t q_at = smem_u32(Qs), v_at = smem_u32(Vs), s_at = smem_u32(Ss);
    const auto along = [](int k) { return static_cast<uint32_t>((k >> 2) * LT_ATOM + (k & 3) * 32); };   // channels 16 k .. of queries or keys
    const int nks = dim16 / 16;
    constexpr uint32_t id_s = make_idesc(0, LT_C, LT_C, 0, 0), id_o = make_idesc(0, LT_C, 64, 0, 1);
    if (products) {
      if (elect_one_sync()) {
  #pragma unroll 1
      for (int k = 0; k < nks; ++k) umma_f16(S0, desc(kmaj, q_at + q_lo + along(k)), desc(kmaj, v_at + along(k)), id_s, k != 0);
  #pragma unroll 1
      for (int k = 0; k < nks; ++k) umma_f16(S0, desc(kmaj, q_at + along(k)), desc(kmaj, v_at + q_lo + along(k)), id_s, 1);
        umma_f16_shift11(S0, desc(kmaj, q_at), desc(kmaj, v_at), id_s);
#pragma unroll 1
        for (int k = 1; k < nks; ++k) umma_f16(S0, desc(kmaj, q_at + along(k)), desc(kmaj, v_at + along(k)), id_s, 1);
        umma_commit(sfull);
      }
      __syncwarp();
    }
    alive = mbar_wait_soft(sfull, 0, poison);
    tc_fence_after();
    uint32_t raw[32];
    if (j <= quarter) {   // true scores, 0 past the row's own token
      tmem_ld_x32(S0 + at + 32 * j, raw);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        const float2 u = *reinterpret_cast<const float2*>(ku + 32 * j + i);
        const f32x2 v = pair_bits(raw[i], raw[i + 1]);
        const float2 y = unpair(mul2(fma2(v, cut_s, v), mul2(pair(qunit), pair(u.x, u.y))));
        raw[i] = __float_as_uint(32 * j + i <= row ? y.x : 0.f);
        raw[i + 1] = __float_as_uint(32 * j + i + 1 <= row ? y.y : 0.f);
      }
      tmem_st_x32(S0 + at + 32 * j, raw);
    } else {   // weights that stay zero
#pragma unroll
      for (int i = 0; i < 32; ++i) raw[i] = 0u;
      uint32_t (&zero)[16] = *reinterpret_cast<uint32_t (*)[16]>(raw);
      tmem_st_x16(P0 + at + 16 * j, zero);
      tmem_st_x16(P0 + at + 64 + 16 * j, zero);
    }
    tmem_st_wait();
    unsigned char* half = Os + (j >> 1) * LT_HALF;   // this warp's 16 columns: 16-byte pieces 4 (j & 1) .. of its rows there
    const auto bulk_of = [&](int hh) { return d.vdim - col_of(hh) >= 64 && nt == LT_C; };   // otherwise a box of outputs would go over other heads' or sequences'
    const bool copies = quarter == 0 && j == 3;      // another such warp: gates in, outputs out
    const auto gate_in = [&](int hh) {
      if (alive && elect_one_sync()) {
        if (d.gate) {
          ++*issued;
          mbar_arrive_expect_tx(gfull, 2 * LT_HALF);
          for (int i = 0; i < 2; ++i) tma_load_2d(Os + i * LT_HALF, &gate_map, gfull, head_of(hh) * d.vdim + col_of(hh) + 32 * i, static_cast<int>(r0));
        } else mbar_arrive(gfull);
      }
      __syncwarp();
    };
    if (copies) gate_in(0);
    const auto skip_of = [&](int hh) { return TD && hh < hp ? ld_as_float(d.skip, d.a_log_dt, h0 + hh) : 0.f; };
    const auto top_of = [&](int hh) { return hh < items ? w.top[slot * d.heads + head_of(hh)] : 0u; };
    float skip = skip_of(0);
    unsigned state_top = top_of(0);
    float f_state = 0.f, f_chunk = 0.f;   // of the head whose outputs are to be brought out
#pragma unroll 1
    for (int hh = 0; hh <= items; ++hh) {
      const int b = hh & 1;
      float fs = 0.f, fc = 0.f;
      if (products && hh < items) {
        alive = mbar_wait_soft(sready, hh & 1, poison) && alive;
        if (hh > 1) alive = mbar_wait_soft(&ofree[b], ((hh >> 1) - 1) & 1, poison) && alive;   // the outputs of two heads ago have been read
        tc_fence_after();
        if (alive && elect_one_sync()) {   // Q S
          const uint32_t D = O0 + b * 128;
    #pragma unroll 1
      for (int k = 0; k < nks; ++k) umma_f16(D, desc(kmaj, q_at + q_lo + along(k)), desc(mnmaj, s_at + k * 2048), id_o, k != 0);
    #pragma unroll 1
      for (int k = 0; k < nks; ++k) umma_f16(D, desc(kmaj, q_at + along(k)), desc(mnmaj, s_at + s_lo + k * 2048), id_o, 1);
          umma_f16_shift11(D, desc(kmaj, q_at), desc(mnmaj, s_at), id_o);
#pragma unroll 1
          for (int k = 1; k < nks; ++k) umma_f16(D, desc(kmaj, q_at + along(k)), desc(mnmaj, s_at + k * 2048), id_o, 1);
          umma_commit(sdone);
        }
        __syncwarp();
      }
      if (hh < items) {
        alive = mbar_wait_soft(&filled[b], (hh >> 1) & 1, poison) && alive;
        const float* mine = decays + (TD ? hh : 0) * 5 * LT_C;
        const float* units = vu + b * LT_C;
        fs = pow2i(split_exponent(__uint_as_float(state_top)) - SPLIT_TOP) * qunit * mine[3 * LT_C + row];
        float top = 0.f, mul = 1.f;   // mul: what the row's weights of this run still lack
        if (j <= quarter) {
          tmem_ld_x32(S0 + at + 32 * j, raw);
          const float* key = mine + 32 * j;
          const auto times = [&](float4 by, int i) {
            const float4 u = *reinterpret_cast<const float4*>(units + 32 * j + i);
            const float2 a = unpair(mul2(pair_bits(raw[i], raw[i + 1]), mul2(two_of(by), two_of(u)))), c = unpair(mul2(pair_bits(raw[i + 2], raw[i + 3]), mul2(other_two_of(by), other_two_of(u))));
            raw[i] = __float_as_uint(a.x);
            raw[i + 1] = __float_as_uint(a.y);
            raw[i + 2] = __float_as_uint(c.x);
            raw[i + 3] = __float_as_uint(c.y);
          };
          if constexpr (!TD) {
            const float* powers = mine + 2 * LT_C;
            const int away = row - 32 * j;
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; i += 4)
              times(make_float4(powers[max(away - i, 0)], powers[max(away - i - 1, 0)], powers[max(away - i - 2, 0)], powers[max(away - i - 3, 0)]), i);
          } else if (j < quarter) {   // the decay from a key to the row in two factors, at the end of the key's run
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; i += 4) times(*reinterpret_cast<const float4*>(key + 4 * LT_C + i), i);
            mul = expf(fminf((key[31] - mine[row]) + (key[LT_C + 31] - mine[LT_C + row]), 0.f));
          } else {
            const f32x2 Lh = pair(-mine[row]), Ll = pair(-mine[LT_C + row]);
            const float diag = skip * units[row];
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              const float4 hi = *reinterpret_cast<const float4*>(key + i), lo = *reinterpret_cast<const float4*>(key + LT_C + i);
              const float2 x = unpair(add2(add2(Lh, two_of(hi)), add2(Ll, two_of(lo)))), y = unpair(add2(add2(Lh, other_two_of(hi)), add2(Ll, other_two_of(lo))));
              const float4 by = *reinterpret_cast<const float4*>(key + 2 * LT_C + i);
              const float2 ea = unpair(mul2(two_of(by), pair(expf(fminf(x.x, 0.f)), expf(fminf(x.y, 0.f)))));
              const float2 eb = unpair(mul2(other_two_of(by), pair(expf(fminf(y.x, 0.f)), expf(fminf(y.y, 0.f)))));
              times(make_float4(ea.x, ea.y, eb.x, eb.y), i);
            }
#pragma unroll
            for (int i = 0; i < 32; ++i) raw[i] = __float_as_uint(__uint_as_float(raw[i]) + (i == lane ? diag : 0.f));
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) top = fmaxf(top, fabsf(__uint_as_float(raw[i])));
          top *= mul;
          float* all = tops + b * 4 * LT_C + row;
          all[j * LT_C] = top;
        }
        skip = skip_of(hh + 1);
        state_top = top_of(hh + 1);
        named_bar_sync(2 + quarter, 128);
        for (int k = 0; k <= quarter; ++k) top = fmaxf(top, tops[(b * 4 + k) * LT_C + row]);
        const int e = split_exponent(top);
        fc = pow2i(e - SPLIT_TOP) * pow2i(-SPLIT_TOP);
        if (j <= quarter) {
          const f32x2 f = pair(split_scale(e) * mul), f_lo = pair(split_scale(e) * mul * (1.f / LO_UNIT));
          uint32_t hi[16], lo[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) split_pair(pair_bits(raw[2 * i], raw[2 * i + 1]), f, f_lo, hi[i], lo[i]);
          if (hh > 0) {   // the head before has been multiplied
            alive = mbar_wait_soft(&ofull[b ^ 1], ((hh - 1) >> 1) & 1, poison) && alive;
            tc_fence_after();
          }
          tmem_st_x16(P0 + at + 16 * j, hi);
          tmem_st_x16(P0 + at + 64 + 16 * j, lo);
          tmem_st_wait();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&pfull[b]);
        if (products) {
          alive = mbar_wait_soft(&pfull[b], (hh >> 1) & 1, poison) && alive;
          tc_fence_after();
          if (alive && elect_one_sync()) {   // weights V
            const uint32_t D = O0 + b * 128 + 64, V = v_at + b * 2 * LT_ATOM;
#pragma unroll 1
            for (int k = 0; k < LT_C / 16; ++k) umma_f16_ta(D, P0 + 64 + 8 * k, desc(mnmaj, V + k * 2048), id_o, k != 0);
#pragma unroll 1
            for (int k = 0; k < LT_C / 16; ++k) umma_f16_ta(D, P0 + 8 * k, desc(mnmaj, V + LT_ATOM + k * 2048), id_o, 1);
            umma_f16_ta_shift11(D, P0, desc(mnmaj, V), id_o);
#pragma unroll 1
            for (int k = 1; k < LT_C / 16; ++k) umma_f16_ta(D, P0 + 8 * k, desc(mnmaj, V + k * 2048), id_o, 1);
            umma_commit(&ofull[b]);   // of both products
          }
          __syncwarp();
        }
      }
      if (hh > 0) {   // bring out the head before
        const int ob = b ^ 1, h = head_of(hh - 1), v0 = col_of(hh - 1), vw = min(64, d.vdim - v0);
        const bool bulk = bulk_of(hh - 1);
        alive = mbar_wait_soft(&ofull[ob], ((hh - 1) >> 1) & 1, poison) && alive;
        tc_fence_after();
        uint32_t os[16], oc[16];
        tmem_ld_x16(O0 + ob * 128 + at + 16 * j, os);
        tmem_ld_x16(O0 + ob * 128 + 64 + at + 16 * j, oc);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ofree[ob]);
        alive = mbar_wait_soft(gfull, (hh - 1) & 1, poison) && alive;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          f32x2 y[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const f32x2 a = pair_bits(os[4 * k + 2 * e], os[4 * k + 2 * e + 1]), p = pair_bits(oc[4 * k + 2 * e], oc[4 * k + 2 * e + 1]);
            y[e] = fma2(fma2(p, cut_v, p), pair(f_chunk), mul2(fma2(a, cut_s, a), pair(f_state)));
          }
          float4* piece = reinterpret_cast<float4*>(half + row * 128 + (((4 * (j & 1) + k) ^ (row & 7)) << 4));
          if (d.gate) {
            const float4 g = *piece;
            f32x2 ga = two_of(g), gb = other_two_of(g);
            if (d.gate_act == VY_UACT_SILU) {
              ga = silu_pair(ga);
              gb = silu_pair(gb);
            } else {
              ga = pair(gate_any(g.x, d.gate_act), gate_any(g.y, d.gate_act));
              gb = pair(gate_any(g.z, d.gate_act), gate_any(g.w, d.gate_act));
            }
            y[0] = mul2(y[0], ga);
            y[1] = mul2(y[1], gb);
          }
          const float2 ya = unpair(y[0]), yb = unpair(y[1]);
          *piece = make_float4(ya.x, ya.y, yb.x, yb.y);
        }
        if (!bulk) {
          __syncwarp();
          const int tcol = lane & 3;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int i = quarter * 32 + 8 * k + (lane >> 2);
            const float4 y = *reinterpret_cast<const float4*>(half + i * 128 + (((4 * (j & 1) + tcol) ^ (i & 7)) << 4));
            if (i < nt && 16 * j + 4 * tcol < vw) *reinterpret_cast<float4*>(reinterpret_cast<float*>(d.out) + (r0 + i) * d.ld_out + static_cast<long long>(h) * d.vdim + v0 + 16 * j + 4 * tcol) = y;
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(odone);
        if (copies) {
          alive = mbar_wait_soft(odone, (hh - 1) & 1, poison) && alive;
          if (alive && bulk && elect_one_sync()) {
            for (int i = 0; i < 2; ++i) tma_store_2d(&out_map, Os + i * LT_HALF, h * d.vdim + v0 + 32 * i, static_cast<int>(r0));
            tma_store_commit();
            tma_store_wait_read<0>();
          }
          __syncwarp();
          if (hh < items) gate_in(hh);
        }
      }
      f_state = fs;
      f_chunk = fc;
    }
  }
  tc_fence_before();
  if (__syncthreads_or(!alive) && warp == LT_SPLIT + 8) {   // a wait has timed out: the products in flight end before the memory is given back
    if (elect_one_sync()) umma_commit(done);
    __syncwarp();
    for (uint32_t spins = 0; spins < (1u << 20) && !mbar_try_wait(done, 0); ++spins) {}
    mbar_drain(gfull, issued, 1);
  }
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

template <bool TD, int ACT>
static bool la_registers() {   // with fewer registers at launch than the warps share out, the first to ask for more would wait for ever: what a compiler gives another number does without this form
  static const bool enough = [] {
    cudaFuncAttributes a;
    return cudaFuncGetAttributes(&a, la_outputs_tc_kernel<TD, ACT>) == cudaSuccess && (a.numRegs + 7) / 8 * 8 == LT_REGS;
  }();
  return enough;
}

static bool row_map(CUtensorMap* m, const void* p, long long cols, long long rows, long long ld, int box_rows) {
  const uint64_t dims[2] = {static_cast<uint64_t>(cols), static_cast<uint64_t>(rows)}, strides[2] = {0, static_cast<uint64_t>(ld) * 4};
  const uint32_t box[2] = {32, static_cast<uint32_t>(box_rows)};
  return get_tensor_map_cached(m, VY_F32, 2, p, dims, strides, box, 1) == VY_OK;
}

template <bool TD, int ACT>
static cudaError_t launch_states(const RecDev& d, const LaChunks& w, int hp, int n_seqs, int max_new, long long rows, cudaStream_t st) {
  const int vslices = (d.vdim + 63) / 64;
  const size_t smem = static_cast<size_t>(6) * LT_ATOM + static_cast<size_t>(6) * LT_HALF + sizeof(float) * ((LT_HEADS + 1) * LT_C + 4 * 64) + 4 * sizeof(Range) + 128;
  static std::atomic<unsigned long long> allowed{0};
  cudaError_t e = allow_smem(la_states_tc_kernel<TD, ACT>, allowed);
  if (e != cudaSuccess) return e;
  PoisonRef poison = {};
  if (!poison_ref(&poison)) return cudaErrorMemoryAllocation;
  CUtensorMap v_map, u_map;
  const long long slots = rows / LM_C + n_seqs;
  if (!row_map(&v_map, d.v, static_cast<long long>(d.heads) * d.vdim, rows, d.ldv, LT_C) || !row_map(&u_map, w.U, d.vdim, slots * d.heads * d.dim, d.vdim, d.dim)) return cudaErrorInvalidValue;
  const dim3 grid(static_cast<unsigned>((max_new + LT_C - 1) / LT_C) * (TD ? vslices : 1), d.heads / hp, n_seqs);
  return launch_kernel(la_states_tc_kernel<TD, ACT>, grid, dim3(LTS_THREADS), smem, st, v_map, u_map, d, w, hp, vslices, poison);
}

template <bool TD, int ACT>
static cudaError_t launch_outputs(const RecDev& d, const LaChunks& w, int hp, int n_seqs, int max_new, long long rows, cudaStream_t st) {
  const int dim16 = (d.dim + 15) & ~15, vslices = (d.vdim + 63) / 64;
  const size_t smem = static_cast<size_t>(2 * ((dim16 + 63) / 64) + 4) * LT_ATOM + static_cast<size_t>(2) * dim16 * 128 + 2 * LT_HALF + sizeof(float) * (12 + 5 * LT_HEADS) * LT_C + 128;
  static std::atomic<unsigned long long> allowed{0};
  cudaError_t e = allow_smem(la_outputs_tc_kernel<TD, ACT>, allowed);
  if (e != cudaSuccess) return e;
  PoisonRef poison = {};
  if (!poison_ref(&poison)) return cudaErrorMemoryAllocation;
  CUtensorMap gate_map, out_map;
  const long long cols = static_cast<long long>(d.heads) * d.vdim;
  if (!row_map(&out_map, d.out, cols, rows, d.ld_out, LT_C) || !row_map(&gate_map, d.gate ? d.gate : d.out, cols, rows, d.gate ? d.ld_gate : d.ld_out, LT_C)) return cudaErrorInvalidValue;
  const dim3 grid(static_cast<unsigned>((max_new + LT_C - 1) / LT_C) * (TD ? vslices : 1), d.heads / hp, n_seqs);
  return launch_kernel(la_outputs_tc_kernel<TD, ACT>, grid, dim3(LT_THREADS), smem, st, gate_map, out_map, d, w, hp, vslices, dim16, poison);
}

#ifdef VY_LA_FIXED   // linear_attn_tc_fixed.cu: decays by head, silu
bool la_fixed_registers() { return la_registers<false, VY_UACT_SILU>(); }
cudaError_t launch_la_states_fixed(const RecDev& d, const LaChunks& w, int hp, int n_seqs, int max_new, long long rows, cudaStream_t st) {
  return launch_states<false, VY_UACT_SILU>(d, w, hp, n_seqs, max_new, rows, st);
}
cudaError_t launch_la_outputs_fixed(const RecDev& d, const LaChunks& w, int hp, int n_seqs, int max_new, long long rows, cudaStream_t st) {
  return launch_outputs<false, VY_UACT_SILU>(d, w, hp, n_seqs, max_new, rows, st);
}
#else
// In place of the 64-token chunks wherever rows come in quads (values and outputs by bulk copies), us of vy_ssd, mma.sync / here, 32 heads of 128 x 64 in groups of 8: one
// prompt of 200 tokens 63 / 42, 512 69 / 45, 2048 250 / 88, 4096 494 / 142; 16 of 150 453 / 142; 32 heads each with q and k of its own, one of 512 78 / 50, 4096 577 / 320;
// 24 heads of 64 x 64 over one q and k, 2048 152 / 64; 8 of 128 x 128 in two groups, 2048 135 / 59.
// Decays by head with silu of q, k and v (vy_linear_attn): 4 x 2048 tokens, 16 heads of 128 x 128 1005 / 415; 129 tokens, 4 heads of 64 x 64 62 / 46; 32 x 256, 16 heads of 64 x 64 499 / 286. Not
// with 32 channels, whose outputs' error would be 1.02 times what it is there (with more it is 0.94 to 1.0), nor without silu: 2 x 1437, 8 heads of 128 x 128 83 / 81, error 1.01
static bool linear_attn_tc_applies(const RecDev& d) {
  const auto quads = [](const void* p, long long ld) { return reinterpret_cast<uintptr_t>(p) % 16 == 0 && ld % 4 == 0; };
  const bool silu = d.in_act == VY_UACT_SILU;
  if (d.dim > 128 || d.vdim < 32 || (d.dt ? d.in_act != VY_UACT_NONE : !silu || d.dim <= 32)) return false;
  if (!(d.dt ? la_registers<true, VY_UACT_NONE>() : la_fixed_registers())) return false;
  return d.out_dt == VY_F32 && quads(d.out, d.ld_out) && (!d.gate || quads(d.gate, d.ld_gate));
}

// A CTA takes about as long before its first head as for two heads (17,000 cycles and 9,500), one CTA per SM at a time. The grid has the longest portion's chunks for every sequence,
// and a CTA without a chunk waits for a whole SM too: with a head per CTA and more than eight such per SM, chunks of 64 are faster. 16 heads of 64 x 64 with q and k of their own, one prompt
// beside single tokens, mma.sync / here, us of vy_ssd: 512 beside 31 129 / 145, 2048 beside 31 230 / 265, 1000 beside 15 108 / 115; 200 beside 31 (three per SM) 89 / 73
int linear_attn_tc_heads(const RecDev& d, int n_seqs, int max_new, long long rows, int vslices) {
  if (!linear_attn_tc_applies(d)) return 0;
  const int rep = d.dt ? d.heads / d.kv_heads : 1, sms = num_sms();
  const long long most = static_cast<long long>(n_seqs) * ((max_new + LT_C - 1) / LT_C), chunks = most < rows / LT_C + n_seqs ? most : rows / LT_C + n_seqs;
  int best = 1;
  long long least = 0;
  for (int hp = 1; hp <= LT_HEADS && hp <= rep; ++hp) {
    if (rep % hp) continue;
    const long long time = (chunks * vslices * (d.heads / hp) + sms - 1) / sms * (hp + 2);
    if (least == 0 || time <= least) {
      least = time;
      best = hp;
    }
  }
  return best == 1 && (most - chunks) * (d.dt ? vslices : 1) * d.heads > 8LL * sms ? 0 : best;
}

cudaError_t launch_la_states_tc(const RecDev& d, const LaChunks& w, int hp, int n_seqs, int max_new, long long rows, cudaStream_t st) {
  return d.dt ? launch_states<true, VY_UACT_NONE>(d, w, hp, n_seqs, max_new, rows, st) : launch_la_states_fixed(d, w, hp, n_seqs, max_new, rows, st);
}
cudaError_t launch_la_outputs_tc(const RecDev& d, const LaChunks& w, int hp, int n_seqs, int max_new, long long rows, cudaStream_t st) {
  return d.dt ? launch_outputs<true, VY_UACT_NONE>(d, w, hp, n_seqs, max_new, rows, st) : launch_la_outputs_fixed(d, w, hp, n_seqs, max_new, rows, st);
}
#endif

}  // namespace vy
