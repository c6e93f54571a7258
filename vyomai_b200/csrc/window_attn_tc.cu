// Prompt-sized windowed attention over pages on tcgen05 (vy_window_attn, long portions, up to 128 channels): the same arithmetic as
// window_attn_mma.cu - fp32 precision from fp16 halves - with scores, weights and weighted values in tensor memory.
//
// A CTA owns 128 rows: 2^hl query heads of one key / value head times 128 / 2^hl queries. Tiles of 64 keys go in turn to two groups of four
// warps (tile t to group t % 2), a thread per row, each group with maxima, sums and outputs (in registers) of its own, which meet at the end: while
// one group turns scores into weights, the tensor pipe works for the other. Per tile
//   scores:  two tiles by one product of 128 columns: small products lo hi + hi lo first, then hi hi onto 2^-11 of them (scale-input-d);
//   weights: a row's 64 scores in registers (final score, maximum, exp, the value row's unit, the split into halves), the halves over the scores
//            (32 columns of hi, 32 of lo);
//   values:  the weights as A out of tensor memory, values as B out of shared memory, the tile's own sum; added to the registers once the group
//            has its next tile's weights. (Sums over all tiles in tensor memory would cut off at every step: see SPLIT_CUT.)
// Split rows come from a workspace (window_attn_split_kernel, second layout) by tensor maps; K and V tiles have rings of their own.
//
// What bounds it: the two softmax groups' own instructions (3400 cycles per pair of tiles with 96 / 64 channels, 4400 with 128 / 128; the products beside them take 2400), and
// 16,000 to 22,000 cycles (8 to 11 us) per CTA before the first and after the last tile. 4 x 2048 tokens, 16 heads of 96 / 64 channels over the whole context: 182 us and 42 for the
// splitting (mma.sync: 545 and 41); 8 heads of 128 over 2, window 512, capped, sloped: 98 and 8 (236 and 8); sigmoid weights 97 and 8 (237 and 8).
// Tried: 128-key tiles with one buffer of scores per group 284 us, the same with two threads per row 250 (of the first); 64-key scores alone per product 185.
#include "seqmix.cuh"
#include "split_mma.cuh"
#include "vy_ptx.cuh"

namespace vy {

constexpr int TC_ROWS = 128;   // rows of a CTA
constexpr int TC_KEYS = 64;    // keys of a tile; scores come two tiles at a time (with 64 columns a product reads 192 bytes of shared memory a cycle that it has not)
constexpr int TC_ATOM2 = TC_ROWS * 128, TC_ATOM = TC_KEYS * 128;   // 64 fp16 entries of each of 128 queries or keys, of 64 values; 128-byte swizzle
constexpr int TC_BUFS = 4;     // tiles whose scores or weights are in tensor memory
constexpr int TC_STAGES = 4;   // tiles of values, or pairs of tiles of keys, in shared memory, at most
constexpr int TC_THREADS = 384;   // four warps: 0 copies of keys, 1 products, 2 tensor memory, 3 copies of values; then the two softmax groups
constexpr int TC_REGS = 168, TC_REGS_SOFTMAX = 232, TC_REGS_REST = 40;   // a thread: at launch, and as three groups of four warps share them out: 2 x 232 + 40 = 3 x 168

struct TcGeo {
  int hl, dim16, vdim16, nks;   // nks: steps of 16 channels
  int k_atoms, v_atoms;   // of a pair of tiles: K hi | K lo together; of a tile: V hi and V lo
  int ks, vs;   // stages of the two rings
  int qvec, ovec;
  // where the halves of channels 16 k .. lie, in 16 bytes from the start of the queries or of a pair of key tiles
  unsigned short hi[8], lo[8];
};

// VD: value channels the registers hold (64 | 128)
template <int VD, bool SIG>
__global__ void __launch_bounds__(TC_THREADS, 1)
window_attn_tc_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ WinDev d, const __grid_constant__ SplitKv w, const __grid_constant__ TcGeo geo,
                      const __grid_constant__ PoisonRef poison) {
  pdl_trigger();
  extern __shared__ __align__(1024) unsigned char tc_smem[];
  const int k_bytes = geo.k_atoms * TC_ATOM2, v_bytes = geo.v_atoms * TC_ATOM;
  unsigned char* Qs = tc_smem;   // the keys' layout
  unsigned char* Ks = Qs + k_bytes;   // [stages]
  unsigned char* Vs = Ks + geo.ks * k_bytes;   // [stages]
  float* units = reinterpret_cast<float*>(Vs + geo.vs * v_bytes);   // [group][turn of three][K | V][key]
  float* qe = units + 2 * 3 * 2 * TC_KEYS;
  uint64_t* bars = reinterpret_cast<uint64_t*>(qe + TC_ROWS);
  uint64_t *kfull = bars, *kempty = kfull + TC_STAGES, *vfull = kempty + TC_STAGES, *vempty = vfull + TC_STAGES;
  uint64_t *sfull = vempty + TC_STAGES, *pfull = sfull + 2, *ofull = pfull + TC_BUFS, *done = ofull + 2;
  int* kissued = reinterpret_cast<int*>(done + 1);   // copies sent for, per buffer
  int* vissued = kissued + TC_STAGES;
  uint32_t* tmem_at = reinterpret_cast<uint32_t*>(vissued + TC_STAGES);
  float* about = reinterpret_cast<float*>(tmem_at + 1);   // of the list: its keys' largest entry, whether it is not for fp16 halves; the values' largest entry that the CTA sees
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int hl = geo.hl, hm = (1 << hl) - 1, qn = TC_ROWS >> hl;
  if (warp == 1 && lane == 0) {
    for (int i = 0; i < TC_STAGES; ++i) {
      mbar_init(&kfull[i], 1);
      mbar_init(&kempty[i], 1);
      mbar_init(&vfull[i], 1);
      mbar_init(&vempty[i], 1);
      kissued[i] = vissued[i] = 0;
    }
    for (int i = 0; i < TC_BUFS; ++i) mbar_init(&pfull[i], 4);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sfull[i], 1);
      mbar_init(&ofull[i], 1);
    }
    mbar_init(done, 1);
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) tma_prefetch_desc(&map);
  __syncthreads();
  pdl_wait();
  const int s = blockIdx.y, h0 = blockIdx.x << hl, g = h0 / (d.heads / d.kv_heads), sg = s * d.kv_heads + g;
  const int base = d.cu[s], n = d.cu[s + 1] - base;
  const int blk = (n + qn - 1) / qn - 1 - static_cast<int>(blockIdx.z);   // the last queries see the most keys: they go first, those of all heads and sequences
  if (blk < 0) return;
  if (warp == 2) {
    tmem_alloc(tmem_at, 512);
    tmem_relinquish();
  }
  const int i0 = blk * qn, nq = min(qn, n - i0);
  const int p0 = d.pos0[s], p_lo = p0 + i0, p_hi = p_lo + nq - 1;
  // visible keys of the CTA's queries: [0, nA) (kept first tokens outside the band) and [lo, p_hi]; tiles of the one, then of the other
  int nA, lo, nA0, lo0;
  portion_keys(d, p_lo, nA, lo);
  portion_keys(d, p0, nA0, lo0);   // where the workspace keeps a key
  const int keep_tiles = (nA + TC_KEYS - 1) / TC_KEYS, tiles = keep_tiles + (p_hi - lo + TC_KEYS) / TC_KEYS;
  const int band0 = nA0 + lo - lo0;   // slot of the band's first key
  const auto slot_of = [&](int t) { return t < keep_tiles ? t * TC_KEYS : band0 + (t - keep_tiles) * TC_KEYS; };
  const long long list0 = static_cast<long long>(sg) * w.cap;
  const int pairs = (tiles + 1) / 2;   // the last one's second tile may lie past the keys: rows of zeros, scores nobody reads
  const auto load_k = [&](int k, int b) {   // by one elected lane
    ++kissued[b];
    mbar_arrive_expect_tx(&kfull[b], k_bytes);
    for (int a = 0; a < geo.k_atoms; ++a)
      for (int i = 0; i < 2; ++i) tma_load_2d(Ks + b * k_bytes + a * TC_ATOM2 + i * TC_ATOM, &map, &kfull[b], 64 * a, static_cast<int>(list0) + slot_of(2 * k + i));
  };
  const auto load_v = [&](int t, int b) {
    ++vissued[b];
    mbar_arrive_expect_tx(&vfull[b], v_bytes);
    for (int a = 0; a < geo.v_atoms; ++a) tma_load_2d(Vs + b * v_bytes + a * TC_ATOM, &map, &vfull[b], (w.v_at >> 1) + 64 * a, static_cast<int>(list0) + slot_of(t));
  };
  if (warp == 0) {
    if (elect_one_sync()) {
      for (int k = 0; k < min(geo.ks, pairs); ++k) load_k(k, k);
      for (int t = 0; t < min(geo.vs, tiles); ++t) load_v(t, t);
    }
    __syncwarp();
  }
  if (warp == 3) {
    float top_k;
    const bool odd = split_odd(w, sg, nA0 + p0 + n - lo0, top_k);
    unsigned tv = 0u;
    for (int x = lane; x < (nA0 + p0 + n - lo0 + SPLIT_ROWS - 1) / SPLIT_ROWS; x += 32)
      if (x * SPLIT_ROWS < nA || ((x + 1) * SPLIT_ROWS > band0 && x * SPLIT_ROWS <= band0 + p_hi - lo)) tv = max(tv, w.range[static_cast<long long>(sg) * w.blocks + x].y);
    tv = __reduce_max_sync(0xffffffffu, tv);
    if (lane == 0) {
      about[0] = top_k;
      about[1] = odd ? 1.f : 0.f;
      about[2] = __uint_as_float(tv);
    }
  }
  // queries: rows [hi | lo] as the keys', swizzled. Eight lanes share a row, the next row's entries are on their way while one is split: a short loop,
  // since code that a CTA runs once comes cold (unrolled over four rows it took as long)
  if (warp >= 4) {
    const int l8 = lane & 7, r_0 = (warp - 4) * 4 + (lane >> 3);
    float4 next[4];
    const auto fetch = [&](int r) {
      const bool there = r < TC_ROWS && (r >> hl) < nq;
      const long long at = static_cast<long long>(base + i0 + (r >> hl)) * d.ldq + static_cast<long long>(h0 + (r & hm)) * d.dim;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = l8 * 4 + 32 * i;
        next[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (there && c < d.dim) next[i] = geo.qvec ? *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(d.q) + at + c) : load4_any(d.q, d.q_dt, at, c, d.dim);
      }
    };
    fetch(r_0);
#pragma unroll 1
    for (int r = r_0; r < TC_ROWS; r += 32) {
      float4 x[4];
      float top = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[i] = next[i];
        top = fmaxf(top, fmaxf(fmaxf(fabsf(x[i].x), fabsf(x[i].y)), fmaxf(fabsf(x[i].z), fabsf(x[i].w))));
      }
      fetch(r + 32);
#pragma unroll
      for (int k = 1; k < 8; k <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, k));
      const int e = split_exponent(top);
      const float sc = split_scale(e);
      if (l8 == 0) qe[r] = pow2i(e - SPLIT_TOP);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = l8 * 4 + 32 * i;
        if (c < geo.dim16) {
          uint2 hi, lo_;
          split2(x[i].x * sc, x[i].y * sc, hi.x, lo_.x);
          split2(x[i].z * sc, x[i].w * sc, hi.y, lo_.y);
          const auto put = [&](int at, uint2 v) { *reinterpret_cast<uint2*>(Qs + (at >> 6) * TC_ATOM2 + r * 128 + (((at & 63) * 2) ^ ((r & 7) << 4))) = v; };
          put(c, hi);
          put(geo.dim16 + c, lo_);
        }
      }
    }
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();   // Q and its units are there, and the address of the tensor memory
  tc_fence_after();
  const uint32_t tmem = *tmem_at, tmem_o = tmem + TC_BUFS * TC_KEYS;
  const int row = threadIdx.x & (TC_ROWS - 1), h = h0 + (row & hm);
  const float qmul = head_scale_of(d, h) * qe[row];
  if (__syncthreads_or(about[1] != 0.f || !(fabsf(qmul) * about[0] <= SPLIT_SCORE))) {   // not for fp16 halves: the fp32 form's
    if (warp == 0) {
      mbar_drain(kfull, kissued, TC_STAGES);   // the copies in flight write to this CTA's memory
      mbar_drain(vfull, vissued, TC_STAGES);
      if (lane == 0) w.odd[sg] = 1;
    }
    __syncthreads();
    if (warp == 2) tmem_dealloc(tmem, 512);
    return;
  }
  bool alive = true;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(TC_REGS_REST));
    if (warp == 0 || warp == 3) {
      // ---- copies: keys by one warp, values by another (scores run up to four tiles ahead of the weighted values) ----
      uint64_t* empty = warp == 0 ? kempty : vempty;
      const int stages = warp == 0 ? geo.ks : geo.vs, end = warp == 0 ? pairs : tiles;
      int b = 0, ph = 0;
      for (int t = stages; t < end && alive; ++t) {
        alive = mbar_wait_soft(&empty[b], ph, poison);
        if (alive && elect_one_sync()) {
          if (warp == 0) load_k(t, b);
          else load_v(t, b);
        }
        __syncwarp();
        if (++b == stages) {
          b = 0;
          ph ^= 1;
        }
      }
    } else if (warp == 1) {
      // ---- products. The issue loops are kept short: descriptors are a base plus offsets out of the arguments ----
      constexpr uint32_t id_s = make_idesc(0, TC_ROWS, 2 * TC_KEYS, 0, 0);
      const uint32_t id_o = make_idesc(0, TC_ROWS, 0, 0, 1) | static_cast<uint32_t>(geo.vdim16 >> 3) << 17;
      const uint64_t kd = make_smem_desc_sw128(0, 16, 1024), vd = make_smem_desc_sw128(0, TC_ATOM, 1024);
      const uint32_t khi = static_cast<uint32_t>(kd >> 32), klo = static_cast<uint32_t>(kd), vhi = static_cast<uint32_t>(vd >> 32), vlo = static_cast<uint32_t>(vd);
      const auto desc = [](uint32_t hi, uint32_t lo_) { return static_cast<uint64_t>(hi) << 32 | lo_; };
      const uint32_t q_at = klo + (smem_u32(Qs) >> 4), v_small = static_cast<uint32_t>(geo.v_atoms / 2) * (TC_ATOM >> 4);
      const int nks = geo.nks;
      int kb = 0, kph = 0, vb = 0, vph = 0;
      const auto scores = [&](int k2) {   // of pair k2
        alive = mbar_wait_soft(&kfull[kb], kph, poison) && alive;
        tc_fence_after();
        if (alive && elect_one_sync()) {
          const uint32_t k_at = klo + (smem_u32(Ks + kb * k_bytes) >> 4), D = tmem + (k2 & 1) * 2 * TC_KEYS;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k < nks) umma_f16(D, desc(khi, q_at + geo.lo[k]), desc(khi, k_at + geo.hi[k]), id_s, k != 0);
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k < nks) umma_f16(D, desc(khi, q_at + geo.hi[k]), desc(khi, k_at + geo.lo[k]), id_s, 1);
          umma_f16_shift11(D, desc(khi, q_at), desc(khi, k_at), id_s);
#pragma unroll
          for (int k = 1; k < 8; ++k)
            if (k < nks) umma_f16(D, desc(khi, q_at + geo.hi[k]), desc(khi, k_at + geo.hi[k]), id_s, 1);
          umma_commit(&kempty[kb]);
          umma_commit(&sfull[k2 & 1]);
        }
        __syncwarp();
        if (++kb == geo.ks) {
          kb = 0;
          kph ^= 1;
        }
      };
      const auto values = [&](int t) {
        alive = mbar_wait_soft(&vfull[vb], vph, poison) && alive;
        alive = mbar_wait_soft(&pfull[t % TC_BUFS], (t / TC_BUFS) & 1, poison) && alive;
        tc_fence_after();
        if (alive && elect_one_sync()) {
          const uint32_t v_at = vlo + (smem_u32(Vs + vb * v_bytes) >> 4), D = tmem_o + (t & 1) * VD, P = tmem + (t % TC_BUFS) * TC_KEYS;
          // weights of keys 16 k ..: 8 columns of hi, 32 columns on 8 of lo
#pragma unroll
          for (int k = 0; k < TC_KEYS / 16; ++k) umma_f16_ta(D, P + 32 + 8 * k, desc(vhi, v_at + k * 128), id_o, k != 0);
#pragma unroll
          for (int k = 0; k < TC_KEYS / 16; ++k) umma_f16_ta(D, P + 8 * k, desc(vhi, v_at + v_small + k * 128), id_o, 1);
          umma_f16_ta_shift11(D, P, desc(vhi, v_at), id_o);
#pragma unroll
          for (int k = 1; k < TC_KEYS / 16; ++k) umma_f16_ta(D, P + 8 * k, desc(vhi, v_at + k * 128), id_o, 1);
          umma_commit(&vempty[vb]);
          umma_commit(&ofull[t & 1]);
        }
        __syncwarp();
        if (++vb == geo.vs) {
          vb = 0;
          vph ^= 1;
        }
      };
      scores(0);
      if (pairs > 1) scores(1);
      for (int k2 = 0; k2 < pairs; ++k2) {
        values(2 * k2);
        if (2 * k2 + 1 < tiles) values(2 * k2 + 1);
        if (k2 + 2 < pairs) scores(k2 + 2);   // over the weights that the products before it read: the pipe keeps the order
      }
    }
    __syncwarp();
  } else {
    // ---- softmax: thread <-> row ----
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(TC_REGS_SOFTMAX));
    const int grp = (warp >> 2) - 1;
    const uint32_t quarter = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t O = tmem_o + quarter + grp * VD;
    const int p = p_lo + (row >> hl);
    // scores are kept as exponents of 2: q k scale log2(e), its factor in two parts so that it is as good as fp32 arithmetic in units of e
    constexpr float L2E = 1.4426950408889634f, L2E_LO = static_cast<float>(1.4426950408889634 - static_cast<double>(L2E));
    const float to2 = d.softcap > 0.f ? 2.f * L2E / d.softcap : L2E, q1 = qmul * to2, q2 = d.softcap > 0.f ? fmaf(qmul, to2, -q1) : fmaf(qmul, L2E_LO, fmaf(qmul, L2E, -q1));
    const f32x2 qhi = pair(q1), qlo = pair(q2), badd = pair(head_bias_of(d, h) * to2);
    const float slope = -head_slope_of(d, h) * L2E;
    float m = d.sink && grp == 0 ? ld_as_float(d.sink, d.sink_dt, h) * L2E : -INFINITY, l = d.sink && grp == 0 ? 1.f : 0.f;
    // outputs in units of 2^(E - 2 SPLIT_TOP), E the exponent of the largest value that the CTA sees
    const int E = split_exponent(about[2]);
    const float v_unit = pow2i(SPLIT_TOP - E);
    f32x2 o[VD / 2];
#pragma unroll
    for (int i = 0; i < VD / 2; ++i) o[i] = pair(0.f);
    const auto take_o = [&]() {   // the group's last weighted values
      const f32x2 cut = pair(0.5f * (TC_KEYS / 16 + 1) * 0x1p-25f);   // SPLIT_CUT, of a sum of TC_KEYS / 16 accumulations
#pragma unroll
      for (int c = 0; c < VD; c += 32) {
        uint32_t raw[32];
        tmem_ld_x32(O + c, raw);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const f32x2 v = pair_bits(raw[i], raw[i + 1]);
          o[(c + i) / 2] = add2(o[(c + i) / 2], fma2(v, cut, v));
        }
      }
    };
    // the tiles' units: thread i brings those of key i % 64, of K or of V, a tile ahead into the next of three buffers
    const float* unit0 = w.unit + 2 * (list0 + (row & (TC_KEYS - 1))) + (row >> 6);
    float* my_unit = units + grp * 3 * 2 * TC_KEYS + row;
    const auto get_unit = [&](int t) { return t < tiles ? unit0[2 * slot_of(t)] : 0.f; };
    const float my_scale = row >> 6 ? v_unit : 1.f;
    if (grp < tiles) *my_unit = get_unit(grp) * my_scale;
    float unit = get_unit(grp + 2);
    int turn = 0;
    for (int t = grp; t < tiles; t += 2) {
      const int buf = t % TC_BUFS, next = turn == 2 ? 0 : turn + 1;
      named_bar_sync(1 + grp, TC_ROWS);   // this tile's units; nobody reads the next buffer any more
      my_unit[next * 2 * TC_KEYS] = unit * my_scale;
      unit = get_unit(t + 4);
      const float* ku = units + (grp * 3 + turn) * 2 * TC_KEYS;
      const float* vu = ku + TC_KEYS;
      turn = next;
      const int f = t < keep_tiles ? t * TC_KEYS : lo + (t - keep_tiles) * TC_KEYS;   // position of the tile's first key
      const int nk = t < keep_tiles ? nA - f : p_hi + 1 - f;   // its keys, if fewer than a tile's
      const bool whole = t >= keep_tiles && f + TC_KEYS - 1 <= p_lo && (d.window <= 0 || p_hi - f < d.window) && (d.chunk <= 0 || f >= p_hi / d.chunk * d.chunk);
      if (t == 1) named_bar_sync(4, 2 * TC_ROWS);   // the groups start a phase apart: exponentials of one beside the other's sums (3400 cycles a pair of tiles instead of 3850)
      alive = mbar_wait_soft(&sfull[(t >> 1) & 1], (t / TC_BUFS) & 1, poison) && alive;
      tc_fence_after();
      const uint32_t S = tmem + quarter + buf * TC_KEYS;
      f32x2 x[TC_KEYS / 2];
      {
        uint32_t r0[32], r1[32];
        tmem_ld_x32(S, r0);
        tmem_ld_x32(S + 32, r1);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          x[i] = pair_bits(r0[2 * i], r0[2 * i + 1]);
          x[16 + i] = pair_bits(r1[2 * i], r1[2 * i + 1]);
        }
      }
#pragma unroll
      for (int i = 0; i < TC_KEYS / 2; i += 2) {
        const ulonglong2 kx = *reinterpret_cast<const ulonglong2*>(ku + 2 * i);
        const f32x2 y0 = mul2(x[i], kx.x), y1 = mul2(x[i + 1], kx.y);
        x[i] = fma2(y0, qhi, fma2(y0, qlo, badd));
        x[i + 1] = fma2(y1, qhi, fma2(y1, qlo, badd));
      }
      if (d.softcap > 0.f) {   // cap tanh(s / cap) = cap - 2 cap / (1 + e^(2 s / cap)); an overflow gives cap, an underflow -cap
        const f32x2 cap = pair(d.softcap * L2E), cap2 = pair(-2.f * d.softcap * L2E), one = pair(1.f);
#pragma unroll
        for (int i = 0; i < TC_KEYS / 2; ++i) {
          const float2 e = unpair(x[i]);
          const float2 y = unpair(add2(pair(vy_ex2_approx(e.x), vy_ex2_approx(e.y)), one));
          x[i] = fma2(cap2, pair(vy_rcp_approx(y.x), vy_rcp_approx(y.y)), cap);
        }
      }
      if (d.head_slope) {
        const f32x2 away = pair(static_cast<float>(p - f)), sl = pair(slope);
#pragma unroll
        for (int i = 0; i < TC_KEYS / 2; ++i) x[i] = fma2(sl, add2(away, pair(-2.f * i, -2.f * i - 1.f)), x[i]);
      }
      if (!whole) {   // the row's visible keys of the tile: [jlo, jhi) and [0, jkeep)
        const int jhi = min(nk, p - f + 1), jlo = d.chunk > 0 ? p / d.chunk * d.chunk - f : d.window > 0 ? p - d.window + 1 - f : 0, jkeep = d.window > 0 ? d.keep - f : 0;
        const auto below = [](int j) { return j <= 0 ? 0u : j >= 32 ? 0xffffffffu : (1u << j) - 1u; };   // bits of the keys before j
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const unsigned vis = below(jhi - 32 * q) & (~below(jlo - 32 * q) | below(jkeep - 32 * q));
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 e = unpair(x[16 * q + i]);
            x[16 * q + i] = pair(vis >> (2 * i) & 1u ? e.x : -INFINITY, vis >> (2 * i + 1) & 1u ? e.y : -INFINITY);
          }
        }
      }
      float cr = 1.f;
      if constexpr (!SIG) {
        float top[4] = {m, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < TC_KEYS / 2; ++i) {
          const float2 e = unpair(x[i]);
          top[i & 3] = fmaxf(top[i & 3], fmaxf(e.x, e.y));
        }
        const float mn = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
        cr = mn == -INFINITY ? 1.f : vy_ex2_approx(m - mn);
        m = mn;
      }
      const f32x2 mm = pair(m == -INFINITY ? 0.f : -m);   // 2^(-inf - 0) = 0 where nothing is visible yet
      f32x2 sum[2] = {pair(0.f), pair(0.f)};
#pragma unroll
      for (int q = 0; q < 2; ++q) {   // 32 keys: 16 columns of hi, 16 of lo, over the scores
        uint32_t hi[16], lo_[16];
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          const ulonglong2 vx = *reinterpret_cast<const ulonglong2*>(vu + 32 * q + 2 * i);
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            f32x2 e = x[16 * q + i + k];
            if constexpr (SIG) {
              const float2 z = unpair(e);
              const float2 y = unpair(add2(pair(vy_ex2_approx(-z.x), vy_ex2_approx(-z.y)), pair(1.f)));
              e = pair(vy_rcp_approx(y.x), vy_rcp_approx(y.y));   // of -inf: 0
            } else {
              const float2 z = unpair(add2(e, mm));
              e = pair(vy_ex2_approx(z.x), vy_ex2_approx(z.y));
              sum[k] = add2(sum[k], e);
            }
            const f32x2 y = mul2(e, k ? vx.y : vx.x);
            const float2 yf = unpair(y);
            const __half2 hv = __floats2half2_rn(yf.x, yf.y);
            const float2 hf = __half22float2(hv);
            const float2 lf = unpair(fma2(pair(hf.x, hf.y), pair(-1.f / LO_UNIT), mul2(y, pair(1.f / LO_UNIT))));
            hi[i + k] = pack_h2(hv);
            lo_[i + k] = pack_h2(__floats2half2_rn(lf.x, lf.y));
          }
        }
        tmem_st_x16(S + 16 * q, hi);
        tmem_st_x16(S + 32 + 16 * q, lo_);
      }
      if (t == 0 && tiles > 1) asm volatile("bar.arrive 4, %0;" ::"n"(2 * TC_ROWS) : "memory");
      if (t != grp) {
        alive = mbar_wait_soft(&ofull[grp], ((t >> 1) - 1) & 1, poison) && alive;
        tc_fence_after();
        take_o();
      }
      if constexpr (!SIG) {
        const float2 a = unpair(add2(sum[0], sum[1]));
        l = fmaf(l, cr, a.x + a.y);
        if (__any_sync(0xffffffffu, cr != 1.f)) {
#pragma unroll
          for (int i = 0; i < VD / 2; ++i) o[i] = mul2(o[i], pair(cr));
        }
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&pfull[buf]);
    }
    if (grp < tiles) {   // the group's last weighted values
      alive = mbar_wait_soft(&ofull[grp], ((tiles - 1 - grp) >> 1) & 1, poison) && alive;
      tc_fence_after();
      take_o();
    }
    // ---- the two groups meet: each hands the other its maximum, its sum and half of its output columns, through the rings' memory once neither's
    // products read it any more, and finishes the other half ----
    float* xo = reinterpret_cast<float*>(Ks);   // [group][m, l, columns][row]
    const auto at = [&](int who, int what) -> float& { return xo[(who * (2 + VD / 2) + what) * TC_ROWS + row]; };
    named_bar_sync(3, 2 * TC_ROWS);
    at(grp, 0) = m;
    at(grp, 1) = l;
#pragma unroll
    for (int i = 0; i < VD / 4; ++i) {
      const float2 y = unpair(grp == 0 ? o[VD / 4 + i] : o[i]);
      at(grp, 2 + 2 * i) = y.x;
      at(grp, 3 + 2 * i) = y.y;
    }
    named_bar_sync(3, 2 * TC_ROWS);
    const int i = row >> hl;
    if (i < nq) {
      float a0 = 1.f, a1 = 1.f, og = d.out_scale;   // shares of the own and of the other's outputs
      if constexpr (!SIG) {
        const float m1 = at(grp ^ 1, 0), mx = fmaxf(m, m1);
        a0 = m == -INFINITY ? 0.f : vy_ex2_approx(m - mx);
        a1 = m1 == -INFINITY ? 0.f : vy_ex2_approx(m1 - mx);
        og /= l * a0 + at(grp ^ 1, 1) * a1;
      }
      const long long qrow = base + i0 + i;
      if (d.gate) og *= sigmoidf_(ld_as_float(d.gate, d.gate_dt, qrow * d.ld_gate + h));
      const float un = pow2i(E - 2 * SPLIT_TOP);
      const long long ob = qrow * d.ld_out + static_cast<long long>(h) * d.vdim;
#pragma unroll
      for (int j = 0; j < VD / 2; j += 8) {
        const int c = grp * (VD / 2) + j;
        float y[8];
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          const float2 own = unpair(grp == 0 ? o[(j + k) / 2] : o[VD / 4 + (j + k) / 2]);
          y[k] = (own.x * a0 + at(grp ^ 1, 2 + j + k) * a1) * un * og;
          y[k + 1] = (own.y * a0 + at(grp ^ 1, 3 + j + k) * a1) * un * og;
        }
        if (geo.ovec && c + 8 <= d.vdim) st8_from_float(d.out, d.out_dt, ob + c, y);
        else
          for (int k = 0; k < 8; k += 2) store2_any(d.out, d.out_dt, ob + c + k, y[k], y[k + 1], d.vdim - c - k);
      }
    }
  }
  tc_fence_before();
  if (__syncthreads_or(!alive)) {   // a wait has timed out: what is still in flight ends before the memory is given back
    if (warp == 0) {
      mbar_drain(kfull, kissued, TC_STAGES);
      mbar_drain(vfull, vissued, TC_STAGES);
    } else if (warp == 1) {
      if (elect_one_sync()) umma_commit(done);
      __syncwarp();
      for (uint32_t spins = 0; spins < (1u << 20) && !mbar_try_wait(done, 0); ++spins) {}
    }
  }
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

static int round_to(int n, int m) { return (n + m - 1) / m * m; }

// heads per tile: the largest power of two, at most 16, that divides the heads of a key / value head
static int tc_head_bits(const WinDev& d) {
  const int rep = d.heads / d.kv_heads;
  int hl = 0;
  while (hl < 4 && rep % (2 << hl) == 0) ++hl;
  return hl;
}

SplitKv window_attn_tc_layout(const WinDev& d, int n_seqs, int max_new, float* ws) {
  const int dim16 = round_to(d.dim, 16), kd = round_to(2 * dim16, 64), vd = round_to(d.vdim, 64);
  SplitKv w = {};
  w.tail = 2 * TC_KEYS;
  w.cap = split_slots(d, max_new) + w.tail;
  w.row_bytes = 2 * kd + 4 * vd;
  w.k_lo = 2 * dim16;
  w.v_at = 2 * kd;
  w.v_lo = 2 * vd;
  w.vpad = vd;
  w.ustep = 2;
  w.blocks = static_cast<int>((w.cap + SPLIT_ROWS - 1) / SPLIT_ROWS);
  const long long lists = static_cast<long long>(n_seqs) * d.kv_heads;
  w.rows = reinterpret_cast<unsigned char*>(ws);
  w.range = reinterpret_cast<uint4*>(w.rows + lists * w.cap * w.row_bytes);
  w.odd = reinterpret_cast<int*>(w.range + lists * w.blocks);
  w.unit = reinterpret_cast<float*>(w.odd + (lists + 3) / 4 * 4);
  return w;
}

long long window_attn_tc_floats(const WinDev& d, int n_seqs, int max_new) {
  if (d.dim > 128 || d.vdim > 128) return 0;
  const SplitKv w = window_attn_tc_layout(d, 1, max_new, nullptr);
  return static_cast<long long>(n_seqs) * d.kv_heads * (w.cap * (w.row_bytes / 4 + 2) + 4LL * w.blocks + 4);
}

// with fewer registers at launch than the warps share out, the first to ask for more would wait for ever: what a compiler gives another number does without this form
template <int VD, bool SIG>
static bool tc_registers() {
  static const bool enough = [] {
    cudaFuncAttributes a;
    return cudaFuncGetAttributes(&a, window_attn_tc_kernel<VD, SIG>) == cudaSuccess && (a.numRegs + 7) / 8 * 8 == TC_REGS;
  }();
  return enough;
}

// Is this form faster than window_attn_mma.cu's? Microseconds of either, from the CTAs that find rows and those that find none (the grid has the longest portion's for every
// sequence) and the keys a block of rows sees. Here a CTA has an SM to itself, its fixed time is that of some ten tiles, and a CTA without rows waits for a whole SM too: a prompt
// beside many single tokens is as slow as its rounds of CTAs. Fitted to batches of 2 to 32 heads of 16 to 128 channels with both forms timed; of 1353 it takes the one slower by more
// than 4 % in 11 (by 27 % at most). mma.sync / tcgen05, us, splitting included: 4 x 2048 tokens, 16 heads of 96 / 64, whole context 590 / 231; 16 portions of 130, 8 heads of 128 over 2, window 64 28 / 35
// (160 CTAs: two rounds); one of 512 beside 31 single tokens, window 64, 16 heads of 96 / 64 51 / 85, 12 of 64 39 / 61, window 512, 8 of 128 over 2 93 / 46
static bool tc_pays(const WinDev& d, int n_seqs, int max_new, int hl) {
  const double sms = num_sms(), channels = (round_to(d.dim, 16) + round_to(d.vdim, 16)) / 128.0;
  const long long all = static_cast<long long>(d.tw) * d.bs, blocks_of_heads = d.heads >> hl;
  const long long band = d.chunk > 0 ? d.chunk : static_cast<long long>(d.window) + d.keep, seen = band + (TC_ROWS >> hl);
  const double tiles = (d.chunk > 0 || d.window > 0 ? static_cast<double>(seen < all ? seen : all) : 0.6 * all) / TC_KEYS;
  const auto ctas = [&](int qn, double& idle) {   // that find rows, at most
    const long long grid = static_cast<long long>(n_seqs) * ((max_new + qn - 1) / qn), most = d.rows / qn + n_seqs, live = grid < most ? grid : most;
    idle = static_cast<double>(blocks_of_heads * (grid - live));
    return static_cast<double>(blocks_of_heads * live);
  };
  double idle_tc, idle_mma;
  const double live_tc = ctas(TC_ROWS >> hl, idle_tc), live_mma = ctas(64 >> hl, idle_mma), rounds = ceil(live_tc / sms) + (idle_tc > sms ? 0.4 : 0.0);
  const double tc = rounds * (d.vdim > 64 ? 13.0 : 10.5) + rounds * (0.1 + 0.15 * channels) * tiles + 0.75 * idle_tc / sms;
  const double mma = fmax(1.0, live_mma / (2.0 * sms)) * (13.0 + (0.5 + 3.0 * channels) * tiles) + 0.1 * idle_mma / (2.0 * sms);
  return tc <= mma;
}

bool window_attn_tc_applies(const WinDev& d, int n_seqs, int max_new) {
  if (d.dim > 128 || d.vdim > 128) return false;
  if (!(d.vdim > 64 ? (d.sigmoid ? tc_registers<128, true>() : tc_registers<128, false>()) : d.sigmoid ? tc_registers<64, true>() : tc_registers<64, false>())) return false;
  // tensor-map rows are counted in 32 bits
  if (static_cast<long long>(n_seqs) * d.kv_heads * (split_slots(d, max_new) + 2 * TC_KEYS) > 0x7fffffffLL - 2 * TC_KEYS) return false;
  const int hl = tc_head_bits(d);
  const long long rows = static_cast<long long>(max_new) << hl;
  if (rows < TC_ROWS || rows / TC_ROWS >= 65535) return false;   // the last: a grid's limit
  // A CTA takes 8 to 11 us before its first tile and after its last; with a tile or two between them the 64-row CTAs of window_attn_mma.cu are as good.
  // Splitting and attention, mma.sync / tcgen05, four portions of n tokens from position 0, 8 heads of 128 over 2: n = 128 25.0 / 22.6 us, 300 41.5 / 26.8;
  // 16 heads of 96 / 64 with keys of their own: 128 22.5 / 22.6, 300 45.5 / 35.3, 1000 200 / 101. Portions of 32 tokens on 2000 cached
  // ones, 8 heads over 2, window 512: 57 / 31
  return split_slots(d, max_new) >= (hl > 0 ? 128 : 192) && tc_pays(d, n_seqs, max_new, hl);
}

template <int VD, bool SIG>
static cudaError_t launch_tc(const CUtensorMap& map, const WinDev& d, const SplitKv& w, TcGeo geo, const dim3& grid, cudaStream_t st) {
  const size_t kt = static_cast<size_t>(geo.k_atoms) * TC_ATOM2, vt = static_cast<size_t>(geo.v_atoms) * TC_ATOM, rest = kt + sizeof(float) * (12 * TC_KEYS + TC_ROWS) + 512;
  const auto total = [&] { return rest + geo.ks * kt + geo.vs * vt; };
  geo.ks = 2;
  geo.vs = TC_STAGES;
  while (total() > 232448 && geo.vs > 2) --geo.vs;
  while (total() > 232448 && geo.ks > 1) --geo.ks;
  while (geo.vs < TC_STAGES && total() + vt <= 232448) ++geo.vs;
  static std::atomic<unsigned long long> allowed{0};
  cudaError_t e = allow_smem(window_attn_tc_kernel<VD, SIG>, allowed);
  if (e != cudaSuccess) return e;
  PoisonRef poison = {};
  if (!poison_ref(&poison)) return cudaErrorMemoryAllocation;
  return launch_kernel(window_attn_tc_kernel<VD, SIG>, grid, dim3(TC_THREADS), total(), st, map, d, w, geo, poison);
}

cudaError_t launch_window_attn_tc(const WinDev& d, int n_seqs, int max_new, float* ws, const int** odd, cudaStream_t st) {
  const SplitKv w = window_attn_tc_layout(d, n_seqs, max_new, ws);
  *odd = w.odd;
  cudaError_t e = launch_split_rows(d, n_seqs, w, st);
  if (e != cudaSuccess) return e;
  const uint64_t dims[2] = {static_cast<uint64_t>(w.row_bytes / 2), static_cast<uint64_t>(n_seqs) * d.kv_heads * w.cap}, strides[2] = {0, static_cast<uint64_t>(w.row_bytes)};
  const uint32_t box[2] = {64, TC_KEYS};
  CUtensorMap map;
  if (get_tensor_map_cached(&map, VY_BF16, 2, ws, dims, strides, box, 1) != VY_OK) return cudaErrorInvalidValue;   // 16-bit entries of either kind
  const auto al = [](const void* p, int a) { return reinterpret_cast<uintptr_t>(p) % a == 0; };
  TcGeo geo = {};
  geo.hl = tc_head_bits(d);
  geo.dim16 = round_to(d.dim, 16);
  geo.vdim16 = round_to(d.vdim, 16);
  geo.nks = geo.dim16 / 16;
  for (int k = 0; k < geo.nks; ++k) {
    const auto at = [](int e) { return static_cast<unsigned short>((e / 64 * TC_ATOM2 + e % 64 * 2) / 16); };
    geo.hi[k] = at(16 * k);
    geo.lo[k] = at(geo.dim16 + 16 * k);
  }
  geo.k_atoms = round_to(2 * geo.dim16, 64) / 64;
  geo.v_atoms = 2 * (round_to(d.vdim, 64) / 64);
  geo.qvec = d.q_dt == VY_F32 && d.dim % 4 == 0 && d.ldq % 4 == 0 && al(d.q, 16);
  geo.ovec = d.vdim % 8 == 0 && d.ld_out % 8 == 0 && al(d.out, 16);
  const int qn = TC_ROWS >> geo.hl;
  const dim3 grid(d.heads >> geo.hl, n_seqs, (max_new + qn - 1) / qn);
  if (d.vdim > 64) return d.sigmoid ? launch_tc<128, true>(map, d, w, geo, grid, st) : launch_tc<128, false>(map, d, w, geo, grid, st);
  return d.sigmoid ? launch_tc<64, true>(map, d, w, geo, grid, st) : launch_tc<64, false>(map, d, w, geo, grid, st);
}

}  // namespace vy
