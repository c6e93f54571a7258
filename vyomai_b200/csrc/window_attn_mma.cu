// Prompt-sized windowed attention over pages (vy_window_attn, portions of several tokens) where window_attn_tc.cu does not apply - short portions, more
// than 128 channels, little scratch - and the splitting of keys and values for both: scores and weighted values in fp32 precision
// on the tensor cores, operands split into two fp16 parts (split_mma.cuh), online softmax in registers.
//
// A first launch splits every key and value row that some query of the step sees, once, into a workspace in the order the tiles read
// them ([sequence][key / value head][key]: K hi | K lo | V hi | V lo, the bytes of the fp32 rows). In the second, a CTA owns 16 rows per warp:
// 2^hl query heads of one key / value head times the rows / 2^hl queries, so that heads that share keys share the key tiles and the window's
// edges waste little. A warp keeps its scores, weights and outputs in registers from one product to the next. Tiles of keys arrive by bulk copies
// into a ring of buffers; a warp waits for a tile, never for another warp, and the warp that is through with a buffer last refills it. (With CTA
// barriers per tile all warps are in the same phase: 267 and 854 us where the ring takes 228 and 548.)
//
// Halves suit keys and values of a moderate range: where a list's (one sequence, one key / value head) is too wide, or its scores too large, the kernel leaves it
// to the fp32 tiles (seqmix_tiled.cu), which are launched behind it and serve calls without a workspace too. 2.3 us where they find nothing to do.
//
// What bounds it: the tensor pipe (three fp16 products per fp32 one on mma.sync) and the shared-memory reads that feed it, about alike, then the
// instructions of the softmax. 4 x 2048 tokens, 8 heads of 128 over 2 key / value heads, window 512, capped: 236 us and 8 for the splitting (fp32 tiles, at 15 TFLOP/s: 943);
// 16 heads of 96 / 64 channels over the whole context: 545 and 41 us (2812).
#include "seqmix.cuh"
#include "split_mma.cuh"
#include "vy_ptx.cuh"

namespace vy {

constexpr int WS_T = 8 * SPLIT_ROWS;   // splitting launch: eight lanes per row

// bound by the bytes: every row read once and written once (8000 rows of 2 x (128 + 128) channels: 33 MB)
template <int MAXD>
__global__ void __launch_bounds__(WS_T) window_attn_split_kernel(WinDev d, SplitKv w, int dim16, bool kvvec) {
  pdl_trigger();
  pdl_wait();
  const int s = blockIdx.z, g = blockIdx.y, n = d.cu[s + 1] - d.cu[s], p0 = d.pos0[s];
  int nA, lo;
  portion_keys(d, p0, nA, lo);
  const int count = n > 0 ? nA + p0 + n - lo : 0;
  const int* tab = d.table + static_cast<long long>(s) * d.tw;
  const long long slot0 = (static_cast<long long>(s) * d.kv_heads + g) * w.cap;
  const int r0 = blockIdx.x * SPLIT_ROWS, sg = s * d.kv_heads + g;
  if (blockIdx.x == 0 && threadIdx.x == 0) w.odd[sg] = 0;
  // zeros behind the list, units too (rows the last tile's box takes in must not hold what their bits happen to say)
  // all the CTA's at once (a row after the other cost 32 single tokens beside a prompt 20 of 39 us)
  const int z0 = max(r0, count), zeros = min(min(r0 + SPLIT_ROWS, count + w.tail), static_cast<int>(w.cap)) - z0;
  if (w.tail > 0 && zeros > 0) {
    uint4* at = reinterpret_cast<uint4*>(w.rows + (slot0 + z0) * w.row_bytes);
    for (int x = threadIdx.x; x < zeros * (w.row_bytes / 16); x += WS_T) at[x] = make_uint4(0, 0, 0, 0);
    for (int x = threadIdx.x; x < zeros * 2; x += WS_T) w.unit[(slot0 + z0) * w.ustep + x] = 0.f;   // ustep is 2 with a tail
  }
  if (r0 >= count) return;
  __shared__ unsigned top_k, top_v, low_v;   // positive numbers order like their bits (and NaN after infinity)
  __shared__ long long row_s[SPLIT_ROWS];
  const int rows = min(SPLIT_ROWS, count - r0);
  const auto row_of = [&](int r) {
    const int kp = r0 + r < nA ? r0 + r : lo + (r0 + r - nA);
    return static_cast<long long>(tab[kp / d.bs] * d.bs + kp % d.bs);
  };
  if (threadIdx.x < rows) row_s[threadIdx.x] = row_of(threadIdx.x) * d.v_row + static_cast<long long>(g) * d.vdim;
  if (threadIdx.x == 0) {
    top_k = top_v = 0u;
    low_v = 0x7f800000u;
  }
  __syncthreads();
  unsigned char* out = w.rows + (slot0 + r0) * w.row_bytes;
  float* unit = w.unit + (slot0 + r0) * w.ustep;
  split_rows<WS_T / 32, MAXD>(out, out + w.k_lo, w.row_bytes, unit, SPLIT_TOP, rows, d.dim, dim16, d.kp, d.pool_dt, kvvec,
                              [&](int r) { return row_of(r) * d.k_row + static_cast<long long>(g) * d.dim; }, SameValue(), w.ustep,
                              [&](float m) { atomicMax(&top_k, __float_as_uint(m)); });
  out += w.v_at;
  split_rows<WS_T / 32, MAXD>(out, out + w.v_lo, w.row_bytes, unit + 1, 0, rows, d.vdim, w.vpad, d.vp, d.pool_dt, kvvec,
                              [&](int r) { return row_s[r]; }, SameValue(), w.ustep, [&](float m) {
                                if (m > 0.f) atomicMin(&low_v, __float_as_uint(m));
                              });
  for (int c0 = 0; c0 < d.vdim; c0 += WS_T) {   // columns, from the L1 cache
    const int c = c0 + threadIdx.x;
    unsigned m = 0u;
    if (c < d.vdim) {
#pragma unroll 8
      for (int r = 0; r < rows; ++r) m = max(m, __float_as_uint(fabsf(ld_as_float(d.vp, d.pool_dt, row_s[r] + c))));
    }
    const unsigned top = __reduce_max_sync(0xffffffffu, m), low = __reduce_min_sync(0xffffffffu, m && rows >= 8 ? m : 0x7f800000u);   // of fewer rows the largest may be small by chance
    if ((threadIdx.x & 31) == 0) {
      atomicMax(&top_v, top);
      atomicMin(&low_v, low);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) w.range[static_cast<long long>(sg) * w.blocks + blockIdx.x] = make_uint4(top_k, top_v, low_v, 0u);
}

// MAXD: most query / key channels; VT: value channels the accumulators hold; NW: warps (16 rows each); N: keys per tile; NS: tile buffers; SIG: sigmoid weights
template <int MAXD, int VT, int NW, int N, int NS, bool SIG>
__global__ void __launch_bounds__(32 * NW, 1) window_attn_mma_kernel(WinDev d, SplitKv w, PoisonRef poison, int hl, int dim16, int vdim16, bool qvec, bool ovec) {
  pdl_trigger();
  pdl_wait();
  constexpr int R = 16 * NW, NT = N / 8, KT = N / 16;   // rows of a CTA; the tile's keys as score columns of 8 and value steps of 16
  constexpr int NC = VT / 32;   // value columns go in blocks of 32
  extern __shared__ __align__(16) unsigned char wm_smem[];
  // bytes between rows (odd multiples of 16: ldmatrix without bank conflicts), from a hi entry to its lo entry, to the values, of a tile buffer
  const int qb = dim16 * 2 + 16, kb = w.row_bytes, k_lo = 2 * dim16, v_lo = 2 * vdim16, v_at = 2 * k_lo, buf = N * kb;
  unsigned char* Qh = wm_smem;
  unsigned char* Ts = Qh + 2 * R * qb;     // [buffers]: rows of the workspace
  float* qe = reinterpret_cast<float*>(Ts + NS * buf);   // powers of two that undo the scaling of the rows of Q
  uint64_t* full = reinterpret_cast<uint64_t*>(qe + R);  // a buffer's tile has arrived
  int* done = reinterpret_cast<int*>(full + NS);         // warps that are through with a buffer, counted up for ever
  int* issued = done + NS;                               // tiles sent for into a buffer
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
  const int s = blockIdx.z, h0 = blockIdx.y << hl, qn = R >> hl;
  const int base = d.cu[s], n = d.cu[s + 1] - base;
  // the last queries see the most keys: they go first
  const int blk = (n + qn - 1) / qn - 1 - static_cast<int>(blockIdx.x);
  if (blk < 0) return;
  const int i0 = blk * qn, nq = min(qn, n - i0), hm = (1 << hl) - 1;
  const int g = h0 / (d.heads / d.kv_heads);
  const int p0 = d.pos0[s], p_lo = p0 + i0, p_hi = p_lo + nq - 1;
  // visible keys of the tile's queries: [0, nA) (kept first tokens outside the band) and [lo, p_hi] (the band); masks are per pair
  int nA, lo;
  portion_keys(d, p_lo, nA, lo);
  const int count = nA + (p_hi - lo + 1);
  int nA0, lo0;   // the same of the portion: where the workspace keeps a key
  portion_keys(d, p0, nA0, lo0);
  const long long slot0 = (static_cast<long long>(s) * d.kv_heads + g) * w.cap;
  const auto key_of = [&](int c) { return c < nA ? c : lo + (c - nA); };
  const auto fetch = [&](int c0, int b) {   // tile of keys c0 .. into buffer b, by one warp: runs of neighbouring slots, one copy each; rows past the end are zeros
    unsigned char* T = Ts + b * buf;
    const int nk = min(N, count - c0);
    for (int x = lane; x < (N - nk) * (kb / 16); x += 32) *reinterpret_cast<uint4*>(T + nk * kb + 16 * x) = make_uint4(0, 0, 0, 0);
    __syncwarp();
    if (lane == 0) {
      ++issued[b];
      mbar_arrive_expect_tx(&full[b], static_cast<unsigned>(nk) * w.row_bytes);
      for (int j = 0; j < nk;) {   // kept tokens and the band are a run each; kept tokens beyond the portion's own lie at the band's start
        const int c = c0 + j, kp = key_of(c);
        const int run = min(nk - j, c >= nA ? nk : (kp < nA0 ? nA0 - c : nA - c));
        bulk_load(T + j * kb, w.rows + (slot0 + (kp >= lo0 ? nA0 + kp - lo0 : kp)) * w.row_bytes, static_cast<unsigned>(run) * w.row_bytes, &full[b]);
        j += run;
      }
    }
  };
  const int tiles = (count + N - 1) / N;
  if (threadIdx.x < NS) {
    mbar_init(&full[threadIdx.x], 1);
    done[threadIdx.x] = issued[threadIdx.x] = 0;
  }
  fence_mbar_init();
  __syncthreads();
  if (warp < min(NS, tiles)) fetch(warp * N, warp);
  split_rows<NW, MAXD>(Qh, Qh + R * qb, qb, qe, SPLIT_TOP, R, d.dim, dim16, d.q, d.q_dt, qvec, [&](int r) {
    return (r >> hl) < nq ? static_cast<long long>(base + i0 + (r >> hl)) * d.ldq + static_cast<long long>(h0 + (r & hm)) * d.dim : -1LL;
  });
  // this lane's two rows: 16 warp + gq and the one 8 below
  int pos[2];
  float m[2], l[2], qmul[2], badd[2], slope[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int r = 16 * warp + gq + 8 * e, h = h0 + (r & hm);
    pos[e] = p_lo + (r >> hl);
    m[e] = d.sink ? ld_as_float(d.sink, d.sink_dt, h) : -INFINITY;
    l[e] = d.sink && tq == 0 ? 1.f : 0.f;   // a row's sum is spread over its four lanes
    badd[e] = head_bias_of(d, h);
    slope[e] = head_slope_of(d, h);
    qmul[e] = head_scale_of(d, h);
  }
  const float two_over_cap = d.softcap > 0.f ? 2.f / d.softcap : 0.f;
  float o[NC * 4][4];
#pragma unroll
  for (int i = 0; i < NC * 4; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[i][e] = 0.f;
  int E = SPLIT_MIN_E;   // the outputs are kept in units of 2^(E - 2 SPLIT_TOP), E the largest exponent of a value row so far
  const unsigned qa_h = smem_addr(Qh) + 16 * warp * qb + lane_a(lane, qb), qa_l = qa_h + R * qb;
  const unsigned kb_0 = smem_addr(Ts) + lane_b(lane, kb), vb_0 = smem_addr(Ts) + v_at + lane_bt(lane, kb);
  float top_k;
  const bool odd = split_odd(w, s * d.kv_heads + g, nA0 + p0 + n - lo0, top_k);
  __syncthreads();   // Q is there
  bool big = false;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    qmul[e] *= qe[16 * warp + gq + 8 * e];
    big = big || !(fabsf(qmul[e]) * top_k <= SPLIT_SCORE);
  }
  if (__syncthreads_or(odd || big)) {   // not for fp16 halves: the fp32 form's
    for (int b = 0; b < min(NS, tiles); ++b)   // the copies in flight write to this CTA's memory
      if (!mbar_wait_soft(&full[b], 0, poison)) mbar_drain(full, issued, NS);
    if (threadIdx.x == 0) w.odd[s * d.kv_heads + g] = 1;
    return;
  }
  // from here on the warps wait for tiles, not for one another, so that one's softmax meets another's products
  bool alive = true;   // no wait of this thread has timed out; lane 0 sends for tiles
  for (int it = 0; it < tiles; ++it) {
    const int c0 = it * N, b = it % NS;
    alive = mbar_wait_soft(&full[b], (it / NS) & 1, poison) && alive;
    const unsigned kb_h = kb_0 + b * buf, vb_h = vb_0 + b * buf;
    // 2^(exponent - SPLIT_TOP) of each key row, 2^exponent of each value row
    const int ustep = kb / 4;
    const float* ke = reinterpret_cast<const float*>(Ts + b * buf + 4 * (dim16 + vdim16));
    const float* ve = ke + 1;
    // ---- scores ----
    float sc[NT][4], x[NT][4];   // hi hi, and the two small products
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) sc[i][e] = x[i][e] = 0.f;
#pragma unroll 2
    for (int k = 0; k < dim16; k += 16) {
      unsigned ah[4], al[4];
      ldsm_x4(ah, qa_h + k * 2);
      ldsm_x4(al, qa_l + k * 2);
#pragma unroll
      for (int j = 0; j < NT / 2; ++j) {
        unsigned bh[4], bl[4];
        ldsm_x4(bh, kb_h + 16 * j * kb + k * 2);
        ldsm_x4(bl, kb_h + k_lo + 16 * j * kb + k * 2);
        mma_f16(x[2 * j], al, bh[0], bh[1]);
        mma_f16(x[2 * j + 1], al, bh[2], bh[3]);
        mma_f16(sc[2 * j], ah, bh[0], bh[1]);
        mma_f16(sc[2 * j + 1], ah, bh[2], bh[3]);
        mma_f16(x[2 * j], ah, bl[0], bl[1]);
        mma_f16(x[2 * j + 1], ah, bl[2], bl[3]);
      }
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const float kx[2] = {ke[(8 * i + 2 * tq) * ustep], ke[(8 * i + 2 * tq + 1) * ustep]};
#pragma unroll
      for (int e = 0; e < 4; ++e) sc[i][e] = fmaf(fmaf(x[i][e], LO_UNIT, sc[i][e]) * kx[e & 1], qmul[e >> 1], badd[e >> 1]);
    }
    // a tile of neighbouring keys (no kept ones) that every query sees needs no mask per pair
    const int f = lo + (c0 - nA), t = f + N - 1;
    const bool whole = c0 >= nA && c0 + N <= count && t <= p_lo && (d.window <= 0 || p_hi - f < d.window) && (d.chunk <= 0 || f >= p_hi / d.chunk * d.chunk);
    if (d.softcap > 0.f) {
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[i][e] = cap_score(sc[i][e], d.softcap, two_over_cap);
    }
    if (d.head_slope) {
      const float away[2] = {static_cast<float>(pos[0] - f - 2 * tq), static_cast<float>(pos[1] - f - 2 * tq)};   // distance to the tile's first key of this lane
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int j = 8 * i + (e & 1), r = e >> 1, c = c0 + j + 2 * tq;
          sc[i][e] = fmaf(-slope[r], c0 >= nA || c >= nA ? away[r] - static_cast<float>(j) : static_cast<float>(pos[r] - c), sc[i][e]);
        }
    }
    if (!whole) {
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int c = c0 + 8 * i + 2 * tq + (e & 1), kp = key_of(c), p = pos[e >> 1];
          const bool vis = c < count && kp <= p && (d.window <= 0 || p - kp < d.window || kp < d.keep) && (d.chunk <= 0 || kp >= p / d.chunk * d.chunk);
          if (!vis) sc[i][e] = -INFINITY;
        }
    }
    // ---- weights, times 2^SPLIT_TOP and each value row's exponent against the running one ----
    unsigned ev = __float_as_uint(ve[lane * ustep]);   // positive numbers order like their bits
    if constexpr (N == 64) ev = max(ev, __float_as_uint(ve[(lane + 32) * ustep]));
    const int e_new = max(E, static_cast<int>(__reduce_max_sync(0xffffffffu, ev) >> 23) - 127);
    float keep_o[2] = {pow2i(E - e_new), pow2i(E - e_new)};
    E = e_new;
    const float v_unit = pow2i(SPLIT_TOP - E);
    if constexpr (!SIG) {
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
    }
    const float mm[2] = {m[0] == -INFINITY ? 0.f : m[0], m[1] == -INFINITY ? 0.f : m[1]};   // e^(-inf - 0) = 0 where nothing is visible yet
    unsigned ph[KT][4], pl[KT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const float vx[2] = {ve[(8 * i + 2 * tq) * ustep] * v_unit, ve[(8 * i + 2 * tq + 1) * ustep] * v_unit};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if constexpr (SIG) sc[i][e] = sigmoidf_(sc[i][e]);   // of -inf: 0
        else {
          sc[i][e] = expf(sc[i][e] - mm[e >> 1]);
          l[e >> 1] += sc[i][e];
        }
        sc[i][e] *= vx[e & 1];
      }
      split2(sc[i][0], sc[i][1], ph[i >> 1][(i & 1) * 2], pl[i >> 1][(i & 1) * 2]);
      split2(sc[i][2], sc[i][3], ph[i >> 1][(i & 1) * 2 + 1], pl[i >> 1][(i & 1) * 2 + 1]);
    }
    // ---- weighted values: the tile's own sum first, then one fp32 addition to the running output ----
#pragma unroll
    for (int cc = 0; cc < NC; ++cc) {
      if (32 * cc >= vdim16) break;
      float y[4][4], z[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) y[i][e] = z[i][e] = 0.f;
#pragma unroll
      for (int k = 0; k < KT; ++k) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (32 * cc + 16 * i < vdim16) {
            unsigned bh[4], bl[4];
            ldsm_x4_t(bh, vb_h + 16 * k * kb + (32 * cc + 16 * i) * 2);
            ldsm_x4_t(bl, vb_h + v_lo + 16 * k * kb + (32 * cc + 16 * i) * 2);
            mma_f16(z[2 * i], pl[k], bh[0], bh[1]);
            mma_f16(z[2 * i + 1], pl[k], bh[2], bh[3]);
            mma_f16(y[2 * i], ph[k], bh[0], bh[1]);
            mma_f16(y[2 * i + 1], ph[k], bh[2], bh[3]);
            mma_f16(z[2 * i], ph[k], bl[0], bl[1]);
            mma_f16(z[2 * i + 1], ph[k], bl[2], bl[3]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[4 * cc + i][e] = fmaf(o[4 * cc + i][e], keep_o[e >> 1], fmaf(z[i][e], LO_UNIT, y[i][e]));
    }
    // the warp that is through with a buffer last refills it
    __syncwarp();
    int last = 0;
    if (lane == 0) {
      __threadfence_block();
      last = atomicAdd(&done[b], 1) % NW == NW - 1 && alive;
      __threadfence_block();
      if (last) fence_proxy_async_smem();   // the reads of the buffer come before the copy that refills it
    }
    if (__shfl_sync(0xffffffffu, last, 0) && it + NS < tiles) fetch((it + NS) * N, b);
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    if constexpr (!SIG) {
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
    }
    const int row = 16 * warp + gq + 8 * r, i = row >> hl, h = h0 + (row & hm);
    if (i >= nq) continue;
    const long long qrow = base + i0 + i;
    float og = SIG ? d.out_scale : d.out_scale / l[r];
    if (d.gate) og *= sigmoidf_(ld_as_float(d.gate, d.gate_dt, qrow * d.ld_gate + h));
    const float unit = pow2i(E - 2 * SPLIT_TOP);
    const long long ob = qrow * d.ld_out + static_cast<long long>(h) * d.vdim;
#pragma unroll
    for (int t = 0; t < NC * 4; ++t) {
      const int col = 8 * t + 2 * tq;
      const float y0 = o[t][2 * r] * unit * og, y1 = o[t][2 * r + 1] * unit * og;
      if (ovec) {
        if (col < d.vdim) {
          if (d.out_dt == VY_BF16) *reinterpret_cast<__nv_bfloat162*>(reinterpret_cast<__nv_bfloat16*>(d.out) + ob + col) = __floats2bfloat162_rn(y0, y1);
          else *reinterpret_cast<float2*>(reinterpret_cast<float*>(d.out) + ob + col) = make_float2(y0, y1);
        }
      } else {
        store2_any(d.out, d.out_dt, ob + col, y0, y1, d.vdim - col);
      }
    }
  }
  if (__syncthreads_or(!alive)) mbar_drain(full, issued, NS);
}

static int round16(int n) { return (n + 15) & ~15; }

long long split_slots(const WinDev& d, int max_new) {
  const long long all = static_cast<long long>(d.tw) * d.bs;
  const long long seen = d.chunk > 0 ? static_cast<long long>(d.chunk) + max_new : d.window > 0 ? static_cast<long long>(d.window) + d.keep + max_new : all;
  return seen < all ? seen : all;
}

static long long split_blocks(const WinDev& d, int max_new) { return (split_slots(d, max_new) + SPLIT_ROWS - 1) / SPLIT_ROWS; }

// rows, ranges of blocks, and `odd` (in fours: whole 16 bytes)
long long window_attn_split_floats(const WinDev& d, int n_seqs, int max_new) {
  return static_cast<long long>(n_seqs) * d.kv_heads * (split_slots(d, max_new) * (round16(d.dim) + round16(d.vdim) + 4) + 4 * split_blocks(d, max_new) + 4);
}

static bool kv_quads(const WinDev& d) {
  const auto al = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  return d.pool_dt == VY_F32 && d.dim % 4 == 0 && d.vdim % 4 == 0 && d.k_row % 4 == 0 && d.v_row % 4 == 0 && al(d.kp) && al(d.vp);
}

cudaError_t launch_window_attn_split(const WinDev& d, int n_seqs, int max_new, float* ws, SplitKv* w, cudaStream_t st) {
  const int dim16 = round16(d.dim), vdim16 = round16(d.vdim);
  w->cap = split_slots(d, max_new);
  w->row_bytes = 4 * (dim16 + vdim16) + 16;
  w->k_lo = 2 * dim16;
  w->v_at = 4 * dim16;
  w->v_lo = 2 * vdim16;
  w->vpad = vdim16;
  w->ustep = w->row_bytes / 4;
  w->tail = 0;
  w->blocks = static_cast<int>(split_blocks(d, max_new));
  const long long lists = static_cast<long long>(n_seqs) * d.kv_heads;
  w->rows = reinterpret_cast<unsigned char*>(ws);
  w->range = reinterpret_cast<uint4*>(w->rows + lists * w->cap * w->row_bytes);
  w->odd = reinterpret_cast<int*>(w->range + lists * w->blocks);
  w->unit = reinterpret_cast<float*>(w->rows + 4 * (dim16 + vdim16));
  return launch_split_rows(d, n_seqs, *w, st);
}

cudaError_t launch_split_rows(const WinDev& d, int n_seqs, const SplitKv& w, cudaStream_t st) {
  const dim3 grid(w.blocks, d.kv_heads, n_seqs);
  return d.dim <= 128 && d.vdim <= 128 ? launch_kernel(window_attn_split_kernel<128>, grid, dim3(WS_T), 0, st, d, w, round16(d.dim), kv_quads(d))
                                       : launch_kernel(window_attn_split_kernel<256>, grid, dim3(WS_T), 0, st, d, w, round16(d.dim), kv_quads(d));
}

template <int MAXD, int VT, int NW, int N, int NS, bool SIG>
static cudaError_t launch_wm(const WinDev& d, const SplitKv& w, int n_seqs, int max_new, int hl, cudaStream_t st) {
  constexpr int R = 16 * NW;
  const int dim16 = round16(d.dim), vdim16 = round16(d.vdim);
  const size_t smem = 2 * R * (dim16 * 2 + 16) + static_cast<size_t>(NS) * N * w.row_bytes + sizeof(float) * R + 16 * NS;
  const auto al = [](const void* p, int a) { return reinterpret_cast<uintptr_t>(p) % a == 0; };
  const bool qvec = d.q_dt == VY_F32 && d.dim % 4 == 0 && d.ldq % 4 == 0 && al(d.q, 16);
  const bool ovec = d.vdim % 2 == 0 && d.ld_out % 2 == 0 && al(d.out, d.out_dt == VY_BF16 ? 4 : 8);
  static std::atomic<unsigned long long> allowed{0};
  if (smem > 48 * 1024) {
    cudaError_t e = allow_smem(window_attn_mma_kernel<MAXD, VT, NW, N, NS, SIG>, allowed);
    if (e != cudaSuccess) return e;
  }
  PoisonRef poison = {};
  if (!poison_ref(&poison)) return cudaErrorMemoryAllocation;
  const int qn = R >> hl;
  return launch_kernel(window_attn_mma_kernel<MAXD, VT, NW, N, NS, SIG>, dim3((max_new + qn - 1) / qn, d.heads >> hl, n_seqs), dim3(32 * NW), smem, st, d, w, poison, hl,
                       dim16, vdim16, qvec, ovec);
}

template <int MAXD, int VT>
static cudaError_t launch_wm_pick(const WinDev& d, const SplitKv& w, int n_seqs, int max_new, int hl, cudaStream_t st) {
  const auto go = [&](auto sig) {
    constexpr bool S = decltype(sig)::value;
    constexpr int N = VT <= 64 ? 64 : 32;
    // CTAs of 64 rows, two per SM (key tiles as wide as that allows), so that one's softmax runs beside the other's products; wide values on
    // long prompts take one CTA of 192 rows with three warps per scheduler instead, where that still is two rounds of CTAs over the SMs.
    // 8 heads of 128 over 2, 4 x 2048 tokens, window 512, capped / sigmoid: 192 rows 235 / 237 us, 64 rows 240 / 262 us, 128 rows 236 / 270 us;
    // portions of 1000 and 37 tokens: 123, 56, 62 us; 96 / 64 channels, whole context, 64 / 128 / 192 rows: 548, 590, 656 us
    if constexpr (VT == 128) {
      const int qn = 192 >> hl;
      if (static_cast<long long>((max_new + qn - 1) / qn) * (d.heads >> hl) * n_seqs >= 2 * num_sms())
        return launch_wm<MAXD, VT, 12, 32, 3, S>(d, w, n_seqs, max_new, hl, st);
    }
    return launch_wm<MAXD, VT, 4, N, 2, S>(d, w, n_seqs, max_new, hl, st);
  };
  return d.sigmoid ? go(std::true_type{}) : go(std::false_type{});
}

static cudaError_t launch_window_attn_mma(const WinDev& d, const SplitKv& w, int n_seqs, int max_new, cudaStream_t st) {
  // heads per tile: the largest power of two, at most 16, that divides the heads of a key / value head
  const int rep = d.heads / d.kv_heads;
  int hl = 0;
  while (hl < 4 && rep % (2 << hl) == 0) ++hl;
  if (d.vdim > 128 || d.dim > 128) return launch_wm_pick<256, 256>(d, w, n_seqs, max_new, hl, st);   // callers keep both <= 256
  if (d.vdim > 64) return launch_wm_pick<128, 128>(d, w, n_seqs, max_new, hl, st);
  return d.dim <= 64 ? launch_wm_pick<64, 64>(d, w, n_seqs, max_new, hl, st) : launch_wm_pick<128, 64>(d, w, n_seqs, max_new, hl, st);
}

static WinDev from_sequence(const WinDev& d, int s) {
  WinDev e = d;
  e.cu += s;
  e.pos0 += s;
  e.table += static_cast<long long>(s) * d.tw;
  return e;
}

cudaError_t launch_window_attn_prompt(const WinDev& d, int n_seqs, int max_new, float* ws, long long ws_floats, cudaStream_t st, int* launches) {
  *launches = 1;
  const bool aligned = ws && reinterpret_cast<uintptr_t>(ws) % 16 == 0 && d.kv_heads <= 65535;
  if (aligned && window_attn_tc_applies(d, n_seqs, max_new) && window_attn_tc_floats(d, 1, max_new) <= ws_floats) {
    const long long fit = ws_floats / window_attn_tc_floats(d, 1, max_new);
    *launches = 0;
    for (int s = 0; s < n_seqs; s += static_cast<int>(fit < n_seqs ? fit : n_seqs)) {
      const int ns = static_cast<int>(fit < n_seqs - s ? fit : n_seqs - s);
      const WinDev e = from_sequence(d, s);
      const int* odd = nullptr;
      cudaError_t err = launch_window_attn_tc(e, ns, max_new, ws, &odd, st);
      if (err == cudaSuccess) err = launch_window_attn_tiled(e, ns, max_new, odd, st);
      if (err != cudaSuccess) return err;
      *launches += 3;
    }
    return cudaSuccess;
  }
  const long long fit = aligned ? ws_floats / window_attn_split_floats(d, 1, max_new) : 0;
  if (fit < 1) return launch_window_attn_tiled(d, n_seqs, max_new, nullptr, st);
  *launches = 0;
  for (int s = 0; s < n_seqs; s += static_cast<int>(fit < n_seqs ? fit : n_seqs)) {   // as many sequences at a time as the workspace holds
    const int ns = static_cast<int>(fit < n_seqs - s ? fit : n_seqs - s);
    const WinDev e = from_sequence(d, s);
    SplitKv w = {};
    cudaError_t err = launch_window_attn_split(e, ns, max_new, ws, &w, st);
    if (err == cudaSuccess) err = launch_window_attn_mma(e, w, ns, max_new, st);
    if (err == cudaSuccess) err = launch_window_attn_tiled(e, ns, max_new, w.odd, st);
    if (err != cudaSuccess) return err;
    *launches += 3;
  }
  return cudaSuccess;
}

}  // namespace vy
