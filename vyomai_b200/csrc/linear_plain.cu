// vy_linear_plain: out = act(A W^T + bias) * scale + addend for any M, N, K and any alignment, fp32 accumulation.
// Five kernels: for many rows 64 x 64 tiles on the tensor cores in fp32 precision where both operands are fp32, aligned and K is long, else
// 64 x 64 x 16 shared-memory tiles of FMAs (4 x 4 outputs per thread) or, for K up to 32, weights in registers; a weight-streaming kernel
// (one warp per output feature, lanes over K) for at most 8 rows, and a 32-feature tile for 9 .. 32 rows. A call may hold a batch
// of independent products of one shape (blockIdx z / y picks the product). This is the exact-fp32 arm of every projection of the
// sequence-mixer models and the bf16 arm of the shapes the tensor-core GEMM does not take (a contraction over a
// low rank, a handful of output features, strides that are not 16-byte multiples). vy_unary and vy_embed_rows live
// here as well.
#include "linear_plain.cuh"

namespace vy {

constexpr int LT = 64, LK = 16;

__global__ void __launch_bounds__(256) linear_tile_kernel(LinDev d) {
  pdl_trigger();
  pdl_wait();
  lin_select(d, blockIdx.z);
  __shared__ float As[LK][LT + 4];
  __shared__ float Ws[LK][LT + 4];
  const int m0 = blockIdx.y * LT, n0 = blockIdx.x * LT;
  const int tid = threadIdx.x;
  const int lr = tid >> 2, lk = (tid & 3) * 4;  // loader: row 0..63, 4 consecutive k
  const int tm = (tid >> 4) * 4, tn = (tid & 15) * 4;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < d.K; k0 += LK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = k0 + lk + i;
      const int am = m0 + lr, wn = n0 + lr;
      As[lk + i][lr] = (am < d.M && k < d.K) ? ld_as_float(d.A, d.a_dt, static_cast<long long>(am) * d.lda + k) : 0.f;
      Ws[lk + i][lr] = (wn < d.N && k < d.K) ? ld_as_float(d.W, d.w_dt, static_cast<long long>(wn) * d.ldw + k) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < LK; ++k) {
      const float4 a = *reinterpret_cast<const float4*>(&As[k][tm]);
      const float4 w = *reinterpret_cast<const float4*>(&Ws[k][tn]);
      const float av[4] = {a.x, a.y, a.z, a.w}, wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (m0 + tm + i < d.M && n0 + tn + j < d.N) lin_store(d, m0 + tm + i, n0 + tn + j, acc[i][j]);
}

// Contractions of up to 32 over many rows: bound by the bytes of the results. A thread keeps the weights of two neighbouring features in registers, rows of A come from shared memory
// as broadcasts, results leave as pairs. The same sums in the same order as the tiles above. 7970 x 1024, K 16: 16 us, 30 in tiles
// of 64 x 64 (four results per thread for 32 scalar loads); x 2048 27, 52.
constexpr int LN_ROWS = 64, LN_K = 32;   // rows per CTA: half as many where CTAs would be too few
template <int KP>
__device__ __forceinline__ void thin_weights(const LinDev& d, int n, float (&w)[KP]) {
  const bool al = n < d.N && reinterpret_cast<uintptr_t>(d.W) % 16 == 0;
  if (al && d.w_dt == VY_BF16 && d.K % 8 == 0 && d.ldw % 8 == 0) {
    const uint4* p = reinterpret_cast<const uint4*>(static_cast<const char*>(d.W) + 2 * static_cast<long long>(n) * d.ldw);
#pragma unroll
    for (int i = 0; i < KP / 8; ++i) {
      const uint4 v = 8 * i < d.K ? p[i] : make_uint4(0u, 0u, 0u, 0u);
      const unsigned u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        w[8 * i + 2 * j] = __uint_as_float(u[j] << 16);
        w[8 * i + 2 * j + 1] = __uint_as_float(u[j] & 0xffff0000u);
      }
    }
    return;
  }
  if (al && d.w_dt == VY_F32 && d.K % 4 == 0 && d.ldw % 4 == 0) {
    const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(d.W) + static_cast<long long>(n) * d.ldw);
#pragma unroll
    for (int i = 0; i < KP / 4; ++i) {
      const float4 v = 4 * i < d.K ? p[i] : make_float4(0.f, 0.f, 0.f, 0.f);
      w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
    }
    return;
  }
#pragma unroll
  for (int k = 0; k < KP; ++k) w[k] = n < d.N && k < d.K ? ld_as_float(d.W, d.w_dt, static_cast<long long>(n) * d.ldw + k) : 0.f;
}
template <int KP>
__global__ void __launch_bounds__(256) linear_thin_kernel(const __grid_constant__ LinDev d0, int per_cta) {
  pdl_trigger();
  pdl_wait();
  LinDev d = d0;
  lin_select(d, blockIdx.z);
  __shared__ __align__(16) float as[LN_ROWS][KP];
  const int m0 = blockIdx.y * per_cta, n = 2 * (blockIdx.x * 256 + threadIdx.x);
  for (int e = threadIdx.x; e < per_cta * KP; e += 256) {
    const int r = e / KP, k = e % KP;
    as[r][k] = m0 + r < d.M && k < d.K ? ld_as_float(d.A, d.a_dt, static_cast<long long>(m0 + r) * d.lda + k) : 0.f;
  }
  float w[2][KP];
  thin_weights(d, n, w[0]);
  thin_weights(d, n + 1, w[1]);
  const float b0 = d.bias && n < d.N ? ld_as_float(d.bias, d.bias_dt, n) : 0.f, b1 = d.bias && n + 1 < d.N ? ld_as_float(d.bias, d.bias_dt, n + 1) : 0.f;
  __syncthreads();
  if (n >= d.N) return;
  const int rows = min(per_cta, d.M - m0);
  float* out = static_cast<float*>(d.out) + static_cast<long long>(m0) * d.ld_out + n;
#pragma unroll 4
  for (int r = 0; r < rows; ++r, out += d.ld_out) {
    float y0 = 0.f, y1 = 0.f;
#pragma unroll
    for (int k = 0; k < KP; k += 4) {
      const float4 x = *reinterpret_cast<const float4*>(&as[r][k]);
      y0 = fmaf(x.x, w[0][k], y0); y0 = fmaf(x.y, w[0][k + 1], y0); y0 = fmaf(x.z, w[0][k + 2], y0); y0 = fmaf(x.w, w[0][k + 3], y0);
      y1 = fmaf(x.x, w[1][k], y1); y1 = fmaf(x.y, w[1][k + 1], y1); y1 = fmaf(x.z, w[1][k + 2], y1); y1 = fmaf(x.w, w[1][k + 3], y1);
    }
    if (d.bias) { y0 += b0; y1 += b1; }
    y0 = uact(y0, d.act) * d.scale;
    y1 = uact(y1, d.act) * d.scale;
    if (n + 1 < d.N) *reinterpret_cast<float2*>(out) = make_float2(y0, y1);
    else *out = y0;
  }
}

// fp32 operands with 16-byte aligned rows: fp32 precision on the tensor cores (split_mma.cuh). 64 rows x 64 features per CTA, a warp 32 x 16.
// Tiles of 64 k: loaded into registers while the tile before is multiplied, then split, with a scale per row and tile, into one of two buffers; a
// tile's sums (chains of 4 steps) are added to fp32 registers. 8 warps and two CTAs per SM hide the loads and the splitting behind the products.
// The FMA form / this, us: 1600 x 3072, K 1024 460 / 178; 8192 x 1024, K 1024 696 / 275; 512 x 1024, K 1024 82 / 28; 8192 x 16, K 1024 77 / 27 (error
// against 64 bits 5.7e-7 / 1.6e-7; without the second look at small products 173, 264, 26, 25 us).
// Bound by the instructions that split the tiles (three products take a third of the time)
constexpr int LS_KT = 64, LS_KB = LS_KT * 2 + 16, LS_PLANE = LT * LS_KB, LS_BUF = 4 * LS_PLANE + 2 * LT * 4;

__global__ void __launch_bounds__(256, 2) linear_split_kernel(const LinDev d0) {
  pdl_trigger();
  pdl_wait();
  LinDev d = d0;
  lin_select(d, blockIdx.z);
  extern __shared__ __align__(16) unsigned char lin_smem[];
  const int m0 = blockIdx.y * LT, n0 = blockIdx.x * LT;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wm = (warp >> 2) * 32, wn = (warp & 3) * 16;
  const int lr = 4 * warp + (lane >> 3), lc = (lane & 7) * 4;   // loader: rows lr, lr + 32 of A and of W, columns lc .., lc + 32 ..
  const float* src[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int r = lr + 32 * (u & 1);
    src[u] = nullptr;
    if (u < 2 && m0 + r < d.M) src[u] = static_cast<const float*>(d.A) + static_cast<long long>(m0 + r) * d.lda + lc;
    if (u >= 2 && n0 + r < d.N) src[u] = static_cast<const float*>(d.W) + static_cast<long long>(n0 + r) * d.ldw + lc;
  }
  float4 x[4][2];
  const auto load = [&](int k0) {
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        x[u][i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (src[u] && k0 + lc + 32 * i < d.K) x[u][i] = *reinterpret_cast<const float4*>(src[u] + k0 + 32 * i);
      }
  };
  float acc[2][2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
  float top_a[2][2] = {}, top_w[2][2] = {};   // the largest units of this lane's rows of A (and of 8 below) and of W
  load(0);
  for (int k0 = 0, b = 0; k0 < d.K; k0 += LS_KT, b ^= 1) {
    unsigned char* buf = lin_smem + b * LS_BUF;   // A hi | A lo | W hi | W lo | units of A and W rows
    float* unit = reinterpret_cast<float*>(buf + 4 * LS_PLANE);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float m = 0.f;
#pragma unroll
      for (int i = 0; i < 2; ++i) m = fmaxf(m, fmaxf(fmaxf(fabsf(x[u][i].x), fabsf(x[u][i].y)), fmaxf(fabsf(x[u][i].z), fabsf(x[u][i].w))));
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      const int ex = split_exponent(m), r = lr + 32 * (u & 1);
      const float sc = split_scale(ex);
      if (lc == 0) unit[LT * (u >> 1) + r] = m > 0.f ? pow2i(ex - SPLIT_TOP) : 0.f;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        uint2 h, l;
        split2(x[u][i].x * sc, x[u][i].y * sc, h.x, l.x);
        split2(x[u][i].z * sc, x[u][i].w * sc, h.y, l.y);
        unsigned char* o = buf + (u & 2) * LS_PLANE + r * LS_KB + 2 * (lc + 32 * i);
        *reinterpret_cast<uint2*>(o) = h;
        *reinterpret_cast<uint2*>(o + LS_PLANE) = l;
      }
    }
    if (k0 + LS_KT < d.K) load(k0 + LS_KT);
    __syncthreads();   // the only one per tile: the buffer written next was read before this barrier
    float y[2][2][4], z[2][2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) y[i][j][e] = z[i][j][e] = 0.f;
    const unsigned aa = smem_addr(buf) + wm * LS_KB + lane_a(lane, LS_KB), wa = smem_addr(buf) + 2 * LS_PLANE + wn * LS_KB + lane_b(lane, LS_KB);
#pragma unroll
    for (int k = 0; k < LS_KT; k += 16) {
      unsigned ah[2][4], al[2][4], bh[4], bl[4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        ldsm_x4(ah[i], aa + 16 * i * LS_KB + 2 * k);
        ldsm_x4(al[i], aa + LS_PLANE + 16 * i * LS_KB + 2 * k);
      }
      ldsm_x4(bh, wa + 2 * k);
      ldsm_x4(bl, wa + LS_PLANE + 2 * k);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) mma_f16(z[i][j], al[i], bh[2 * j], bh[2 * j + 1]);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) mma_f16(y[i][j], ah[i], bh[2 * j], bh[2 * j + 1]);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) mma_f16(z[i][j], ah[i], bl[2 * j], bl[2 * j + 1]);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float u0 = unit[wm + 16 * i + (lane >> 2)], u1 = unit[wm + 16 * i + 8 + (lane >> 2)];
      top_a[i][0] = fmaxf(top_a[i][0], u0);
      top_a[i][1] = fmaxf(top_a[i][1], u1);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float2 w = *reinterpret_cast<const float2*>(unit + LT + wn + 8 * j + 2 * (lane & 3));
        if (i == 0) {
          top_w[j][0] = fmaxf(top_w[j][0], w.x);
          top_w[j][1] = fmaxf(top_w[j][1], w.y);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][j][e] = fmaf(fmaf(z[i][j][e], LO_UNIT, y[i][j][e]) * (e < 2 ? u0 : u1), e & 1 ? w.y : w.x, acc[i][j][e]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int m = m0 + wm + 16 * i + (lane >> 2) + 8 * (e >> 1), n = n0 + wn + 8 * j + 2 * (lane & 3) + (e & 1);
        const bool in = m < d.M && n < d.N;
        const float y = fabsf(acc[i][j][e]);
        for (unsigned again = __ballot_sync(0xffffffffu, in && !(y >= LS_SMALL * top_a[i][e >> 1] * top_w[j][e & 1] && y < INFINITY)); again; again &= again - 1) {
          const int src = __ffs(again) - 1, ms = __shfl_sync(0xffffffffu, m, src), ns = __shfl_sync(0xffffffffu, n, src);
          const float x = lin_dot(static_cast<const float*>(d.A) + ms * d.lda, static_cast<const float*>(d.W) + ns * d.ldw, d.K);
          if (lane == src) acc[i][j][e] = x;
        }
        if (in) lin_store(d, m, n, acc[i][j][e]);
      }
}

// at most 8 rows: one warp per output feature, lanes stride over K (coalesced weight rows), shuffle reduction
__global__ void __launch_bounds__(256) linear_rows_kernel(LinDev d) {
  pdl_trigger();
  pdl_wait();
  lin_select(d, blockIdx.y);
  const int n = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (n >= d.N) return;
  float acc[8];
#pragma unroll
  for (int m = 0; m < 8; ++m) acc[m] = 0.f;
  for (int k = lane; k < d.K; k += 32) {
    const float w = ld_as_float(d.W, d.w_dt, static_cast<long long>(n) * d.ldw + k);
#pragma unroll
    for (int m = 0; m < 8; ++m)
      if (m < d.M) acc[m] = fmaf(ld_as_float(d.A, d.a_dt, static_cast<long long>(m) * d.lda + k), w, acc[m]);
  }
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    float v = acc[m];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0 && m < d.M) lin_store(d, m, n, v);
  }
}

// 9 .. 32 rows (a decode batch; the per-head products of latent attention): a CTA takes 32 output features of one product, thread
// (feature, group of 4 rows); A and W pass through shared memory 64 k at a time, W transposed so that a warp's features are adjacent
constexpr int LS_N = 32, LS_K = 64, LS_M = 32;
__global__ void __launch_bounds__(256) linear_small_kernel(LinDev d) {
  pdl_trigger();
  pdl_wait();
  lin_select(d, blockIdx.y);
  __shared__ __align__(16) float xs[LS_M][LS_K + 4];
  __shared__ float ws[LS_K][LS_N + 1];
  const int t = threadIdx.x, n = t & 31, mg = t >> 5;
  const int n0 = blockIdx.x * LS_N;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int k0 = 0; k0 < d.K; k0 += LS_K) {
    {
      const int r = t >> 3, kk = (t & 7) * 8;   // 32 rows x 8 threads x 8 k
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int k = k0 + kk + j;
        xs[r][kk + j] = (r < d.M && k < d.K) ? ld_as_float(d.A, d.a_dt, static_cast<long long>(r) * d.lda + k) : 0.f;
        ws[kk + j][r] = (n0 + r < d.N && k < d.K) ? ld_as_float(d.W, d.w_dt, static_cast<long long>(n0 + r) * d.ldw + k) : 0.f;
      }
    }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < LS_K; k += 4) {
      const float w0 = ws[k][n], w1 = ws[k + 1][n], w2 = ws[k + 2][n], w3 = ws[k + 3][n];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 x = *reinterpret_cast<const float4*>(&xs[4 * mg + i][k]);
        acc[i] = fmaf(x.x, w0, acc[i]);
        acc[i] = fmaf(x.y, w1, acc[i]);
        acc[i] = fmaf(x.z, w2, acc[i]);
        acc[i] = fmaf(x.w, w3, acc[i]);
      }
    }
    __syncthreads();
  }
  if (n0 + n < d.N)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (4 * mg + i < d.M) lin_store(d, 4 * mg + i, n0 + n, acc[i]);
}

__global__ void __launch_bounds__(256) unary_kernel(long long rows, int cols, const void* x, long long ldx, int x_dt, int act,
                                                     void* out, long long ld_out, int out_dt) {
  pdl_trigger();
  pdl_wait();
  const long long n = rows * cols;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / cols;
    const int c = static_cast<int>(i - r * cols);
    st_from_float(out, out_dt, r * ld_out + c, uact(ld_as_float(x, x_dt, r * ldx + c), act));
  }
}

__global__ void __launch_bounds__(128) embed_rows_kernel(int rows, int width, int vocab, const int* __restrict__ ids,
                                                         const void* table, long long ld_table, int table_dt, float scale, void* out,
                                                         long long ld_out, int out_dt) {
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x;
  const int id = ids[r];
  const bool ok = id >= 0 && id < vocab;
  for (int c = threadIdx.x; c < width; c += blockDim.x)
    st_from_float(out, out_dt, static_cast<long long>(r) * ld_out + c,
                  ok ? scale * ld_as_float(table, table_dt, static_cast<long long>(id) * ld_table + c) : 0.f);
}

struct PairDev {
  const int* cu; const int* pos0; const int* slot; const int* ids;
  int width, vocab, table_dt;
  const void* table; long long ld_table; const void* pairs; long long ld_pairs;
  float scale;
  long long mul_prev, mul_cur; int buckets;   // multipliers reduced modulo buckets by the host: the products fit 64 bits
  int* prev;
  void* out; long long ld_out; int out_dt;
};

// blockIdx.x = token of the portion, blockIdx.y = sequence. Only the portion's first token's CTA touches the sequence's prev_state: it
// reads the token before the portion and leaves the portion's last one
__global__ void __launch_bounds__(128) pair_embed_kernel(PairDev d) {
  pdl_trigger();
  pdl_wait();
  __shared__ int prev_s;
  const int s = blockIdx.y;
  const int base = d.cu[s], n = d.cu[s + 1] - base;
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const int r = base + i, id = d.ids[r], pos = d.pos0[s] + i;
    int prev = 0;
    if (i > 0) prev = d.ids[r - 1];
    else {
      if (threadIdx.x == 0) {
        int* st = d.prev + d.slot[s];
        prev_s = pos > 0 ? *st : 0;
        *st = d.ids[base + n - 1];
      }
      __syncthreads();
      prev = prev_s;
    }
    long long b = d.buckets;
    if (pos > 0) {
      b = (prev * d.mul_prev + id * d.mul_cur) % d.buckets;
      if (b < 0) b += d.buckets;   // ids below zero
    }
    const bool ok = id >= 0 && id < d.vocab;
    for (int c = threadIdx.x; c < d.width; c += blockDim.x) {
      const float e = ok ? d.scale * ld_as_float(d.table, d.table_dt, static_cast<long long>(id) * d.ld_table + c) : 0.f;
      st_from_float(d.out, d.out_dt, static_cast<long long>(r) * d.ld_out + c, e + ld_as_float(d.pairs, d.table_dt, b * d.ld_pairs + c));
    }
  }
}

}  // namespace vy

extern "C" int vy_pair_embed(const VyPairEmbed* p) {
  using namespace vy;
  VY_CHECK_ARG(p != nullptr, "vy_pair_embed: null params");
  if (!vy_device_ok()) {
    set_error("vy_pair_embed: no sm_100 device (there is no CPU fallback)");
    return VY_ERR_NO_DEVICE;
  }
  VY_CHECK_ARG(p->n_seqs > 0 && p->n_seqs <= 65535 && p->max_new > 0 && p->cu_tokens && p->pos0 && p->slot && p->ids, "vy_pair_embed: bad batch");
  VY_CHECK_ARG(p->width > 0 && p->vocab > 0 && p->table && p->pairs && p->prev_state && p->out && dtype_ok(p->table_dtype) && dtype_ok(p->out_dtype),
               "vy_pair_embed: bad tensors");
  VY_CHECK_ARG(p->buckets > 0 && p->mul_prev >= 0 && p->mul_cur >= 0, "vy_pair_embed: %d buckets and the multipliers must be positive", p->buckets);
  PairDev d;
  d.cu = p->cu_tokens; d.pos0 = p->pos0; d.slot = p->slot; d.ids = p->ids;
  d.width = p->width; d.vocab = p->vocab; d.table_dt = p->table_dtype;
  d.table = p->table; d.ld_table = p->ld_table; d.pairs = p->pairs; d.ld_pairs = p->ld_pairs;
  d.scale = p->scale;
  d.mul_prev = p->mul_prev % p->buckets; d.mul_cur = p->mul_cur % p->buckets; d.buckets = p->buckets;
  d.prev = p->prev_state;
  d.out = p->out; d.ld_out = p->ld_out; d.out_dt = p->out_dtype;
  const unsigned gx = static_cast<unsigned>(p->max_new < 65535 ? p->max_new : 65535);
  VY_CUDA_OK(launch_kernel(pair_embed_kernel, dim3(gx, p->n_seqs), dim3(128), 0, static_cast<cudaStream_t>(p->stream), d));
  VY_LAUNCH_OK();
  count_launch();
  return VY_OK;
}

extern "C" int64_t vy_linear_plain_bytes(int32_t M, int32_t N, int32_t K) { return vy::linear_split_bytes(M, N, K); }

extern "C" int vy_linear_plain(const VyLinear* p) {
  using namespace vy;
  VY_CHECK_ARG(p != nullptr, "vy_linear_plain: null params");
  if (!vy_device_ok()) {
    set_error("vy_linear_plain: no sm_100 device (there is no CPU fallback)");
    return VY_ERR_NO_DEVICE;
  }
  VY_CHECK_ARG(p->M > 0 && p->N > 0 && p->K > 0, "vy_linear_plain: bad shape M=%d N=%d K=%d", p->M, p->N, p->K);
  VY_CHECK_ARG(p->A && p->W && p->out, "vy_linear_plain: null operand");
  VY_CHECK_ARG(dtype_ok(p->a_dtype) && dtype_ok(p->w_dtype) && dtype_ok(p->out_dtype), "vy_linear_plain: bad dtype");
  VY_CHECK_ARG(p->lda >= p->K && p->ldw >= p->K && p->ld_out >= p->N, "vy_linear_plain: leading dimension smaller than the row");
  VY_CHECK_ARG(p->act >= VY_UACT_NONE && p->act <= VY_UACT_GELU_TANH, "vy_linear_plain: bad act %d", p->act);
  const int batch = p->batch > 1 ? p->batch : 1;
  VY_CHECK_ARG(batch <= 65535 && (batch == 1 || ((!p->bias || p->bias_batch != 0) && !p->addend)), "vy_linear_plain: a batched call takes no addend, a bias with its stride (batch %d)", batch);
  if (p->bias) VY_CHECK_ARG(dtype_ok(p->bias_dtype), "vy_linear_plain: bad bias_dtype");
  if (p->addend) VY_CHECK_ARG(dtype_ok(p->addend_dtype) && p->ld_addend >= p->N, "vy_linear_plain: bad addend");
  LinDev d;
  d.M = p->M; d.N = p->N; d.K = p->K;
  d.A = p->A; d.lda = p->lda; d.a_dt = p->a_dtype;
  d.W = p->W; d.ldw = p->ldw; d.w_dt = p->w_dtype;
  d.bias = p->bias; d.bias_dt = p->bias_dtype;
  d.addend = p->addend; d.ld_addend = p->ld_addend; d.addend_dt = p->addend_dtype;
  d.act = p->act; d.scale = p->scale == 0.f ? 1.f : p->scale;
  d.out = p->out; d.ld_out = p->ld_out; d.out_dt = p->out_dtype;
  d.a_batch = p->a_batch; d.w_batch = p->w_batch; d.out_batch = p->out_batch; d.bias_batch = p->bias_batch;
  cudaStream_t st = static_cast<cudaStream_t>(p->stream);
  if (p->M <= 8) {
    VY_CUDA_OK(launch_kernel(linear_rows_kernel, dim3((p->N + 7) / 8, batch), dim3(256), 0, st, d));
  } else if (p->M <= LS_M) {
    VY_CUDA_OK(launch_kernel(linear_small_kernel, dim3((p->N + LS_N - 1) / LS_N, batch), dim3(256), 0, st, d));
  } else {
    VY_CHECK_ARG((p->M + LT - 1) / LT <= 65535, "vy_linear_plain: too many rows (%d)", p->M);
    const auto rows16 = [](const void* q, int dt, long long ld, long long step) { return dt == VY_F32 && reinterpret_cast<uintptr_t>(q) % 16 == 0 && ld % 4 == 0 && step % 4 == 0; };
    // from K = 256 on: below, a chain of FMAs is at least as exact (all terms positive, K 256: 2.5e-7 by FMAs, 2.1e-7 split; K 64: 1.2e-7, 2.1e-7), and the
    // two cost the same at 64 (9 us for 33 x 64)
    if (p->K >= 256 && p->K % 4 == 0 && rows16(d.A, d.a_dt, d.lda, batch > 1 ? d.a_batch : 0) && rows16(d.W, d.w_dt, d.ldw, batch > 1 ? d.w_batch : 0)) {
      const long long need = batch == 1 ? linear_split_bytes(p->M, p->N, p->K) : 0;
      if (need > 0 && p->workspace && reinterpret_cast<uintptr_t>(p->workspace) % 128 == 0 && p->workspace_bytes >= need) {
        if (poison_raised("vy_linear_plain")) return VY_ERR_CUDA;
        VY_CUDA_OK(launch_linear_split_tc(d, p->workspace, st));
        VY_LAUNCH_OK();
        count_launch(2);
        return VY_OK;
      }
      static std::atomic<unsigned long long> allowed{0};
      VY_CUDA_OK(allow_smem(linear_split_kernel, allowed));
      VY_CUDA_OK(launch_kernel(linear_split_kernel, dim3((p->N + LT - 1) / LT, (p->M + LT - 1) / LT, batch), dim3(256), 2 * LS_BUF, st, d));
      VY_LAUNCH_OK();
      count_launch();
      return VY_OK;
    }
    // K up to 32, fp32 results in pairs. A CTA has 512 features: 128 of them, 7970 rows 7.2 us in tiles, 7.9 here; 512 16.9, 9.7; 33 x 512 5.8, 5.0; 2000 x 2048, K 32 22.3, 14.2. Beyond 16
    // a CTA's weights take longer to come than few rows' tiles: K 24 44 x 4034 7.2, 8.2, 187 x 316 7.6, 8.2, 2061 x 478 8.9, 8.5; 32 81 x 462 7.2, 8.1, 355 x 2830 9.0, 8.3
    if (p->K <= LN_K && p->N >= 256 && (p->K <= 16 || static_cast<long long>(p->M) * p->N >= 200000) && !d.addend && d.out_dt == VY_F32 && reinterpret_cast<uintptr_t>(d.out) % 8 == 0 && d.ld_out % 2 == 0 && (batch == 1 || d.out_batch % 2 == 0) &&
        p->M <= 65535 * (LN_ROWS / 4)) {
      const long long wide = (p->N + 511LL) / 512 * batch;
      const int per_cta = wide * (p->M / LN_ROWS) >= num_sms() ? LN_ROWS : wide * (2 * p->M / LN_ROWS) >= num_sms() ? LN_ROWS / 2 : LN_ROWS / 4;
      const dim3 grid((p->N + 511) / 512, (p->M + per_cta - 1) / per_cta, batch);
      VY_CUDA_OK(p->K <= 16 ? launch_kernel(linear_thin_kernel<16>, grid, dim3(256), 0, st, d, per_cta) : launch_kernel(linear_thin_kernel<32>, grid, dim3(256), 0, st, d, per_cta));
      VY_LAUNCH_OK();
      count_launch();
      return VY_OK;
    }
    VY_CUDA_OK(launch_kernel(linear_tile_kernel, dim3((p->N + LT - 1) / LT, (p->M + LT - 1) / LT, batch), dim3(256), 0, st, d));
  }
  VY_LAUNCH_OK();
  count_launch();
  return VY_OK;
}

extern "C" int vy_unary(int64_t rows, int32_t cols, const void* x, int64_t ldx, int32_t x_dtype, int32_t act, void* out,
                        int64_t ld_out, int32_t out_dtype, void* stream) {
  using namespace vy;
  if (!vy_device_ok()) {
    set_error("vy_unary: no sm_100 device (there is no CPU fallback)");
    return VY_ERR_NO_DEVICE;
  }
  VY_CHECK_ARG(rows > 0 && cols > 0 && x && out, "vy_unary: bad arguments");
  VY_CHECK_ARG(dtype_ok(x_dtype) && dtype_ok(out_dtype) && act >= VY_UACT_NONE && act <= VY_UACT_GELU_TANH, "vy_unary: bad dtype / act");
  long long blocks = (rows * cols + 255) / 256;
  if (blocks > 16LL * num_sms()) blocks = 16LL * num_sms();
  VY_CUDA_OK(launch_kernel(unary_kernel, dim3(static_cast<int>(blocks)), dim3(256), 0, static_cast<cudaStream_t>(stream),
                           static_cast<long long>(rows), cols, x, static_cast<long long>(ldx), x_dtype, act, out,
                           static_cast<long long>(ld_out), out_dtype));
  VY_LAUNCH_OK();
  count_launch();
  return VY_OK;
}

extern "C" int vy_embed_rows(int32_t rows, int32_t width, int32_t vocab, const int32_t* ids, const void* table, int64_t ld_table,
                             int32_t table_dtype, float scale, void* out, int64_t ld_out, int32_t out_dtype, void* stream) {
  using namespace vy;
  if (!vy_device_ok()) {
    set_error("vy_embed_rows: no sm_100 device (there is no CPU fallback)");
    return VY_ERR_NO_DEVICE;
  }
  VY_CHECK_ARG(rows > 0 && width > 0 && vocab > 0 && ids && table && out, "vy_embed_rows: bad arguments");
  VY_CHECK_ARG(dtype_ok(table_dtype) && dtype_ok(out_dtype), "vy_embed_rows: bad dtype");
  VY_CUDA_OK(launch_kernel(embed_rows_kernel, dim3(rows), dim3(128), 0, static_cast<cudaStream_t>(stream), rows, width, vocab, ids,
                           table, static_cast<long long>(ld_table), table_dtype, scale, out, static_cast<long long>(ld_out), out_dtype));
  VY_LAUNCH_OK();
  count_launch();
  return VY_OK;
}
