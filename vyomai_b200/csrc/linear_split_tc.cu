// fp32 products of many rows on tcgen05 in fp32 precision (split_mma.cuh), in two launches:
//   linear_halves_kernel      a warp per row of either operand: its largest entry, then its two fp16 halves, filled up with zeros to a multiple of 64
//   linear_split_tc_kernel    128 x 128 results per tile. A warp brings stages of 64 k (both halves of both operands), one sends off the products - the small ones and hi hi have an
//                             accumulator each - and eight add what 128 k gave to fp32 registers: chains of 8 and 16 steps
// What linear_split_kernel does over again in every tile, the splitting, is done once; a tile is then bound by its products (12 of 128 x 128 x 16 per 64 k) and by 9 us around them. us, that
// kernel / here: 1600 x 3072, K 1024 183 / 6 + 51; 1963 x 5152, K 1024 336 / 10 + 87; 700 x 10304, K 2048 452 / 30 + 115; 8192 x 1024, K 1024 281 / 13 + 69; error against 64 bits 1.55e-7 / 1.44e-7.
// Splitting in the kernel (sixteen warps beside sixteen that add): 140 at the first size, bound by the splitting warps.
#include "linear_plain.cuh"

namespace vy {
namespace {

constexpr int ST_T = 128, ST_K = 64, ST_STAGES = 3, ST_PART = ST_T * 128, ST_STAGE = 4 * ST_PART;   // a stage: A hi | A lo | W hi | W lo, 128-byte swizzle
constexpr int ST_DRAIN = 2;                                  // stages per addition to the registers
constexpr int ST_EPI = 8, ST_THREADS = 32 * (ST_EPI + 2);
constexpr int ST_LD = 20, ST_OUT = 32 * ST_LD + 64;          // floats a warp turns 32 rows of 16 results in; the units of its 64 columns
constexpr int ST_SMEM = ST_STAGES * ST_STAGE + ST_EPI * ST_OUT * 4 + 128;

struct HalvesDev {
  const float* A; const float* W; long long lda, ldw;
  int M, N, K, kp;
  __half* a_hi; __half* a_lo; __half* w_hi; __half* w_lo;
  float* units;   // of A's rows, then of W's: 0 for a row of zeros, NaN for one that holds a NaN
};

__global__ void __launch_bounds__(256) linear_halves_kernel(const __grid_constant__ HalvesDev d) {
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= d.M + d.N) return;
  const bool isa = row < d.M;
  const int r = isa ? row : row - d.M;
  const float* p = isa ? d.A + static_cast<long long>(r) * d.lda : d.W + static_cast<long long>(r) * d.ldw;
  __half* hi = (isa ? d.a_hi : d.w_hi) + static_cast<long long>(r) * d.kp;
  __half* lo = (isa ? d.a_lo : d.w_lo) + static_cast<long long>(r) * d.kp;
  unsigned top = 0u;   // as bits: a NaN's are the largest
  for (int k0 = 4 * lane; k0 < d.K; k0 += 512) {
    float4 x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      x[u] = k0 + 128 * u < d.K ? *reinterpret_cast<const float4*>(p + k0 + 128 * u) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      top = max(top, max(max(__float_as_uint(fabsf(x[u].x)), __float_as_uint(fabsf(x[u].y))), max(__float_as_uint(fabsf(x[u].z)), __float_as_uint(fabsf(x[u].w)))));
  }
  const float m = __uint_as_float(__reduce_max_sync(0xffffffffu, top));
  const int e = split_exponent(m);
  const float sc = split_scale(e);
  if (lane == 0) d.units[row] = m != m ? m : m > 0.f ? pow2i(e - SPLIT_TOP) : 0.f;
  for (int k0 = 8 * lane; k0 < d.kp; k0 += 512) {
    float4 x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = k0 + 256 * (u >> 1) + 4 * (u & 1);
      x[u] = k < d.K ? *reinterpret_cast<const float4*>(p + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (k0 + 256 * u >= d.kp) break;
      const float4 a = x[2 * u], b = x[2 * u + 1];
      uint4 h, l;
      split2(a.x * sc, a.y * sc, h.x, l.x);
      split2(a.z * sc, a.w * sc, h.y, l.y);
      split2(b.x * sc, b.y * sc, h.z, l.z);
      split2(b.z * sc, b.w * sc, h.w, l.w);
      *reinterpret_cast<uint4*>(hi + k0 + 256 * u) = h;
      *reinterpret_cast<uint4*>(lo + k0 + 256 * u) = l;
    }
  }
}

// 32 rows x 16 columns of results that lack their columns' units: those that are too small beside their rows' largest entries, or not finite (but where a row or column has a NaN and its results
// with it: 40 rows of NaN in 4000 x 1024, K 512, 1020 us otherwise), computed again, then out. A function, since code that is
// unrolled for every run of columns comes from memory (33 x 64, K 256: 23 us instead of 10)
static __device__ __noinline__ void finish(const LinDev& d, float* mine, const float* uw, float small, int m0, int n0) {
  const int lane = threadIdx.x & 31;
  unsigned again = 0u;   // results of this lane's row that are computed again
#pragma unroll 1
  for (int i = 0; i < 16; i += 4) {
    const float4 u = *reinterpret_cast<const float4*>(uw + i), v = *reinterpret_cast<const float4*>(mine + lane * ST_LD + i);
    const float x[4] = {v.x * u.x, v.y * u.y, v.z * u.z, v.w * u.w}, us[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (!(fabsf(x[k]) >= small * us[k] && fabsf(x[k]) < INFINITY)) again |= 1u << (i + k);
    *reinterpret_cast<float4*>(mine + lane * ST_LD + i) = make_float4(x[0], x[1], x[2], x[3]);
  }
  if (m0 + lane >= d.M || small != small) again = 0u;
  if (again)
#pragma unroll 1
    for (int i = 0; i < 16; ++i)
      if (uw[i] != uw[i]) again &= ~(1u << i);
  if (d.N - n0 < 16) again &= d.N > n0 ? (1u << (d.N - n0)) - 1u : 0u;
  for (unsigned rows = __ballot_sync(0xffffffffu, again != 0u); rows; rows &= rows - 1) {
    const int src = __ffs(rows) - 1;
    for (unsigned cols = __shfl_sync(0xffffffffu, again, src); cols; cols &= cols - 1) {
      const int i = __ffs(cols) - 1;
      const float z = lin_dot(static_cast<const float*>(d.A) + static_cast<long long>(m0 + src) * d.lda, static_cast<const float*>(d.W) + static_cast<long long>(n0 + i) * d.ldw, d.K);
      if (lane == src) mine[lane * ST_LD + i] = z;
    }
  }
  __syncwarp();
  const int n = n0 + 4 * (lane & 3);
  const bool quad = d.out_dt == VY_F32 && !d.addend && n + 3 < d.N && d.ld_out % 4 == 0 && reinterpret_cast<uintptr_t>(d.out) % 16 == 0;
  float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
  if (quad && d.bias) b = make_float4(ld_as_float(d.bias, d.bias_dt, n), ld_as_float(d.bias, d.bias_dt, n + 1), ld_as_float(d.bias, d.bias_dt, n + 2), ld_as_float(d.bias, d.bias_dt, n + 3));
#pragma unroll 1
  for (int r = lane >> 2; r < 32 && m0 + r < d.M; r += 8) {
    float4 v = *reinterpret_cast<const float4*>(mine + r * ST_LD + 4 * (lane & 3));
    if (quad) {
      v = make_float4(v.x + b.x, v.y + b.y, v.z + b.z, v.w + b.w);
      if (d.act != VY_UACT_NONE) v = make_float4(uact(v.x, d.act), uact(v.y, d.act), uact(v.z, d.act), uact(v.w, d.act));
      *reinterpret_cast<float4*>(static_cast<float*>(d.out) + static_cast<long long>(m0 + r) * d.ld_out + n) = make_float4(v.x * d.scale, v.y * d.scale, v.z * d.scale, v.w * d.scale);
    } else {
      const float y[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (n + k < d.N) lin_store(d, m0 + r, n + k, y[k]);
    }
  }
  __syncwarp();
}

__global__ void __launch_bounds__(ST_THREADS, 1)
linear_split_tc_kernel(const __grid_constant__ CUtensorMap a_map, const __grid_constant__ CUtensorMap w_map, const __grid_constant__ LinDev d, const float* units, int stages, const __grid_constant__ PoisonRef poison) {
  pdl_trigger();
  extern __shared__ __align__(1024) unsigned char st_smem[];
  float* turn = reinterpret_cast<float*>(st_smem + ST_STAGES * ST_STAGE);   // [warp][32 rows][16 results]
  uint64_t* bars = reinterpret_cast<uint64_t*>(turn + ST_EPI * ST_OUT);
  uint64_t *full = bars, *free_ = bars + ST_STAGES, *dfull = bars + 2 * ST_STAGES, *dfree = dfull + 2, *done = dfree + 2;
  uint32_t* tmem_at = reinterpret_cast<uint32_t*>(done + 1);
  int* issued = reinterpret_cast<int*>(tmem_at + 1);   // [ST_STAGES] loads sent for
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  if (warp == 0) {
    if (lane == 0) {
      for (int i = 0; i < ST_STAGES; ++i) {
        mbar_init(&full[i], 1);
        mbar_init(&free_[i], 1);
        issued[i] = 0;
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&dfull[i], 1);
        mbar_init(&dfree[i], ST_EPI);
      }
      mbar_init(done, 1);
      fence_mbar_init();
    }
    __syncwarp();
    tmem_alloc(tmem_at, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_at;   // [2][hi hi, small][128 columns]
  pdl_wait();
  const int n_tiles = (d.N + ST_T - 1) / ST_T, tiles = n_tiles * ((d.M + ST_T - 1) / ST_T), drains = (stages + ST_DRAIN - 1) / ST_DRAIN;
  bool alive = true;
  if (warp == 0) {
    uint32_t it = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const int m0 = tile / n_tiles * ST_T, n0 = tile % n_tiles * ST_T;
      for (int k = 0; k < stages; ++k, ++it) {
        const uint32_t b = it % ST_STAGES;
        if (it >= ST_STAGES) alive = mbar_wait_soft(&free_[b], (it / ST_STAGES - 1) & 1, poison) && alive;
        if (alive && elect_one_sync()) {
          unsigned char* st = st_smem + b * ST_STAGE;
          ++issued[b];
          mbar_arrive_expect_tx(&full[b], ST_STAGE);
          tma_load_2d(st, &a_map, &full[b], k * ST_K, m0);   // rows past the last one are the lo halves of others: their results are not used
          tma_load_2d(st + ST_PART, &a_map, &full[b], k * ST_K, d.M + m0);
          tma_load_2d(st + 2 * ST_PART, &w_map, &full[b], k * ST_K, n0);
          tma_load_2d(st + 3 * ST_PART, &w_map, &full[b], k * ST_K, d.N + n0);
        }
        __syncwarp();
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t id = make_idesc(0, ST_T, ST_T, 0, 0);
    const uint64_t kmaj = make_smem_desc_sw128(smem_u32(st_smem), 16, 1024);
    uint32_t it = 0, turns = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x)
      for (int k = 0; k < stages; ++k, ++it) {
        const uint32_t b = it % ST_STAGES;
        const bool first = k % ST_DRAIN == 0, last = k % ST_DRAIN == ST_DRAIN - 1 || k == stages - 1;
        if (first && turns >= 2) alive = mbar_wait_soft(&dfree[turns & 1], ((turns >> 1) - 1) & 1, poison) && alive;
        alive = mbar_wait_soft(&full[b], (it / ST_STAGES) & 1, poison) && alive;
        tc_fence_after();
        if (alive && elect_one_sync()) {
          const uint32_t D = tmem + (turns & 1) * 2 * ST_T;
          const uint64_t ah = kmaj + (b * ST_STAGE >> 4), al = ah + (ST_PART >> 4), wh = al + (ST_PART >> 4), wl = wh + (ST_PART >> 4);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            umma_f16(D + ST_T, al + 2 * j, wh + 2 * j, id, !(first && j == 0));
            umma_f16(D + ST_T, ah + 2 * j, wl + 2 * j, id, 1);
            umma_f16(D, ah + 2 * j, wh + 2 * j, id, !(first && j == 0));
          }
          umma_commit(&free_[b]);
          if (last) umma_commit(&dfull[turns & 1]);
        }
        __syncwarp();
        if (last) ++turns;
      }
  } else {
    const int e = warp - 2, quarter = warp & 3, c0 = 64 * (e >> 2), row = quarter * 32 + lane;   // row of the tile, columns c0 ..
    const uint32_t at = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + c0;
    float* mine = turn + e * ST_OUT;
    uint32_t turns = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const int m0 = tile / n_tiles * ST_T, n0 = tile % n_tiles * ST_T, m = m0 + row;
      const float ua = m < d.M ? units[m] : 0.f;
      float* uw = mine + 32 * ST_LD;
      __syncwarp();
#pragma unroll
      for (int i = lane; i < 64; i += 32) uw[i] = n0 + c0 + i < d.N ? units[d.M + n0 + c0 + i] : 0.f;
      __syncwarp();
      f32x2 acc[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) acc[i] = pair(0.f);
#pragma unroll 1
      for (int t = 0; t < drains; ++t, ++turns) {
        const uint32_t b = turns & 1;
        const int steps = min(ST_DRAIN, stages - t * ST_DRAIN) * 4;
        const f32x2 cut = pair(0.5f * (steps + 1) * SPLIT_CUT);
        alive = mbar_wait_soft(&dfull[b], (turns >> 1) & 1, poison) && alive;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 64; c += 16) {
          uint32_t y[16], z[16];
          tmem_ld_x16(at + b * 2 * ST_T + c, y);
          tmem_ld_x16(at + b * 2 * ST_T + ST_T + c, z);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; i += 2) {   // split_sum
            const f32x2 hi = pair_bits(y[i], y[i + 1]);
            acc[(c + i) / 2] = add2(acc[(c + i) / 2], fma2(fma2(hi, cut, pair_bits(z[i], z[i + 1])), pair(LO_UNIT), hi));
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&dfree[b]);
      }
#pragma unroll
      for (int c = 0; c < 64; c += 16) {
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          const float2 p = unpair(mul2(acc[(c + i) / 2], pair(ua))), q = unpair(mul2(acc[(c + i) / 2 + 1], pair(ua)));
          *reinterpret_cast<float4*>(mine + lane * ST_LD + i) = make_float4(p.x, p.y, q.x, q.y);
        }
        finish(d, mine, uw + c, LS_SMALL * ua, m0 + quarter * 32, n0 + c0 + c);
      }
    }
  }
  tc_fence_before();
  if (__syncthreads_or(!alive) && warp == 1) {   // a wait has timed out: what is in flight ends before the memory is given back
    if (elect_one_sync()) umma_commit(done);
    __syncwarp();
    for (uint32_t spins = 0; spins < (1u << 20) && !mbar_try_wait(done, 0); ++spins) {}
    mbar_drain(full, issued, ST_STAGES);
  }
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

int padded(int K) { return (K + ST_K - 1) / ST_K * ST_K; }

}  // namespace

// Where the tiled form (64 x 64, two CTAs per SM) has a CTA for every SM and its estimated time (us) is the longer one. Below, two launches and a tile's start cost more than the splitting saved,
// for the host too: 300 x 1024, K 1024 (80 CTAs) 27 / 23. Splitting ahead pays for results that many tiles of an operand share: it reads and writes both operands, and the tiles read them again, which
// thin results over many rows do not repay. us, tiled / here: K 256 1000 x 1000 (256 CTAs) 15 / 20, 1300 x 1000 23 / 20, 20000 x 30 23 / 37; 512 600 x 1000 (160) 24 / 19, 2000 x 1000 47 / 24, 1000 x
// 512 (128) 17 / 18, 20000 x 16 36 / 37, 40000 x 8 51 / 62; 580 129 x 3300 27 / 22, 3300 x 129 (rows of results not on 16 bytes) 30 / 34; 1024 600 x 1000 41 / 25, 33 x 9700 41 / 29, 9700 x 33 43 / 38,
// 100000 x 8 201 / 245; 2048 40 x 16000 77 / 82; 4096 65 x 4800 143 / 80
long long linear_split_bytes(int M, int N, int K) {
  const long long ctas = ((M + 63LL) / 64) * ((N + 63LL) / 64), tiles = ((M + ST_T - 1LL) / ST_T) * ((N + ST_T - 1LL) / ST_T);
  if (M <= 32 || N <= 0 || K < 256 || ctas <= num_sms()) return 0;
  const double sms = num_sms(), share = ctas / (2.0 * sms), halves = (static_cast<double>(M) + N) * K * 4.0, rounds = ceil(tiles / sms);
  const double tiled = (share > 1.0 ? share + 0.4 : 1.0) * (5.5 + 0.0345 * K);
  const double split = 9.5 + 2.0 * halves / 7e6 + (halves > 1e8 ? halves / 6e6 : 0.0) /* no longer in L2 */ + 3.0 + 0.0094 * K + (rounds - 1.0) * (3.0 + 0.0127 * K) + (N % 4 ? 6.0 : 0.0);
  if (split >= tiled) return 0;
  const long long rows = static_cast<long long>(M) + N, bytes = (rows * padded(K) * 4 + 127) / 128 * 128 + rows * 4;
  return bytes <= (1LL << 30) ? bytes : 0;
}

cudaError_t launch_linear_split_tc(const LinDev& d, void* ws, cudaStream_t st) {
  HalvesDev h;
  h.A = static_cast<const float*>(d.A); h.W = static_cast<const float*>(d.W); h.lda = d.lda; h.ldw = d.ldw;
  h.M = d.M; h.N = d.N; h.K = d.K; h.kp = padded(d.K);
  const long long a = static_cast<long long>(d.M) * h.kp, w = static_cast<long long>(d.N) * h.kp;
  h.a_hi = static_cast<__half*>(ws);
  h.a_lo = h.a_hi + a;
  h.w_hi = h.a_lo + a;
  h.w_lo = h.w_hi + w;
  h.units = reinterpret_cast<float*>(static_cast<char*>(ws) + (4 * (a + w) + 127) / 128 * 128);
  static std::atomic<unsigned long long> allowed{0};
  cudaError_t e = allow_smem(linear_split_tc_kernel, allowed);
  if (e != cudaSuccess) return e;
  PoisonRef poison = {};
  if (!poison_ref(&poison)) return cudaErrorMemoryAllocation;
  CUtensorMap maps[2];
  for (int i = 0; i < 2; ++i) {   // hi halves, the lo ones behind
    const uint64_t dims[2] = {static_cast<uint64_t>(h.kp), 2 * static_cast<uint64_t>(i ? d.N : d.M)}, strides[2] = {0, static_cast<uint64_t>(h.kp) * 2};
    const uint32_t box[2] = {ST_K, ST_T};
    if (get_tensor_map_cached(&maps[i], VY_BF16, 2, i ? h.w_hi : h.a_hi, dims, strides, box, 1) != VY_OK) return cudaErrorInvalidValue;
  }
  e = launch_kernel(linear_halves_kernel, dim3((d.M + d.N + 7) / 8), dim3(256), 0, st, h);
  if (e != cudaSuccess) return e;
  const long long tiles = static_cast<long long>((d.M + ST_T - 1) / ST_T) * ((d.N + ST_T - 1) / ST_T);
  return launch_kernel(linear_split_tc_kernel, dim3(static_cast<unsigned>(tiles < num_sms() ? tiles : num_sms())), dim3(ST_THREADS), ST_SMEM, st, maps[0], maps[1], d, static_cast<const float*>(h.units), h.kp / ST_K, poison);
}

}  // namespace vy
