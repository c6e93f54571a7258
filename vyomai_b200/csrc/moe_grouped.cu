// Mixture of SwiGLU experts over many rows, each expert on the rows that are routed to it (vy_moe_grouped). Five launches and no host decision:
//   moe_plan_kernel      one CTA: the pairs (row, choice) placed by expert in row order, every expert's rows padded to whole tiles of 128; the tiles of both products
//   moe_spread_kernel    a warp per row writes its copies
//   gemm_kernel          twice, over the tiles of all experts (a tile's rows of A and of the result, its expert's rows or runs of k of the weights come from the plan)
//   moe_merge_kernel     a row's results, weighted and summed in the order of its choices
// A shared expert of m ff hidden columns is m experts that see every row in the first product and one with a contraction of m segments in the second.
// Rows that fill up tiles are never written: what they hold meets no other row. 4059 rows, 28 experts of 256 and a shared one of 512, top 4 of 32 (4 identity), width 1024: all experts
// over all rows 118 + 29 + 47 us, here 10 + 8 + 40 + 27 + 24; 2786 rows of width 2048 259 + 44 + 132, here 189. The first product is bound by its tiles' loads and write-back (190
// tiles of rows on 148 SMs), the second and the sum by the bytes of the fp32 results, 83 MB written and read.
#include "gemm_kernel.cuh"

namespace vy {

constexpr int MG_TILE = 128, MG_T = 1024, MG_MAX_EXPERTS = 256;

struct MoeGroupedDev {
  int rows, experts, top, width, ff, shared;   // shared: the shared expert's hidden columns over ff
  int cap, rows_pad;                           // rows of the routed part, of the shared part
  const int* idx; const float* weight;
  const __nv_bfloat16* h; long long ldh;
  const float* gate; long long ld_gate;
  float* out; long long ld_out;
  int* pos;        // [rows, top] row of the copies, -1: none
  int4* up_tiles; int4* down_tiles; int* counts;   // counts: tiles of the first product, of the second
  __nv_bfloat16* copies; float* part;
};

// A warp owns a run of the pairs: it counts them per expert, and after a scan over the warps' counts places them 32 at a time, where lanes that hold the same expert find one another
__global__ void __launch_bounds__(MG_T) moe_plan_kernel(const __grid_constant__ MoeGroupedDev d) {
  pdl_trigger();
  pdl_wait();
  __shared__ int counts[MG_T / 32][MG_MAX_EXPERTS];
  __shared__ int first[MG_MAX_EXPERTS + 1], tiles[MG_MAX_EXPERTS + 1];   // an expert's first row, its first tile
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int pairs = d.rows * d.top, run = (pairs + MG_T - 1) / MG_T * 32, p0 = min(warp * run, pairs), p1 = min(p0 + run, pairs);
  for (int e = lane; e < d.experts; e += 32) counts[warp][e] = 0;
  __syncwarp();
  const auto walk = [&](auto&& found) {
    for (int b0 = p0; b0 < p1; b0 += 32 * 8) {
      int es[8];   // on their way at once
#pragma unroll
      for (int u = 0; u < 8; ++u) es[u] = b0 + 32 * u + lane < p1 ? d.idx[b0 + 32 * u + lane] : -1;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = b0 + 32 * u + lane, e = es[u];
        const bool routed = e >= 0 && e < d.experts;
        unsigned same = __ballot_sync(0xffffffffu, routed);   // lanes with this lane's expert, a bit at a time: the instruction for it goes through the values one by one (24 us a launch for 8)
        for (int bit = 1; bit < d.experts; bit <<= 1) {
          const unsigned set = __ballot_sync(0xffffffffu, e & bit);
          same &= e & bit ? set : ~set;
        }
        const int rank = __popc(same & ((1u << lane) - 1u));
        found(i, e, routed, rank, routed ? counts[warp][e] : 0);
        __syncwarp();
        if (routed && rank == 0) counts[warp][e] += __popc(same);
        __syncwarp();
      }
    }
  };
  for (int b0 = p0 + lane; b0 < p1; b0 += 32 * 8) {
    int es[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) es[u] = b0 + 32 * u < p1 ? d.idx[b0 + 32 * u] : -1;
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (es[u] >= 0 && es[u] < d.experts) atomicAdd(&counts[warp][es[u]], 1);
  }
  __syncthreads();
  for (int e = t; e < d.experts; e += MG_T) {   // exclusive sums over the warps; the expert's number of pairs
    int at = 0;
    for (int w = 0; w < MG_T / 32; ++w) {
      const int c = counts[w][e];
      counts[w][e] = at;
      at += c;
    }
    tiles[e] = (at + MG_TILE - 1) / MG_TILE;
  }
  __syncthreads();
  if (warp == 0) {   // exclusive sums over the experts
    int before = 0;
    for (int e0 = 0; e0 < d.experts; e0 += 32) {
      const int e = e0 + lane, mine = e < d.experts ? tiles[e] : 0;
      int x = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (e < d.experts) {
        first[e] = MG_TILE * (before + x - mine);
        tiles[e] = before + x - mine;
      }
      before += __shfl_sync(0xffffffffu, x, 31);
    }
    if (lane == 0) tiles[d.experts] = before;
  }
  __syncthreads();
  walk([&](int i, int e, bool routed, int rank, int at) {
    if (i < p1) d.pos[i] = routed ? first[e] + at + rank : -1;
  });
  // Tiles: the routed experts', then the shared one's. Rows of the hidden activations: as the copies', the shared part once per ff columns
  const int routed = tiles[d.experts], per = d.rows_pad / MG_TILE;
  for (int i = t; i < routed; i += MG_T) {
    int lo = 0, hi = d.experts - 1;   // the last expert whose first tile is at most i (experts without rows share theirs with the next one)
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (tiles[mid] <= i) lo = mid;
      else hi = mid - 1;
    }
    d.up_tiles[i] = make_int4(i * MG_TILE, i * MG_TILE, lo * 2 * d.ff, 1);
    d.down_tiles[i] = make_int4(i * MG_TILE, i * MG_TILE, lo, 1);
  }
  if (d.shared > 0) {
    for (int i = t; i < d.shared * per; i += MG_T)
      d.up_tiles[routed + i] = make_int4(d.cap + i % per * MG_TILE, d.cap + i * MG_TILE, (d.experts + i / per) * 2 * d.ff, 1);
    for (int i = t; i < per; i += MG_T) d.down_tiles[routed + i] = make_int4(d.cap + i * MG_TILE, d.cap + i * MG_TILE, d.experts, d.shared);
  }
  if (t == 0) {
    d.counts[0] = routed + d.shared * per;
    d.counts[1] = routed + (d.shared > 0 ? per : 0);
  }
}

__global__ void __launch_bounds__(256) moe_spread_kernel(const __grid_constant__ MoeGroupedDev d) {
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= d.rows) return;
  const uint4* from = reinterpret_cast<const uint4*>(d.h + row * d.ldh);
  const int quads = d.width / 8;
  for (int c0 = lane; c0 < quads; c0 += 128) {
    uint4 x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c0 + 32 * u < quads) x[u] = from[c0 + 32 * u];
    for (int k = 0; k <= d.top; ++k) {
      const int to = k < d.top ? d.pos[row * d.top + k] : d.shared > 0 ? d.cap + row : -1;
      if (to < 0) continue;
      uint4* o = reinterpret_cast<uint4*>(d.copies + static_cast<long long>(to) * d.width);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c0 + 32 * u < quads) o[c0 + 32 * u] = x[u];
    }
  }
}

// Bound by the bytes of the results, read once. The rows of up to eight choices are on their way at once
__global__ void __launch_bounds__(256) moe_merge_kernel(const __grid_constant__ MoeGroupedDev d) {
  pdl_trigger();
  pdl_wait();
  const int per_row = d.width / 4;
  const long long i = blockIdx.x * 256LL + threadIdx.x;
  if (i >= static_cast<long long>(d.rows) * per_row) return;
  const int row = static_cast<int>(i / per_row), c = static_cast<int>(i % per_row) * 4;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k0 = 0; k0 < d.top; k0 += 8) {
    float4 x[8];
    float w[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int at = k0 + u < d.top ? d.pos[row * d.top + k0 + u] : -1;
      w[u] = at >= 0 ? d.weight[row * d.top + k0 + u] : 0.f;
      x[u] = at >= 0 ? *reinterpret_cast<const float4*>(d.part + static_cast<long long>(at) * d.width + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      acc.x = fmaf(w[u], x[u].x, acc.x);
      acc.y = fmaf(w[u], x[u].y, acc.y);
      acc.z = fmaf(w[u], x[u].z, acc.z);
      acc.w = fmaf(w[u], x[u].w, acc.w);
    }
  }
  if (d.shared > 0) {
    const float s = d.gate ? 1.f / (1.f + expf(-d.gate[row * d.ld_gate])) : 1.f;
    const float4 x = *reinterpret_cast<const float4*>(d.part + static_cast<long long>(d.cap + row) * d.width + c);
    acc = make_float4(fmaf(s, x.x, acc.x), fmaf(s, x.y, acc.y), fmaf(s, x.z, acc.z), fmaf(s, x.w, acc.w));
  }
  *reinterpret_cast<float4*>(d.out + row * d.ld_out + c) = acc;
}

namespace {

struct MoeLayout {
  long long cap, rows_pad, hidden_rows, part_rows, tiles, copies_at, hidden_at, part_at, pos_at, up_at, down_at, counts_at, bytes;
};
bool moe_layout(MoeLayout& l, long long rows, int experts, int top, int width, int ff, int shared_ff) {
  if (rows <= 0 || experts <= 0 || experts > MG_MAX_EXPERTS || top <= 0 || width <= 0 || ff <= 0 || width % 8 || ff % 8 || shared_ff < 0 || shared_ff % ff || rows * top > (1LL << 24)) return false;
  const long long shared = shared_ff / ff, pairs = rows * top;
  // at most one tile short of full per expert that has rows
  l.cap = (pairs + static_cast<long long>(pairs < experts ? pairs : experts) * (MG_TILE - 1)) / MG_TILE * MG_TILE;
  l.rows_pad = shared ? (rows + MG_TILE - 1) / MG_TILE * MG_TILE : 0;
  l.part_rows = l.cap + l.rows_pad;
  l.hidden_rows = l.cap + shared * l.rows_pad;
  l.tiles = l.hidden_rows / MG_TILE;
  long long at = 0;
  const auto take = [&](long long bytes) { const long long a = at; at += (bytes + 127) / 128 * 128; return a; };
  l.copies_at = take(l.part_rows * width * 2);
  l.hidden_at = take(l.hidden_rows * ff * 2);
  l.part_at = take(l.part_rows * width * 4);
  l.pos_at = take(pairs * 4);
  l.up_at = take(l.tiles * 16);
  l.down_at = take(l.tiles * 16);
  l.counts_at = take(8);
  l.bytes = at;
  return at <= (2LL << 30) && l.hidden_rows < (1 << 30);
}

template <int BN, int WB>
int launch_grouped(const GemmDev& g, const void* a, long long a_rows, long long lda, int ka, const void* b, long long b_rows, long long ldb, int kb, void* out, long long out_rows, int out_cols,
                   long long most_tiles, cudaStream_t st) {
  using Cfg = GemmCfg<__nv_bfloat16, BN>;
  CUtensorMap ta, tb, tout;
  int rc = get_tmap_2d(&ta, VY_BF16, a, ka, a_rows, lda * 2, Cfg::BK, Cfg::BM);
  if (rc == VY_OK && WB == WB_GATED_GROUPED) rc = get_tmap_2d(&tb, VY_BF16, b, kb, b_rows, ldb * 2, Cfg::BK, BN);
  if (rc == VY_OK && WB == WB_F32_GROUPED) {   // [row][expert][ff]: what a contraction reads past an expert's ff is zero, not the next expert's, whose infinity times zero would be a NaN
    const uint64_t dims[3] = {static_cast<uint64_t>(ka), static_cast<uint64_t>(kb / ka), static_cast<uint64_t>(b_rows)}, strides[3] = {0, static_cast<uint64_t>(ka) * 2, static_cast<uint64_t>(ldb) * 2};
    const uint32_t box[3] = {Cfg::BK, 1, BN};
    rc = get_tensor_map_cached(&tb, VY_BF16, 3, b, dims, strides, box, 1);
  }
  if (rc == VY_OK) rc = WB == WB_F32_GROUPED ? get_tmap_2d(&tout, VY_F32, out, out_cols, out_rows, static_cast<uint64_t>(out_cols) * 4, 16, 32, 3)
                                             : get_tmap_2d(&tout, VY_BF16, out, out_cols, out_rows, static_cast<uint64_t>(out_cols) * 2, 32, 32, 3);
  if (rc != VY_OK) return rc;
  auto kern = gemm_kernel<__nv_bfloat16, BN, false, false, false, WB>;
  static std::atomic<unsigned long long> allowed{0};
  VY_CUDA_OK(allow_smem(kern, allowed));
  const long long units = most_tiles * ((g.N + BN - 1) / BN);
  VY_CUDA_OK(launch_kernel(kern, dim3(static_cast<unsigned>(units < num_sms() ? units : num_sms())), dim3(GEMM_THREADS), Cfg::SMEM_BYTES, st, ta, tb, tout, ta, g));
  VY_LAUNCH_OK();
  count_launch();
  return VY_OK;
}

}  // namespace
}  // namespace vy

extern "C" int64_t vy_moe_grouped_bytes(int32_t rows, int32_t experts, int32_t top, int32_t width, int32_t ff, int32_t shared_ff) {
  vy::MoeLayout l;
  return vy::moe_layout(l, rows, experts, top, width, ff, shared_ff) ? l.bytes : 0;
}

extern "C" int vy_moe_grouped(const VyMoeGrouped* p) {
  using namespace vy;
  VY_CHECK_ARG(p != nullptr, "vy_moe_grouped: null params");
  if (!vy_device_ok()) {
    set_error("vy_moe_grouped: no sm_100 device (there is no CPU fallback)");
    return VY_ERR_NO_DEVICE;
  }
  if (poison_raised("vy_moe_grouped")) return VY_ERR_CUDA;
  MoeLayout l;
  VY_CHECK_ARG(moe_layout(l, p->rows, p->experts, p->top, p->width, p->ff, p->shared_ff), "vy_moe_grouped: rows %d, experts %d, top %d, width %d, ff %d, shared_ff %d", p->rows, p->experts,
               p->top, p->width, p->ff, p->shared_ff);
  const auto aligned = [](const void* q, long long ld, int es) { return q && reinterpret_cast<uintptr_t>(q) % 16 == 0 && ld * es % 16 == 0; };
  VY_CHECK_ARG(p->idx && p->weight && aligned(p->h, p->ldh, 2) && aligned(p->up, p->ld_up, 2) && aligned(p->down, p->ld_down, 2) && aligned(p->out, p->ld_out, 4) && p->ldh >= p->width &&
                   p->ld_up >= p->width && p->ld_out >= p->width && p->ld_down >= static_cast<long long>(p->experts) * p->ff + p->shared_ff, "vy_moe_grouped: bad tensors");
  VY_CHECK_ARG(p->workspace && reinterpret_cast<uintptr_t>(p->workspace) % 128 == 0 && p->workspace_bytes >= l.bytes, "vy_moe_grouped: the workspace holds vy_moe_grouped_bytes(...) bytes");
  char* ws = static_cast<char*>(p->workspace);
  MoeGroupedDev d;
  d.rows = p->rows; d.experts = p->experts; d.top = p->top; d.width = p->width; d.ff = p->ff; d.shared = p->shared_ff / p->ff;
  d.cap = static_cast<int>(l.cap); d.rows_pad = static_cast<int>(l.rows_pad);
  d.idx = p->idx; d.weight = p->weight;
  d.h = static_cast<const __nv_bfloat16*>(p->h); d.ldh = p->ldh;
  d.gate = p->shared_gate; d.ld_gate = p->ld_gate;
  d.out = p->out; d.ld_out = p->ld_out;
  d.pos = reinterpret_cast<int*>(ws + l.pos_at);
  d.up_tiles = reinterpret_cast<int4*>(ws + l.up_at);
  d.down_tiles = reinterpret_cast<int4*>(ws + l.down_at);
  d.counts = reinterpret_cast<int*>(ws + l.counts_at);
  d.copies = reinterpret_cast<__nv_bfloat16*>(ws + l.copies_at);
  d.part = reinterpret_cast<float*>(ws + l.part_at);
  void* hidden = ws + l.hidden_at;
  cudaStream_t st = static_cast<cudaStream_t>(p->stream);
  VY_CUDA_OK(launch_kernel(moe_plan_kernel, dim3(1), dim3(MG_T), 0, st, d));
  VY_LAUNCH_OK();
  VY_CUDA_OK(launch_kernel(moe_spread_kernel, dim3((p->rows + 7) / 8), dim3(256), 0, st, d));
  VY_LAUNCH_OK();
  count_launch(2);
  GemmDev g;
  memset(&g, 0, sizeof(g));
  if (!poison_ref(&g.poison)) return VY_ERR_CUDA;
  g.epi = VY_EPI_LINEAR; g.vec_ok = 1; g.k_splits = 1; g.tma_store = 1; g.out_scale = 1.f;
  g.M = static_cast<int>(l.hidden_rows); g.N = 2 * p->ff; g.K = p->width; g.act = VY_ACT_SWIGLU;
  g.groups = d.up_tiles; g.group_count = d.counts; g.seg_k = p->width;
  g.out = hidden; g.ld_out = p->ff; g.out_dtype = VY_BF16;
  const long long up_rows = static_cast<long long>(p->experts) * 2 * p->ff + 2 * p->shared_ff, down_cols = static_cast<long long>(p->experts) * p->ff + p->shared_ff;
  // 128 columns per tile, which spread better over the SMs than 256 (40 / 49 us at the header's size, 29 / 37 for 8000 rows of width 512, 78 / 77 for 2786 of 2048); below, where a tile is
  // mostly write-back, they are alike (27 / 27, 20 / 20, 48 / 46)
  int rc = launch_grouped<128, WB_GATED_GROUPED>(g, d.copies, l.part_rows, p->width, p->width, p->up, up_rows, p->ld_up, p->width, hidden, l.hidden_rows, p->ff, l.tiles, st);
  if (rc != VY_OK) return rc;
  g.M = static_cast<int>(l.part_rows); g.N = p->width; g.K = p->ff; g.act = VY_ACT_NONE;
  g.groups = d.down_tiles; g.group_count = d.counts + 1; g.seg_k = p->ff; g.seg_rows = d.rows_pad;
  g.out = d.part; g.ld_out = p->width; g.out_dtype = VY_F32;
  rc = launch_grouped<256, WB_F32_GROUPED>(g, hidden, l.hidden_rows, p->ff, p->ff, p->down, p->width, p->ld_down, static_cast<int>(down_cols), d.part, l.part_rows, p->width, l.tiles, st);
  if (rc != VY_OK) return rc;
  const long long quads = static_cast<long long>(p->rows) * (p->width / 4);
  VY_CUDA_OK(launch_kernel(moe_merge_kernel, dim3(static_cast<unsigned>((quads + 255) / 256)), dim3(256), 0, st, d));
  VY_LAUNCH_OK();
  count_launch();
  return VY_OK;
}
