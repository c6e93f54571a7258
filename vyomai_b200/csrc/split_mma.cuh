// fp32 contractions on the tensor cores: every operand row is scaled by a power of two (exact) so that its largest entry lies in
// [2^12, 2^13), and each entry becomes two fp16 numbers, x = hi + 2^-11 lo. hi carries 11 significant bits and lo the next 11 or 12; kept 2^11
// times larger, lo stays a normal fp16 number as long as hi does. So the pair is off by at most 2^-23 |x| down to 2^24 below the row's largest
// entry, by 2^-22 |x| down to 2^27 below it, and by 2^-49 of that largest entry further down (lo itself stored instead: 2^-23 |x| only down to 2^14
// below, then 2^-38 of the largest). A product of two such rows is hi hi + 2^-11 (lo hi + hi lo) with fp32 accumulation; the dropped lo lo term is
// below 2^-22 of a product and random in sign. The two small products get an accumulator of their own (LO_UNIT undoes the 2^11), and an accumulator
// takes few steps before it is added to a longer sum in fp32 registers: a tensor-core accumulation does not round to nearest, and this keeps its
// share of the error below that of a serial fp32 FMA chain. Three 16-bit products run at a third of the 16-bit rate where fp32 FMAs run at an eighth
// of it (and need a shared-memory operand read per FMA).
#pragma once
#include <cuda_fp16.h>

#include <type_traits>

#include "vy_common.cuh"

namespace vy {

constexpr int SPLIT_TOP = 12;     // scaled rows have their largest entry in [2^SPLIT_TOP, 2^(SPLIT_TOP + 1))
constexpr float LO_UNIT = 0x1p-11f;   // a lo half is stored in this unit
// A tensor-core accumulation cuts off where fp32 rounds: a result is this share too small on average (in the unit of the small products' sums, to which it can be
// added: sum = (small + hi * cut) * LO_UNIT + hi). A sum of n accumulations loses (n + 1) / 2 such shares of its end value on average
constexpr float SPLIT_CUT = 0x1p-25f / LO_UNIT;
__device__ __forceinline__ float split_sum(float hi, float small, float cut) { return fmaf(fmaf(hi, cut, small), LO_UNIT, hi); }
constexpr int SPLIT_MIN_E = -100; // rows whose largest entry is below 2^-100 (all zero, for one) keep this exponent: scales stay finite

// exponent of a row's largest absolute value
__device__ __forceinline__ int split_exponent(float absmax) {
  const int e = static_cast<int>((__float_as_uint(absmax) >> 23) & 255u) - 127;
  return min(max(e, SPLIT_MIN_E), 127);
}
// 2^e for -126 <= e <= 127; 0 below
__device__ __forceinline__ float pow2i(int e) { return e < -126 ? 0.f : __uint_as_float(static_cast<unsigned>(e + 127) << 23); }
__device__ __forceinline__ float split_scale(int e) { return pow2i(SPLIT_TOP - e); }

__device__ __forceinline__ unsigned pack_h2(__half2 v) { return *reinterpret_cast<unsigned*>(&v); }
// two neighbouring entries -> their hi and lo halves (a is the lower address)
__device__ __forceinline__ void split2(float a, float b, unsigned& hi, unsigned& lo) {
  const __half2 h = __floats2half2_rn(a, b);
  const float2 f = __half22float2(h);
  hi = pack_h2(h);
  lo = pack_h2(__floats2half2_rn((a - f.x) * (1.f / LO_UNIT), (b - f.y) * (1.f / LO_UNIT)));
}

__device__ __forceinline__ unsigned smem_addr(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void ldsm_x4(unsigned (&r)[4], unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_t(unsigned (&r)[4], unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// 16 bytes global -> shared, asynchronous; zeros when !valid (the address must be a legal one all the same)
__device__ __forceinline__ void cp_async16(unsigned dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Byte offsets a lane hands to ldmatrix inside a [row][column] fp16 matrix with `row_bytes` (an odd multiple of 16) between rows:
// A operand, 16 rows x 16 columns: registers are a0 .. a3 of m16n8k16
__device__ __forceinline__ unsigned lane_a(int lane, int row_bytes) { return (lane & 15) * row_bytes + ((lane >> 4) << 4); }
// B operand stored [n][k], 16 n x 16 k: registers 0, 1 are (b0, b1) of the first 8 n, registers 2, 3 of the others
__device__ __forceinline__ unsigned lane_b(int lane, int row_bytes) { return ((lane & 7) + ((lane >> 4) << 3)) * row_bytes + (((lane >> 3) & 1) << 4); }
// B operand stored [k][n] (ldmatrix.trans), 16 k x 16 n: same registers
__device__ __forceinline__ unsigned lane_bt(int lane, int row_bytes) { return ((lane & 7) + (((lane >> 3) & 1) << 3)) * row_bytes + ((lane >> 4) << 4); }

// Rare forms as calls of their own: unrolled into every place that needs them they would push the kernels' loops out of the instruction cache
// (la_outputs_kernel: 4.8 of 9 stall cycles per instruction were instruction fetches)
// entries c .. c + 3 of a row of any type and alignment, zero past `width`
static __device__ __noinline__ float4 load4_any(const void* src, int dt, long long o, int c, int width) {
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
  x.x = ld_as_float(src, dt, o + c);
  if (c + 1 < width) x.y = ld_as_float(src, dt, o + c + 1);
  if (c + 2 < width) x.z = ld_as_float(src, dt, o + c + 2);
  if (c + 3 < width) x.w = ld_as_float(src, dt, o + c + 3);
  return x;
}
// the first `n` (of 2) values to entries at, at + 1
static __device__ __noinline__ void store2_any(void* dst, int dt, long long at, float a, float b, int n) {
  if (n > 0) st_from_float(dst, dt, at, a);
  if (n > 1) st_from_float(dst, dt, at + 1, b);
}

// Rows [0, rows) of a block of `src` as hi / lo planes (`row_bytes` between rows of a plane, columns zero-filled up to pad16, a
// multiple of 16 and at most MAXD), with 2^(a row's exponent - drop) in unit[row * ustep]. Row j starts at element off(j) of src or is all zero when
// off(j) < 0. Eight lanes share a row (coalesced 128-byte runs); a thread has the loads of U rows in flight before it uses any. vec: src
// is fp32, row starts and the width are multiples of 4 elements. map: applied to every entry read, not to the zeros that fill up rows. seen: given each row's largest entry.
struct SameValue {
  __device__ __forceinline__ float operator()(float x) const { return x; }
};
struct NotSeen {
  __device__ __forceinline__ void operator()(float) const {}
};
template <int NW, int MAXD, typename OffFn, typename MapFn = SameValue, typename SeenFn = NotSeen>
__device__ __forceinline__ void split_rows(unsigned char* hi, unsigned char* lo, int row_bytes, float* unit, int drop, int rows, int width, int pad16, const void* src, int dt,
                                           bool vec, OffFn off, MapFn map = MapFn(), int ustep = 1, SeenFn seen = SeenFn()) {
  constexpr int NI = (MAXD + 31) / 32, U = NI <= 4 ? 4 : 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l8 = lane & 7;
  for (int r0 = warp * 4 + (lane >> 3); r0 - (lane >> 3) < rows; r0 += NW * 4 * U) {
    float4 x[U][NI];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = r0 + u * NW * 4;
      const long long o = r < rows ? off(r) : -1LL;
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const int c = l8 * 4 + 32 * i;
        x[u][i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (o >= 0 && c < width) {
          if (vec) x[u][i] = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(src) + o + c);
          else x[u][i] = load4_any(src, dt, o, c, width);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = r0 + u * NW * 4;
      float m = 0.f;
#pragma unroll
      for (int i = 0; i < NI && !std::is_same<MapFn, SameValue>::value; ++i) {
        const int c = l8 * 4 + 32 * i;
        x[u][i] = make_float4(c < width ? map(x[u][i].x) : 0.f, c + 1 < width ? map(x[u][i].y) : 0.f, c + 2 < width ? map(x[u][i].z) : 0.f, c + 3 < width ? map(x[u][i].w) : 0.f);
      }
#pragma unroll
      for (int i = 0; i < NI; ++i) m = fmaxf(m, fmaxf(fmaxf(fabsf(x[u][i].x), fabsf(x[u][i].y)), fmaxf(fabsf(x[u][i].z), fabsf(x[u][i].w))));
#pragma unroll
      for (int k = 1; k < 8; k <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, k));
      if (r < rows) {
        const int e = split_exponent(m);
        const float sc = split_scale(e);
        if (l8 == 0) {
          unit[r * ustep] = pow2i(e - drop);
          seen(m);
        }
#pragma unroll
        for (int i = 0; i < NI; ++i) {
          const int c = l8 * 4 + 32 * i;
          if (c < pad16) {
            uint2 h, l;
            split2(x[u][i].x * sc, x[u][i].y * sc, h.x, l.x);
            split2(x[u][i].z * sc, x[u][i].w * sc, h.y, l.y);
            *reinterpret_cast<uint2*>(hi + r * row_bytes + c * 2) = h;
            *reinterpret_cast<uint2*>(lo + r * row_bytes + c * 2) = l;
          }
        }
      }
    }
  }
}

}  // namespace vy
