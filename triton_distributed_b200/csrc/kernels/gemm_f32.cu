// fp32 GEMM for the models' 32-bit mode: C[M,N] = A[M,K] * B[N,K]^T with products and sums as exact as fp32 ones (no TF32).
//
// On the tensor cores, with every fp32 operand cut into three bf16 values of eight significant bits each, exactly: x = x1 + x2 + x3,
// x1 the upper half of x, x2 that of x - x1, x3 the rest. x2 is held as 2^8 x2 and x3 as 2^16 x3: all three have the exponent range
// of x then, and the cut stays exact down to the smallest subnormal. (Products of bf16 parts in place of fp32 ones are a published
// method: Henry, Tang and Heinecke, 2019.) Eight of the nine products are taken, grouped by their scale: x1 y1; x1 y2, x2 y1 (2^-8);
// x2 y2, x1 y3, x3 y1 (2^-16); x2 y3, x3 y2 (2^-24). The one left out, x3 y3, is below 2^-30 of x y
// (of operands below 2^-133, which have at most 16 bits and no x1, below 2^-15). The tensor core's running fp32
// sum truncates, so x1 y1 is summed there over 64 k only and the sums of 64 are added up in registers; the other groups are 2^-8 and
// less of the result and stay in tensor memory over the whole part of K.
// Errors against 64 bits in units of 2^-24 of sum |x y|, root mean square / largest (fp32 products added in the order of K):
//   normal values   K = 1  0.43 / 1.0 (0.43 / 1.0)   8  0.25 / 2.7 (0.45 / 3.0)   64  0.23 / 1.9 (0.47 / 4.2)   2048  0.06 / 0.4 (0.47 / 5.9)
//   of one sign     K = 1  0.43 / 1.0 (0.43 / 1.0)   8  0.51 / 2.8 (0.77 / 3.7)   64  1.5 / 4.6 (2.0 / 9.1)     2048  1.6 / 4.9 (12 / 49)
// With six products (without x2 y3, x3 y2) and unscaled parts a single product was off by up to 7.8 units, always towards zero, and
// operands below 2^-110 lost bits.
// Infinities and NaNs go through x1: a sum that holds one is x1 y1 alone (a NaN keeps a bit in its upper half).
// Taken again, one product after the other in fp32, are sums above 2^125, whose scaled groups overflow, and NaNs of a tile that also
// holds a value below 2^-133, whose x1 is zero: an infinity times it is no NaN.
//
// A CTA computes 128 columns of C (rows of B, the M side of the MMA) x kT rows over one part of K; the parts of a tile are a
// cluster, whose CTAs add their partial tiles through distributed shared memory in rank order. The number of parts depends on N
// and K alone and the sum inside a part runs in the order of K, so a row's result does not depend on how many other rows share the
// call. Any M, N, K, leading dimensions and alignment.
//   warps 0-3   promotion: x1 y1 from tensor memory into registers, then the partial tile     warp 4  MMA issuer
//   warp 5      A's planes into shared memory by bulk copies, where A was cut beforehand
//   warps 8-15  operands: global memory -> registers, one or two steps of 64 k ahead -> three planes in 128-byte-swizzled shared memory
// In calls of many steps A is cut once, by a kernel in front, when the caller brings room for the planes (b200_gemm_f32_planes_bytes): every
// column tile would cut it again, and without it the registers hold two steps of B's loads instead of one. The planes and their sums are the
// same either way.
// What bounds it: the products, 1830 of 2330 clocks a step at 100 rows (the planes' copies are asked for when their place is free and take
// about as long as a step), and the start and end of a CTA. The rare cases are left to a
// second look per step: a branch for every four values kept the loads, the arithmetic and the stores of neighbouring values apart.
// us, back to back over several B, with A cut by every CTA, one step of loads and parts for 148 CTAs at once -> now (parts by clusters that fit):
//   11264 x 2048   1 row 40 -> 38    100 rows 61 -> 54    1024 rows 516 -> 411
//   2048 x 5632    1 row 39 -> 24    100 rows 60 -> 34    1024 rows 297 -> 195
//   22016 x 4096   1 row 154 -> 123  100 rows 223 -> 159  1024 rows 1954 -> 1347
//   4096 x 11008   1 row 62 -> 56    100 rows 90 -> 82    1024 rows 925 -> 636
//   512 x 1024     1 row 6.2 -> 6.3  32 rows 7.6 -> 7.6   100 rows 14.2 -> 12.2
// fp32 products on the CUDA cores with 4 x 4 outputs per thread took 227 us for 1 x 11264 x 2048 and 336 for 100 x 2048 x 5632.
#include "b200/host.h"
#include "b200/packed_f32.cuh"
#include "b200/primitives.cuh"
#include "b200/tcgen05.cuh"

#include <cfloat>

namespace b200 {

constexpr int kXN = 128, kXK = 64, kXThreads = 512, kXMaxParts = 8;
constexpr int kXPlaneB = kXN * kXK * 2;

template <int kT>
struct F32Tile {
  static constexpr int kPlaneA = kT * kXK * 2, kStage = 3 * (kXPlaneB + kPlaneA), kStages = 2;
  static constexpr int kSmem = kStages * kStage + 1024 + 1024;
  static constexpr int kMain = kT <= 64 ? 2 : 1;   // sums of 64 in tensor memory: two where there is room
  static_assert(kT % 16 == 0 && kT <= 128 && kT * kXN * 4 <= kStages * kStage, "the partial tile takes the stages' place");
};

struct F32Params {
  const float *A, *B;
  float* C;
  int M, N, K, parts, part, lda, ldb, ldc;
  bool vec_a, vec_b;
  uint32_t* status;   // nullable: set non-zero when a pipeline wait expired (the tile's results are NaN then)
  uint8_t* planes;          // nullable: A cut beforehand, [row tiles][steps of 64 k][three planes of kT rows as a stage holds them]
  uint32_t* planes_tiny;    // [row tiles][steps of 64 k] non-zero: the upper half of a value there is zero and the value is not
};

// four consecutive k of a row; zeros behind k_end
__device__ __forceinline__ float4 f32_load4(const float* row, int k, int k_end, bool vec) {
  if (vec && k + 4 <= k_end) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(row + k));
    return v;
  }
  return make_float4(k < k_end ? row[k] : 0.f, k + 1 < k_end ? row[k + 1] : 0.f, k + 2 < k_end ? row[k + 2] : 0.f,
                     k + 3 < k_end ? row[k + 3] : 0.f);
}
__device__ __forceinline__ uint32_t upper_halves(float lo, float hi) { return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632); }
__device__ __forceinline__ float upper_half(float x) { return __uint_as_float(__float_as_uint(x) & 0xffff0000u); }
__device__ __forceinline__ void st_shared_v2(uint32_t at, uint32_t a, uint32_t b) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(a), "r"(b) : "memory");
}
// the planes of four values from their first ones
__device__ __forceinline__ void f32_planes(const float4& v, const float (&h)[4], uint2 (&out)[3], float& any) {
  const f32x2 minus = pack2(-1.f, -1.f), up = pack2(256.f, 256.f);
  f32x2 r[2] = {fma2(pack2(h[0], h[1]), minus, pack2(v.x, v.y)), fma2(pack2(h[2], h[3]), minus, pack2(v.z, v.w))};
  any = fmaf(sum2(add2(r[0], r[1])), 0.f, any);
  out[0] = make_uint2(upper_halves(h[0], h[1]), upper_halves(h[2], h[3]));
#pragma unroll
  for (int g = 1; g < 3; ++g) {
    const float2 a = unpack2(mul2(r[0], up)), b = unpack2(mul2(r[1], up));
    out[g] = make_uint2(upper_halves(a.x, a.y), upper_halves(b.x, b.y));
    r[0] = fma2(pack2(upper_half(a.x), upper_half(a.y)), minus, pack2(a.x, a.y));
    r[1] = fma2(pack2(upper_half(b.x), upper_half(b.y)), minus, pack2(b.x, b.y));
  }
}
__device__ __forceinline__ void f32_store_planes(const float4& v, const float (&h)[4], uint32_t at, int plane, float& any) {
  uint2 out[3];
  f32_planes(v, h, out, any);
#pragma unroll
  for (int g = 0; g < 3; ++g) st_shared_v2(at + g * plane, out[g].x, out[g].y);
}
// falls below 0x1ffff when the upper half of one of the four holds no bit of it (zero is none of these: it wraps around)
__device__ __forceinline__ uint32_t f32_least(const float4& v) {
  const uint32_t ab = min((__float_as_uint(v.x) << 1) - 1u, (__float_as_uint(v.y) << 1) - 1u);
  const uint32_t cd = min((__float_as_uint(v.z) << 1) - 1u, (__float_as_uint(v.w) << 1) - 1u);
  return min(ab, cd);
}
// The cut of four values. `any` becomes NaN when one of them is an infinity or a NaN (or their differences overflow), `least` follows
// f32_least.
__device__ __forceinline__ void f32_cut(const float4& v, uint32_t at, int plane, float& any, uint32_t& least) {
  const float h[4] = {upper_half(v.x), upper_half(v.y), upper_half(v.z), upper_half(v.w)};
  least = min(least, f32_least(v));
  f32_store_planes(v, h, at, plane, any);
}
// the same with a bit in the upper half of every NaN, which an infinity would stand for otherwise
__device__ __forceinline__ void f32_first_odd(const float4& v, float (&h)[4]) {
  const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) h[e] = x[e] != x[e] ? __uint_as_float(0x7fff0000u) : upper_half(x[e]);
}
__device__ __noinline__ void f32_cut_odd(float4 v, uint32_t at, int plane) {
  float h[4], any = 0.f;
  f32_first_odd(v, h);
  f32_store_planes(v, h, at, plane, any);
}

// A cut once for all column tiles, in the form of the GEMM's stages. grid (steps of 64 k, row tiles).
template <int kT>
__global__ void __launch_bounds__(256) f32_planes_kernel(const F32Params p) {
  constexpr int kPlane = F32Tile<kT>::kPlaneA;
  const int c = threadIdx.x & 15, r0 = threadIdx.x >> 4, k = blockIdx.x * kXK + 4 * c, m0 = blockIdx.y * kT;
  const size_t at = static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x;
  uint8_t* out = p.planes + at * (3 * kPlane) + r0 * 128 + (((c >> 1) ^ (r0 & 7)) * 16) + (c & 1) * 8;
  griddep_launch_dependents();
  griddep_wait();
  float4 v[kT / 16];
#pragma unroll
  for (int i = 0; i < kT / 16; ++i) v[i] = f32_load4(p.A + static_cast<size_t>(min(m0 + r0 + 16 * i, p.M - 1)) * p.lda, k, p.K, p.vec_a);
  uint32_t least = ~0u;
#pragma unroll
  for (int i = 0; i < kT / 16; ++i) {
    float h[4], any = 0.f;
    uint2 x[3];
    f32_first_odd(v[i], h);
    f32_planes(v[i], h, x, any);
    least = min(least, f32_least(v[i]));
#pragma unroll
    for (int g = 0; g < 3; ++g) *reinterpret_cast<uint2*>(out + g * kPlane + i * 16 * 128) = x[g];
  }
  const int tiny = __syncthreads_or(least < 0x1ffffu);
  if (threadIdx.x == 0) p.planes_tiny[at] = tiny;
}

// 16 rows of a column of the partial tile from their sums of x1 y1 (`sum`, by row) and the scaled groups in tensor memory (`from`). Returns the
// rows whose sum is finite in x1 y1 but not in the scaled groups, or is no number where an infinity may have met such a value (`small`).
template <typename Sum>
__device__ __forceinline__ uint32_t f32_join(uint32_t from, bool read, bool ok, bool small, float* at, const Sum& sum) {
  uint32_t c1[16] = {}, c2[16] = {}, c3[16] = {}, again = 0;
  if (read) {
    tmem_ld_32x16(from, c1);
    tmem_ld_32x16(from + 128, c2);
    tmem_ld_32x16(from + 256, c3);
    tmem_ld_wait();
  }
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const float main = sum(q);
    const float rest = fmaf(fmaf(__uint_as_float(c3[q]), 0x1p-8f, __uint_as_float(c2[q])), 0x1p-8f, __uint_as_float(c1[q]));
    const bool finite = fabsf(main) <= FLT_MAX;
    const float v = finite ? fmaf(rest, 0x1p-8f, main) : main;
    if (finite ? !(fabsf(rest) <= FLT_MAX) : small && main != main) again |= 1u << q;
    at[q * kXN] = ok ? v : NAN;
  }
  return ok ? again : 0u;
}
// takes the marked rows of column n once more, one product after the other
__device__ __forceinline__ void f32_again(const F32Params& p, uint32_t left, float* at, int m0, int n0, int n, int k_begin, int k_end) {
  const float* b = p.B + static_cast<size_t>(min(n0 + n, p.N - 1)) * p.ldb;
  for (; left != 0u; left &= left - 1) {
    const int q = __ffs(left) - 1;
    const float* a = p.A + static_cast<size_t>(min(m0 + q, p.M - 1)) * p.lda;
    float sum = 0.f;
    for (int k = k_begin; k < k_end; ++k) sum = fmaf(a[k], b[k], sum);
    at[q * kXN] = sum;
  }
}

// The partial tile is finished by three warpgroups, every third 16 rows each, a thread a column of C. (One warpgroup took 8800 of a CTA's
// 45000 clocks for it at 112 rows, with the other warps idle.) 16 rows are finished by the warps that hold x1 y1, straight from their
// registers.
constexpr bool f32_alone(int rows) { return rows <= 16; }
template <int kT>
__device__ __forceinline__ void f32_finish(const F32Params& p, uint32_t tmem_base, float* out, int warp, int group, int m0, int n0, int k_begin,
                                           int k_end, int steps, volatile uint32_t* abort_flag, volatile uint32_t* tiny) {
  asm volatile("bar.sync 1, 384;" ::: "memory");   // x1 y1 is there, whatever became of the waits
  const int n = (warp & 3) * 32 + (threadIdx.x & 31);
  const uint32_t lanes = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
  const bool ok = __all_sync(0xffffffffu, *abort_flag == 0u), small = *tiny != 0u;
  tc_fence_after_sync();
#pragma unroll 1
  for (int h = group; h < kT / 16; h += 3) {
    float* at = out + h * 16 * kXN + n;
    __syncwarp();
    const uint32_t again = f32_join(lanes + 128 + h * 16, steps > 0 && ok, ok, small, at, [&](int q) { return at[q * kXN]; });
    f32_again(p, again, at, m0 + h * 16, n0, n, k_begin, k_end);
  }
  tc_fence_before_sync();
}

__device__ __forceinline__ void bulk_load(void* dst, const void* src, int bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// kPlanes: A has been cut by f32_planes_kernel and arrives by bulk copies. kDepth: steps of loads in flight
template <int kT, bool kPlanes, int kDepth>
__global__ void __launch_bounds__(kXThreads, 1) gemm_f32_kernel(const F32Params p) {
  using T = F32Tile<kT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + T::kStages * T::kStage);
  uint64_t *full_bar = bars, *empty_bar = bars + 2, *dfull_bar = bars + 4, *dempty_bar = bars + 6, *done_bar = bars + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 9);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  volatile uint32_t* tiny = tmem_slot + 2;   // an operand's upper half is zero and the operand is not
  uint64_t* afull_bar = bars + 12;           // kPlanes: A's planes have landed
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x % p.parts;  // in the cluster
  const int n0 = blockIdx.x / p.parts * kXN, m0 = blockIdx.y * kT;
  const int k_begin = rank * p.part, k_end = min(p.K, k_begin + p.part);
  const int steps = max(0, (k_end - k_begin + kXK - 1) / kXK);
  constexpr uint64_t kTimeout = 4000000000ull;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(full_bar + i, 256);
      mbar_init(empty_bar + i, 1);
      mbar_init(dfull_bar + i, 1);
      mbar_init(dempty_bar + i, 4);
      mbar_init(afull_bar + i, 1);
    }
    mbar_init(done_bar, kPlanes ? 2 : 1);
    *abort_flag = 0;
    *tiny = 0;
    mbar_fence_init();
  }
  if (warp == 4) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  // columns: x1 y1 at 0 (up to 64 rows: of odd steps at 64), the products of scale 2^-8, 2^-16, 2^-24 at 128, 256, 384
  const uint32_t tmem_base = *tmem_slot;
  griddep_launch_dependents();
  griddep_wait();

  if (warp < 4) {
    // ------------------------------------------------------------------ promotion: thread = a column of C, kT rows
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");   // 128 * (216 + 40 + 128 + 128) = the launch's 512 * 128
    f32x2 acc[kT / 2];
#pragma unroll
    for (int j = 0; j < kT / 2; ++j) acc[j] = 0ull;
    const uint32_t lanes = tmem_base + (static_cast<uint32_t>(warp * 32) << 16);
    auto add = [&](uint32_t taddr) {
      uint32_t r0[16], r1[16];
      tmem_ld_32x16(taddr, r0);
#pragma unroll
      for (int h = 0; h < kT / 16; ++h) {
        tmem_ld_wait();
        if (h + 1 < kT / 16) tmem_ld_32x16(taddr + (h + 1) * 16, (h & 1) ? r0 : r1);
        uint32_t* r = (h & 1) ? r1 : r0;
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[h * 8 + q] = add2(acc[h * 8 + q], pack2(__uint_as_float(r[2 * q]), __uint_as_float(r[2 * q + 1])));
      }
    };
    bool ok = true;
    for (int s = 0; s < steps && ok; ++s) {
      const int at = s % T::kMain;
      ok = mbar_wait(dfull_bar + at, (s / T::kMain) & 1, abort_flag, kTimeout);
      if (!ok) break;
      tc_fence_after_sync();
      add(lanes + at * 64);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(dempty_bar + at);
    }
    if (steps > 0 && ok) ok = mbar_wait(done_bar, 0, abort_flag, kTimeout);
    // all products are done: the stages give way to the partial tile [kT][128]
    float* out = reinterpret_cast<float*>(smem);
    auto sum = [&](int r) {   // of x1 y1
      const float2 pair = unpack2(acc[r / 2]);
      return (r & 1) ? pair.y : pair.x;
    };
    if (f32_alone(kT)) {
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after_sync();
      const bool small = *tiny != 0u;
      const uint32_t again = f32_join(lanes + 128, steps > 0 && ok, ok, small, out + threadIdx.x, sum);
      f32_again(p, again, out + threadIdx.x, m0, n0, threadIdx.x, k_begin, k_end);
      tc_fence_before_sync();
    } else {
#pragma unroll
      for (int r = 0; r < kT; ++r) out[r * kXN + threadIdx.x] = sum(r);
      f32_finish<kT>(p, tmem_base, out, warp, 0, m0, n0, k_begin, k_end, steps, abort_flag, tiny);
    }
  } else if (warp < 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == 4 && elect_one()) {
      // ---------------------------------------------------------------- MMA issuer
      const uint32_t idesc = umma_idesc_f16(kXN, kT, true);
      bool ok = true;
      for (int s = 0; s < steps; ++s) {
        const uint32_t st = s & 1, phase = (s >> 1) & 1, main = s % T::kMain;
        ok = mbar_wait(dempty_bar + main, ((s / T::kMain) & 1) ^ 1, abort_flag, kTimeout) && mbar_wait(full_bar + st, phase, abort_flag, kTimeout) &&
             (!kPlanes || mbar_wait(afull_bar + st, phase, abort_flag, kTimeout));
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t at = smem_u32(smem + st * T::kStage);
        const uint64_t b1 = umma_desc_sw128_kmajor(at), b2 = umma_desc_sw128_kmajor(at + kXPlaneB), b3 = umma_desc_sw128_kmajor(at + 2 * kXPlaneB);
        const uint32_t aa = at + 3 * kXPlaneB;
        const uint64_t a1 = umma_desc_sw128_kmajor(aa), a2 = umma_desc_sw128_kmajor(aa + T::kPlaneA), a3 = umma_desc_sw128_kmajor(aa + 2 * T::kPlaneA);
#pragma unroll
        for (int k = 0; k < kXK / 16; ++k) umma_f16(tmem_base + main * 64, b1 + 2 * k, a1 + 2 * k, idesc, k != 0 ? 1u : 0u);
        umma_commit(dfull_bar + main);
        // the promotion reads x1 y1 while these run: with one sum of 64 only, the next step's need not wait either
#pragma unroll 1
        for (int k = 0; k < kXK / 16; ++k) {
          const uint32_t more = (s | k) != 0 ? 1u : 0u;
          umma_f16(tmem_base + 128, b1 + 2 * k, a2 + 2 * k, idesc, more);
          umma_f16(tmem_base + 128, b2 + 2 * k, a1 + 2 * k, idesc, 1u);
          umma_f16(tmem_base + 256, b2 + 2 * k, a2 + 2 * k, idesc, more);
          umma_f16(tmem_base + 256, b1 + 2 * k, a3 + 2 * k, idesc, 1u);
          umma_f16(tmem_base + 256, b3 + 2 * k, a1 + 2 * k, idesc, 1u);
          umma_f16(tmem_base + 384, b2 + 2 * k, a3 + 2 * k, idesc, more);
          umma_f16(tmem_base + 384, b3 + 2 * k, a2 + 2 * k, idesc, 1u);
        }
        umma_commit(empty_bar + st);
      }
      if (ok && steps > 0) umma_commit(done_bar);
    }
    if (kPlanes && warp == 5) {
      // ---------------------------------------------------------------- A's planes
      const size_t first = static_cast<size_t>(blockIdx.y) * ((p.K + kXK - 1) / kXK) + k_begin / kXK;
      if (lane == 0) {
        fence_proxy_async();
        int s = 0;
        for (; s < steps; ++s) {
          if (!mbar_wait(empty_bar + (s & 1), ((s >> 1) & 1) ^ 1, abort_flag, kTimeout)) break;
          mbar_expect_tx(afull_bar + (s & 1), 3 * T::kPlaneA);
          bulk_load(smem + (s & 1) * T::kStage + 3 * kXPlaneB, p.planes + (first + s) * (3 * T::kPlaneA), 3 * T::kPlaneA, afull_bar + (s & 1));
        }
        volatile uint32_t never = 0;   // the last copies have to land before shared memory is given back, also after an abort
        for (int c = max(0, s - 2); c < s; ++c) mbar_wait(afull_bar + (c & 1), (c >> 1) & 1, &never, kTimeout);
      }
      __syncwarp();
      uint32_t small = 0;
      for (int s = lane; s < steps; s += 32) small |= __ldcg(p.planes_tiny + first + s);
      if (__any_sync(0xffffffffu, small != 0u) && lane == 0) *tiny = 1;
      __syncwarp();
      if (lane == 0 && steps > 0) mbar_arrive(done_bar);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ operands: half a warp per row of 64 k
    const int t = threadIdx.x - 256, c = t & 15, r0 = t >> 4;
    const int k0 = k_begin + 4 * c;
    // eight rows down the swizzle repeats: the offset inside a row is the same for all rows of this thread
    const uint32_t off = static_cast<uint32_t>(r0 * 128 + (((c >> 1) ^ (r0 & 7)) * 16) + (c & 1) * 8);
    constexpr int kRowsB = kXN / 16, kRowsA = kPlanes ? 0 : kT / 16;
    const float *rb[kRowsB], *ra[kRowsA + 1];
    float4 vb[kDepth][kRowsB], va[kDepth][kRowsA + 1];
#pragma unroll
    for (int i = 0; i < kRowsB; ++i) rb[i] = p.B + static_cast<size_t>(min(n0 + r0 + 16 * i, p.N - 1)) * p.ldb;   // behind the last row
#pragma unroll
    for (int i = 0; i < kRowsA; ++i) ra[i] = p.A + static_cast<size_t>(min(m0 + r0 + 16 * i, p.M - 1)) * p.lda;   // that row again: not stored
#pragma unroll
    for (int d = 0; d < kDepth; ++d) {
#pragma unroll
      for (int i = 0; i < kRowsB; ++i) vb[d][i] = f32_load4(rb[i], k0 + d * kXK, k_end, p.vec_b);
#pragma unroll
      for (int i = 0; i < kRowsA; ++i) va[d][i] = f32_load4(ra[i], k0 + d * kXK, k_end, p.vec_a);
    }
    bool ok = true;
    for (int s0 = 0; s0 < steps && ok; s0 += kDepth) {
#pragma unroll
      for (int d = 0; d < kDepth; ++d) {
        const int s = s0 + d, st = s & 1, next = k0 + (s + kDepth) * kXK;
        if (s >= steps) break;
        ok = mbar_wait(empty_bar + st, ((s >> 1) & 1) ^ 1, abort_flag, kTimeout);
        if (!ok) break;
        const uint32_t at = smem_u32(smem + st * T::kStage) + off;
        float any = 0.f;
        uint32_t least = ~0u;
#pragma unroll
        for (int i = 0; i < kRowsB; ++i) {
          f32_cut(vb[d][i], at + i * 16 * 128, kXPlaneB, any, least);
          vb[d][i] = f32_load4(rb[i], next, k_end, p.vec_b);
        }
#pragma unroll
        for (int i = 0; i < kRowsA; ++i) {
          f32_cut(va[d][i], at + 3 * kXPlaneB + i * 16 * 128, T::kPlaneA, any, least);
          va[d][i] = f32_load4(ra[i], next, k_end, p.vec_a);
        }
        if (least < 0x1ffffu) *tiny = 1;
        if (any != any) {   // rare: this step's values are read again, and cut with a look at each
#pragma unroll 1
          for (int i = 0; i < kRowsB + kRowsA; ++i) {
            const bool of_b = i < kRowsB;
            const int r = r0 + 16 * (of_b ? i : i - kRowsB);
            const float* row = of_b ? p.B + static_cast<size_t>(min(n0 + r, p.N - 1)) * p.ldb : p.A + static_cast<size_t>(min(m0 + r, p.M - 1)) * p.lda;
            f32_cut_odd(f32_load4(row, next - kDepth * kXK, k_end, of_b ? p.vec_b : p.vec_a), at + (of_b ? 0 : 3 * kXPlaneB) + (r - r0) * 128, of_b ? kXPlaneB : T::kPlaneA);
          }
        }
        fence_view_async_shared();
        mbar_arrive(full_bar + st);
      }
    }
    if (!f32_alone(kT)) {
      if (steps > 0 && ok) mbar_wait(done_bar, 0, abort_flag, kTimeout);
      f32_finish<kT>(p, tmem_base, reinterpret_cast<float*>(smem), warp, (warp >> 2) - 1, m0, n0, k_begin, k_end, steps, abort_flag, tiny);
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 4) tmem_dealloc(tmem_base, 512);
  if (threadIdx.x == 0 && *abort_flag != 0u && p.status != nullptr) atomicMax(p.status, static_cast<uint32_t>(kStatusPipeTimeout));
  cluster_sync_all();
  if (warp >= 8) {
    // this CTA's share of the tile: the sum over the parts in order
    const float* out = reinterpret_cast<const float*>(smem);
    for (int i = rank * 256 + threadIdx.x - 256; i < kT * kXN / 4; i += 256 * p.parts) {
      const int r = i / (kXN / 4), n = i % (kXN / 4) * 4;
      if (m0 + r >= p.M || n0 + n >= p.N) continue;
      float v[4] = {};
      constexpr int kReads = kT <= 16 && kDepth == 1 ? 1 : 4;   // on their way at a time; a short sum of few rows gains nothing by more
      for (int q0 = 0; q0 < p.parts; q0 += kReads) {
        float4 x[kReads];
#pragma unroll
        for (int q = 0; q < kReads; ++q)
          if (q0 + q < p.parts)
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(x[q].x), "=f"(x[q].y), "=f"(x[q].z), "=f"(x[q].w)
                         : "r"(mapa_u32(out + r * kXN + n, q0 + q)));
#pragma unroll
        for (int q = 0; q < kReads; ++q)
          if (q0 + q < p.parts) v[0] += x[q].x, v[1] += x[q].y, v[2] += x[q].z, v[3] += x[q].w;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (n0 + n + e < p.N) p.C[static_cast<size_t>(m0 + r) * p.ldc + n0 + n + e] = v[e];
    }
  }
  __syncwarp();
  cluster_sync_all();  // the others have read this CTA's partial tile
}

// Parts of K, from N and K alone: the fewest steps on the busiest SM, where a CTA's start, its sum over the parts and its end cost about
// as much as four steps. A cluster's CTAs, one per SM, lie in one part of the chip, so clusters leave SMs over: 15 of eight run at a time
// and not 18 (2048 x 5632, 100 rows: 16 clusters of eight, two waves, 53 us; of six, one wave, 35). The counts are a B200's, whatever the
// device has: the parts are part of the result's rounding.
constexpr int kF32Clusters[kXMaxParts] = {148, 74, 45, 33, 26, 22, 15, 15};
static int f32_parts(int N, int K) {
  const int tiles = (N + kXN - 1) / kXN, steps = (K + kXK - 1) / kXK;
  int best = 1;
  long long least = 1ll << 62;
  for (int parts = 1; parts <= kXMaxParts && parts <= steps; ++parts) {
    const long long waves = (tiles + kF32Clusters[parts - 1] - 1) / kF32Clusters[parts - 1];
    const long long cost = waves * ((steps + parts - 1) / parts + 4);
    if (cost < least) least = cost, best = parts;
  }
  return best;
}

// row tiles of even height: 100 rows are one of 112, 150 two of 80
static int f32_rows(int M) {
  const int tiles = (M + 127) / 128;
  return ((M + tiles - 1) / tiles + 15) / 16 * 16;
}
// steps of 64 k that the busiest SM takes in all its waves
static int f32_steps(int M, int N, int K) {
  const int parts = f32_parts(N, K), at_once = kF32Clusters[parts - 1];
  const long long tiles = static_cast<long long>((N + kXN - 1) / kXN) * ((M + f32_rows(M) - 1) / f32_rows(M));
  const long long steps = (tiles + at_once - 1) / at_once * (((K + kXK - 1) / kXK + parts - 1) / parts);
  return steps > 1 << 20 ? 1 << 20 : static_cast<int>(steps);
}

template <int kT, bool kPlanes, int kDepth>
static int launch_gemm_f32_form(const F32Params& p, cudaStream_t stream) {
  using T = F32Tile<kT>;
  static bool configured[64] = {false};
  int dev = 0;
  B200_CHECK_CUDA(cudaGetDevice(&dev));
  if (!configured[dev & 63]) {
    B200_CHECK_CUDA(cudaFuncSetAttribute(gemm_f32_kernel<kT, kPlanes, kDepth>, cudaFuncAttributeMaxDynamicSharedMemorySize, T::kSmem));
    configured[dev & 63] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((p.N + kXN - 1) / kXN * p.parts, (p.M + kT - 1) / kT);
  cfg.blockDim = dim3(kXThreads);
  cfg.dynamicSmemBytes = T::kSmem;
  cfg.stream = stream;
  B200_REQUIRE(cfg.gridDim.y <= 65535, "M (%d) is too large", p.M);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.parts;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  if (kPlanes)
    B200_CHECK_CUDA(launch_pdl(f32_planes_kernel<kT>, dim3((p.K + kXK - 1) / kXK, cfg.gridDim.y), dim3(256), 0, stream, p));
  B200_CHECK_CUDA(cudaLaunchKernelEx(&cfg, gemm_f32_kernel<kT, kPlanes, kDepth>, p));
  return kOk;
}
template <int kT>
static int launch_gemm_f32(F32Params& p, void* workspace, cudaStream_t stream) {
  if (workspace == nullptr) {
    // Two steps of B in flight beside 16 rows of A, where a CTA has steps enough to need them. us with one and with two, one row: 64 x 256
    // 5.0, 5.3; 256 x 4096 (8 steps) 12.8, 13.2; 2048 x 4096 (11) 20.0, 19.2; 4096 x 4096 (16) 26.7, 25.4. More rows leave no registers for it.
    if (kT == 16 && f32_steps(p.M, p.N, p.K) > 8) return launch_gemm_f32_form<kT, false, kT == 16 ? 2 : 1>(p, stream);
    return launch_gemm_f32_form<kT, false, 1>(p, stream);
  }
  const size_t stages = static_cast<size_t>((p.M + kT - 1) / kT) * ((p.K + kXK - 1) / kXK);
  p.planes = static_cast<uint8_t*>(workspace);
  p.planes_tiny = reinterpret_cast<uint32_t*>(p.planes + stages * (3 * F32Tile<kT>::kPlaneA));
  return launch_gemm_f32_form<kT, true, 2>(p, stream);
}

}  // namespace b200

using namespace b200;

// Bytes of b200_gemm_f32_planes' workspace.
B200_API long long b200_gemm_f32_workspace_bytes(int M, int K) {
  if (M <= 0 || K <= 0) return 0;
  const int rows = f32_rows(M);
  return static_cast<long long>((M + rows - 1) / rows) * ((K + kXK - 1) / kXK) * (3ll * rows * kXK * 2 + 4);
}

// Bytes of a workspace that makes the call faster, or none: the launch in front costs about 1.2 us, and a step of few rows is no shorter with A's
// planes at hand. us with A cut inside and in front, by rows x N x K (steps of the busiest SM): 32 x 256 x 1024 (2) 7.8, 8.7; 32 x 1024 x 4096
// (8) 16.5, 17.0; 32 x 4096 x 4096 (16) 28.3, 27.7; 48 x 512 x 2048 (4) 11.3, 11.7; 48 x 512 x 4096 (8) 17.8, 17.3; 64 x 2048 x 1024 (3) 12.6, 13.3; 64 x
// 2048 x 2048 (6) 16.8, 17.1; 64 x 512 x 4096 (8) 19.4, 18.3; 100 x 512 x 1024 (2) 12.5, 13.2; 100 x 512 x 2048 (4) 16.1, 16.0; 100 x 2048 x 2048 (6) 21.0,
// 20.2; 256 x 1024 x 1024 (4) 27.1, 27.1; 256 x 4096 x 4096 (32) 83, 70.
B200_API long long b200_gemm_f32_planes_bytes(int M, int N, int K) {
  if (M <= 16 || N <= 0 || K <= 0 || f32_steps(M, N, K) * f32_rows(M) < 384) return 0;
  return b200_gemm_f32_workspace_bytes(M, K);
}

// workspace (nullable, on a 16-byte boundary): A is cut into its planes there, once for all column tiles; results are the same. status
// (device, nullable): raised when a wait inside the kernel runs out.
B200_API int b200_gemm_f32_planes(const float* A, const float* B, float* C, int M, int N, int K, int lda, int ldb, int ldc,
                                  void* workspace, uint32_t* status, void* stream) {
  B200_REQUIRE(M > 0 && N > 0 && K > 0, "empty problem %dx%dx%d", M, N, K);
  B200_REQUIRE(lda >= K && ldb >= K && ldc >= N, "leading dimensions are smaller than the rows");
  B200_REQUIRE(reinterpret_cast<uintptr_t>(workspace) % 16 == 0, "the workspace must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  auto aligned = [](const float* x, int ld) { return ld % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0; };
  F32Params p = {A, B, C, M, N, K, f32_parts(N, K), 0, lda, ldb, ldc, aligned(A, lda), aligned(B, ldb), status, nullptr, nullptr};
  p.part = ((K + p.parts - 1) / p.parts + kXK - 1) / kXK * kXK;
  switch (f32_rows(M) / 16) {
    case 1: return launch_gemm_f32<16>(p, workspace, s);
    case 2: return launch_gemm_f32<32>(p, workspace, s);
    case 3: return launch_gemm_f32<48>(p, workspace, s);
    case 4: return launch_gemm_f32<64>(p, workspace, s);
    case 5: return launch_gemm_f32<80>(p, workspace, s);
    case 6: return launch_gemm_f32<96>(p, workspace, s);
    case 7: return launch_gemm_f32<112>(p, workspace, s);
    default: return launch_gemm_f32<128>(p, workspace, s);
  }
}
// The same without a workspace.
B200_API int b200_gemm_f32_checked(const float* A, const float* B, float* C, int M, int N, int K, int lda, int ldb, int ldc,
                                   uint32_t* status, void* stream) {
  return b200_gemm_f32_planes(A, B, C, M, N, K, lda, ldb, ldc, nullptr, status, stream);
}
B200_API int b200_gemm_f32(const float* A, const float* B, float* C, int M, int N, int K, int lda, int ldb, int ldc,
                           void* stream) {
  return b200_gemm_f32_planes(A, B, C, M, N, K, lda, ldb, ldc, nullptr, nullptr, stream);
}
