// fp32 GEMM for the models' 32-bit mode: C[M,N] = A[M,K] * B[N,K]^T with products and sums as exact as fp32 ones (no TF32).
//
// On the tensor cores, with every fp32 operand cut into three bf16 values of eight significant bits each (x = x1 + x2 + x3, exactly:
// the upper halves of x, x - x1 and x - x1 - x2). Of the nine products x1 y1, x1 y2, x2 y1, x2 y2, x1 y3 and x3 y1 are taken; the
// three left out are below 2^-23 of x y together. The tensor core's running fp32 sum truncates, so x1 y1 is summed there over 64 k
// only and the sums of 64 are added up in registers; the other five are 2^-8 smaller and stay in tensor memory over the whole part
// of K. The error of a SwiGLU block of 2048 / 5632 against 64 bits is 4.2e-7 of its norm (fp32 products on the CUDA cores: 7.7e-7).
// An infinity or a NaN has no such cut: rows that hold one are marked while they are cut, and their results are summed again, one
// product after the other, in fp32.
//
// A CTA computes 128 columns of C (rows of B, the M side of the MMA) x kT rows over one part of K; the parts of a tile are a
// cluster, whose CTAs add their partial tiles through distributed shared memory in rank order. The number of parts depends on N
// and K alone and the sum inside a part runs in the order of K, so a row's result does not depend on how many other rows share the
// call. Any M, N, K, leading dimensions and alignment.
//   warps 0-3   promotion: x1 y1 from tensor memory into registers, then the partial tile     warp 4  MMA issuer
//   warps 8-15  operands: global memory -> registers, one step of 64 k ahead -> three planes in 128-byte-swizzled shared memory
// What bounds it: for few rows the bytes of B; around 128 rows those bytes, the six products and the cutting (about 1000 clocks of a
// step's 1500) are near one another; for many rows the tensor cores.
// Measured against fp32 products on the CUDA cores with 8 x 8 outputs per thread (11264 x 2048 and 2048 x 5632, us):
//   M = 100  183, 101 -> 62, 46
#include "b200/host.h"
#include "b200/packed_f32.cuh"
#include "b200/primitives.cuh"
#include "b200/tcgen05.cuh"

namespace b200 {

constexpr int kXN = 128, kXK = 64, kXThreads = 512, kXMaxParts = 8;
constexpr int kXPlaneB = kXN * kXK * 2;

template <int kT>
struct F32Tile {
  static constexpr int kPlaneA = kT * kXK * 2, kStage = 3 * (kXPlaneB + kPlaneA), kStages = 2;
  static constexpr int kSmem = kStages * kStage + 1024 + 1024;
  static_assert(kT % 16 == 0 && kT <= 128 && kT * kXN * 4 <= kStages * kStage, "the partial tile takes the stages' place");
};

struct F32Params {
  const float *A, *B;
  float* C;
  int M, N, K, parts, part, lda, ldb, ldc;
  bool vec_a, vec_b;
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
// the three planes of four values; whether one of them is no finite number
__device__ __forceinline__ bool f32_cut(const float4& v, uint32_t at, int plane) {
  float x[4] = {v.x, v.y, v.z, v.w}, r[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) r[e] = x[e] - upper_half(x[e]);
  st_shared_v2(at, upper_halves(x[0], x[1]), upper_halves(x[2], x[3]));
  st_shared_v2(at + plane, upper_halves(r[0], r[1]), upper_halves(r[2], r[3]));
#pragma unroll
  for (int e = 0; e < 4; ++e) r[e] -= upper_half(r[e]);
  st_shared_v2(at + 2 * plane, upper_halves(r[0], r[1]), upper_halves(r[2], r[3]));
  const float any = (r[0] + r[1]) + (r[2] + r[3]);   // inf - inf and NaN - NaN are NaN
  return any != any;
}

template <int kT>
__global__ void __launch_bounds__(kXThreads, 1) gemm_f32_kernel(const F32Params p) {
  using T = F32Tile<kT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + T::kStages * T::kStage);
  uint64_t *full_bar = bars, *empty_bar = bars + 2, *dfull_bar = bars + 4, *dempty_bar = bars + 6, *done_bar = bars + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 9);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  volatile uint32_t* marked = tmem_slot + 2;                               // a row of this tile holds an infinity or a NaN
  volatile uint8_t* mark_b = reinterpret_cast<uint8_t*>(tmem_slot + 4);    // [128] which, of B and of A
  volatile uint8_t* mark_a = mark_b + kXN;                                 // [kT]
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
    }
    mbar_init(done_bar, 1);
    *abort_flag = 0;
    *marked = 0;
    mbar_fence_init();
  }
  if (threadIdx.x < kXN) mark_b[threadIdx.x] = 0;
  if (threadIdx.x < kT) mark_a[threadIdx.x] = 0;
  if (warp == 4) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;   // columns: x1 y1 of even and odd steps at 0 and 128, the other products at 256
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
      ok = mbar_wait(dfull_bar + (s & 1), (s >> 1) & 1, abort_flag, kTimeout);
      if (!ok) break;
      tc_fence_after_sync();
      add(lanes + (s & 1) * 128);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(dempty_bar + (s & 1));
    }
    if (steps > 0) {
      ok = ok && mbar_wait(done_bar, 0, abort_flag, kTimeout);
      if (ok) {
        tc_fence_after_sync();
        add(lanes + 256);
        tc_fence_before_sync();
      }
    }
    // all products are done: the stages give way to the partial tile [kT][128]
    float* out = reinterpret_cast<float*>(smem);
    const int n = threadIdx.x;
#pragma unroll
    for (int j = 0; j < kT / 2; ++j) {
      const float2 v = ok ? unpack2(acc[j]) : make_float2(NAN, NAN);
      out[(2 * j) * kXN + n] = v.x;
      out[(2 * j + 1) * kXN + n] = v.y;
    }
    if (ok && *marked != 0u) {
      const float* b = p.B + static_cast<size_t>(min(n0 + n, p.N - 1)) * p.ldb;
      for (int t = 0; t < kT; ++t) {
        if (mark_b[n] == 0 && mark_a[t] == 0) continue;
        const float* a = p.A + static_cast<size_t>(min(m0 + t, p.M - 1)) * p.lda;
        float sum = 0.f;
        for (int k = k_begin; k < k_end; ++k) sum = fmaf(a[k], b[k], sum);
        out[t * kXN + n] = sum;
      }
    }
  } else if (warp < 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == 4 && elect_one()) {
      // ---------------------------------------------------------------- MMA issuer
      const uint32_t idesc = umma_idesc_f16(kXN, kT, true);
      bool ok = true;
      for (int s = 0; s < steps; ++s) {
        const uint32_t st = s & 1, phase = (s >> 1) & 1;
        ok = mbar_wait(dempty_bar + st, phase ^ 1, abort_flag, kTimeout) && mbar_wait(full_bar + st, phase, abort_flag, kTimeout);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t at = smem_u32(smem + st * T::kStage);
        const uint64_t b1 = umma_desc_sw128_kmajor(at), b2 = umma_desc_sw128_kmajor(at + kXPlaneB), b3 = umma_desc_sw128_kmajor(at + 2 * kXPlaneB);
        const uint32_t aa = at + 3 * kXPlaneB;
        const uint64_t a1 = umma_desc_sw128_kmajor(aa), a2 = umma_desc_sw128_kmajor(aa + T::kPlaneA), a3 = umma_desc_sw128_kmajor(aa + 2 * T::kPlaneA);
#pragma unroll
        for (int k = 0; k < kXK / 16; ++k) umma_f16(tmem_base + st * 128, b1 + 2 * k, a1 + 2 * k, idesc, k != 0 ? 1u : 0u);
        umma_commit(dfull_bar + st);
#pragma unroll 1
        for (int k = 0; k < kXK / 16; ++k) {
          umma_f16(tmem_base + 256, b3 + 2 * k, a1 + 2 * k, idesc, (s | k) != 0 ? 1u : 0u);
          umma_f16(tmem_base + 256, b1 + 2 * k, a3 + 2 * k, idesc, 1u);
          umma_f16(tmem_base + 256, b2 + 2 * k, a2 + 2 * k, idesc, 1u);
          umma_f16(tmem_base + 256, b2 + 2 * k, a1 + 2 * k, idesc, 1u);
          umma_f16(tmem_base + 256, b1 + 2 * k, a2 + 2 * k, idesc, 1u);
        }
        umma_commit(empty_bar + st);
      }
      if (ok && steps > 0) umma_commit(done_bar);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ operands: half a warp per row of 64 k
    const int t = threadIdx.x - 256, c = t & 15, r0 = t >> 4;
    const int k0 = k_begin + 4 * c;
    const float *rb[kXN / 16], *ra[kT / 16];
    float4 vb[kXN / 16], va[kT / 16];
#pragma unroll
    for (int i = 0; i < kXN / 16; ++i) {   // behind the last row that row again: its results are not stored
      rb[i] = p.B + static_cast<size_t>(min(n0 + r0 + 16 * i, p.N - 1)) * p.ldb;
      vb[i] = f32_load4(rb[i], k0, k_end, p.vec_b);
    }
#pragma unroll
    for (int i = 0; i < kT / 16; ++i) {
      ra[i] = p.A + static_cast<size_t>(min(m0 + r0 + 16 * i, p.M - 1)) * p.lda;
      va[i] = f32_load4(ra[i], k0, k_end, p.vec_a);
    }
    // eight rows down the swizzle repeats: the offset inside a row is the same for all rows of this thread
    const uint32_t off = static_cast<uint32_t>(r0 * 128 + (((c >> 1) ^ (r0 & 7)) * 16) + (c & 1) * 8);
    for (int s = 0; s < steps; ++s) {
      const int next = k0 + (s + 1) * kXK;
      if (!mbar_wait(empty_bar + (s & 1), ((s >> 1) & 1) ^ 1, abort_flag, kTimeout)) break;
      const uint32_t at = smem_u32(smem + (s & 1) * T::kStage) + off;
#pragma unroll
      for (int i = 0; i < kXN / 16; ++i) {
        if (f32_cut(vb[i], at + i * 16 * 128, kXPlaneB)) {
          mark_b[r0 + 16 * i] = 1;
          *marked = 1;
        }
        vb[i] = f32_load4(rb[i], next, k_end, p.vec_b);
      }
#pragma unroll
      for (int i = 0; i < kT / 16; ++i) {
        if (f32_cut(va[i], at + 3 * kXPlaneB + i * 16 * 128, T::kPlaneA)) {
          mark_a[r0 + 16 * i] = 1;
          *marked = 1;
        }
        va[i] = f32_load4(ra[i], next, k_end, p.vec_a);
      }
      fence_view_async_shared();
      mbar_arrive(full_bar + (s & 1));
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 4) tmem_dealloc(tmem_base, 512);
  cluster_sync_all();
  if (warp >= 8) {
    // this CTA's share of the tile: the sum over the parts in order
    const float* out = reinterpret_cast<const float*>(smem);
    for (int i = rank * 256 + threadIdx.x - 256; i < kT * kXN / 4; i += 256 * p.parts) {
      const int r = i / (kXN / 4), n = i % (kXN / 4) * 4;
      if (m0 + r >= p.M || n0 + n >= p.N) continue;
      float v[4] = {};
      for (int q = 0; q < p.parts; ++q) {
        float4 x;
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w)
                     : "r"(mapa_u32(out + r * kXN + n, q)));
        v[0] += x.x, v[1] += x.y, v[2] += x.z, v[3] += x.w;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (n0 + n + e < p.N) p.C[static_cast<size_t>(m0 + r) * p.ldc + n0 + n + e] = v[e];
    }
  }
  __syncwarp();
  cluster_sync_all();  // the others have read this CTA's partial tile
}

// Parts of K, from N and K alone: the fewest steps on the busiest of 148 SMs (one CTA each), where a CTA's start, its sum over the
// parts and its end cost about as much as three steps.
static int f32_parts(int N, int K) {
  const int tiles = (N + kXN - 1) / kXN, steps = (K + kXK - 1) / kXK;
  int best = 1;
  long long least = 1ll << 62;
  for (int parts = 1; parts <= kXMaxParts && parts <= steps; ++parts) {
    const long long cost = ((static_cast<long long>(tiles) * parts + 147) / 148) * ((steps + parts - 1) / parts + 3);
    if (cost < least) least = cost, best = parts;
  }
  return best;
}

template <int kT>
static int launch_gemm_f32(const F32Params& p, cudaStream_t stream) {
  using T = F32Tile<kT>;
  static bool configured[64] = {false};
  int dev = 0;
  B200_CHECK_CUDA(cudaGetDevice(&dev));
  if (!configured[dev & 63]) {
    B200_CHECK_CUDA(cudaFuncSetAttribute(gemm_f32_kernel<kT>, cudaFuncAttributeMaxDynamicSharedMemorySize, T::kSmem));
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
  B200_CHECK_CUDA(cudaLaunchKernelEx(&cfg, gemm_f32_kernel<kT>, p));
  return kOk;
}

}  // namespace b200

using namespace b200;

B200_API int b200_gemm_f32(const float* A, const float* B, float* C, int M, int N, int K, int lda, int ldb, int ldc,
                           void* stream) {
  B200_REQUIRE(M > 0 && N > 0 && K > 0, "empty problem %dx%dx%d", M, N, K);
  B200_REQUIRE(lda >= K && ldb >= K && ldc >= N, "leading dimensions are smaller than the rows");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  auto aligned = [](const float* x, int ld) { return ld % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0; };
  F32Params p = {A, B, C, M, N, K, f32_parts(N, K), 0, lda, ldb, ldc, aligned(A, lda), aligned(B, ldb)};
  p.part = ((K + p.parts - 1) / p.parts + kXK - 1) / kXK * kXK;
  // row tiles of even height: 100 rows are one of 112, 150 two of 80
  const int tiles = (M + 127) / 128, rows = (M + tiles - 1) / tiles;
  switch ((rows + 15) / 16) {
    case 1: return launch_gemm_f32<16>(p, s);
    case 2: return launch_gemm_f32<32>(p, s);
    case 3: return launch_gemm_f32<48>(p, s);
    case 4: return launch_gemm_f32<64>(p, s);
    case 5: return launch_gemm_f32<80>(p, s);
    case 6: return launch_gemm_f32<96>(p, s);
    case 7: return launch_gemm_f32<112>(p, s);
    default: return launch_gemm_f32<128>(p, s);
  }
}
