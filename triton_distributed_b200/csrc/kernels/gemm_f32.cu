// fp32 GEMM for the models' 32-bit mode: C[M,N] = A[M,K] * B[N,K]^T, true fp32 products and sums (no TF32).
//
// A CTA of 128 threads computes a BM x BN tile over one part of K; the parts of a tile are a cluster, whose CTAs add their partial
// tiles through distributed shared memory in rank order. The number of parts depends on N and K alone and the sum inside a part
// runs in the order of K, so a row's result does not depend on how many other rows share the call. Any M, N, K, leading
// dimensions and alignment.
//
// What bounds it: for many rows the fp32 pipe, fed by two shared-memory reads of 16 bytes for 32 products (a thread has 8 x 8
// outputs) and held back by register-bank conflicts of the products; for few rows the bytes of B. Operands stay as they are in
// memory, rows of 32 consecutive k: cp.async brings them in three or four stages, and with a pitch of 36 words eight
// neighbouring rows are read without a bank conflict. Above 32 rows tiles are up to 64 x 128, of equal height (100 rows: two of
// 56 instead of one of 64 and a rest); below, fewer rows would multiply padding, and 64 columns keep enough CTAs (bytes in
// flight) at narrow N.
// Measured against a 64 x 64 tile per CTA over all of K with 4 x 4 outputs per thread (11264 x 2048 and 2048 x 5632, us):
//   M = 1    218, 398 -> 34, 27      M = 16   219, 397 -> 43, 32      M = 32  220, 396 -> 61, 47
//   M = 100  241, 379 -> 171, 79     M = 256  403, 447 -> 333, 189    M = 1024  1489, 894 -> 1283, 725
// Products of two neighbours in k at a time (fma.rn.f32x2) were no faster: 36 instead of 40 TFLOP/s at 1024 x 22016 x 4096.
#include "b200/host.h"
#include "b200/primitives.cuh"
#include "b200/tcgen05.cuh"

namespace b200 {

constexpr int kFK = 32, kFPitch = kFK + 4, kFThreads = 128, kFMaxParts = 8;

// Thread tiles are TM x TN, lanes 4 x 8, warps kWarpsM x (4 / kWarpsM); rows (columns) of a thread lie 4 (8) apart.
template <int TM, int TN, int kWarpsM>
struct F32Tile {
  static constexpr int BM = kWarpsM * 4 * TM, BN = 4 / kWarpsM * 8 * TN;
  static constexpr int kStages = BN == 128 ? 3 : 4;
  static constexpr int kStage = (BM + BN) * kFPitch;  // floats
  static constexpr int kOutPitch = BN + 8;
  static constexpr int kSmem = 4 * (kStages * kStage > BM * kOutPitch ? kStages * kStage : BM * kOutPitch);
};

__device__ __forceinline__ void cp_async_16(float* dst, const float* src, int bytes) {  // zeros behind `bytes`
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_4(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

// `rows` rows of kFK columns from (r0, k0) of X [count, kend] into shared memory: zeros behind the last column; behind the last row
// that row again (its results are not stored). `vec`: rows start on 16 bytes.
template <int rows>
__device__ __forceinline__ void f32_load(float* dst, const float* __restrict__ X, int r0, int count, int k0, int kend, int ld, bool vec) {
  constexpr int kChunks = kFK / 4;
  const int chunk = threadIdx.x % kChunks, k = k0 + 4 * chunk;
  const int left = min(4, max(0, kend - k));
  const float* src = X + (left > 0 ? k : 0);
#pragma unroll
  for (int r = threadIdx.x / kChunks; r < rows; r += kFThreads / kChunks) {
    const float* from = src + static_cast<size_t>(min(r0 + r, count - 1)) * ld;
    float* to = dst + r * kFPitch + 4 * chunk;
    if (vec) {
      cp_async_16(to, from, 4 * left);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) cp_async_4(to + e, e < left ? from + e : from, e < left ? 4 : 0);
    }
  }
}

template <int TM, int TN, int kWarpsM>
__global__ void __launch_bounds__(kFThreads) gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ B,
                                                             float* __restrict__ C, int M, int N, int K, int parts, int part, int lda,
                                                             int ldb, int ldc, bool vec_a, bool vec_b) {
  using T = F32Tile<TM, TN, kWarpsM>;
  extern __shared__ __align__(16) float sm[];
  const int rank = blockIdx.x % parts;  // in the cluster
  const int n0 = blockIdx.x / parts * T::BN, m0 = blockIdx.y * T::BM;
  const int k_begin = rank * part, k_end = min(K, k_begin + part);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = warp % kWarpsM * (4 * TM) + (lane >> 3), col = warp / kWarpsM * (8 * TN) + (lane & 7);
  griddep_launch_dependents();
  griddep_wait();
  const int steps = (k_end - k_begin + kFK - 1) / kFK;
  auto load = [&](int s) {
    if (s < steps) {
      float* st = sm + s % T::kStages * T::kStage;
      f32_load<T::BM>(st, A, m0, M, k_begin + s * kFK, k_end, lda, vec_a);
      f32_load<T::BN>(st + T::BM * kFPitch, B, n0, N, k_begin + s * kFK, k_end, ldb, vec_b);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int s = 0; s < T::kStages - 1; ++s) load(s);
  float acc[TM][TN] = {};
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(T::kStages - 2) : "memory");
    __syncthreads();  // stage s has landed for all, and stage s - 1 has been read by all
    load(s + T::kStages - 1);
    const float* sa = sm + s % T::kStages * T::kStage + row * kFPitch;
    const float* sb = sm + s % T::kStages * T::kStage + (T::BM + col) * kFPitch;
#pragma unroll
    for (int k = 0; k < kFK; k += 4) {
      float4 a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(sa + 4 * i * kFPitch + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(sb + 8 * j * kFPitch + k);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();  // the stages give way to the partial tile
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) sm[(row + 4 * i) * T::kOutPitch + col + 8 * j] = acc[i][j];
  cluster_sync_all();
  // this CTA's share of the tile: the sum over the parts in order
  const int share = T::BM * T::BN / 4 / parts;  // BM * BN is a multiple of 4 * kFMaxParts
  for (int c = threadIdx.x; c < share; c += kFThreads) {
    const int at = rank * share + c, r = at / (T::BN / 4), n = at % (T::BN / 4) * 4;
    if (m0 + r >= M || n0 + n >= N) continue;
    float v[4] = {};
    for (int q = 0; q < parts; ++q) {
      float4 x;
      asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                   : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w)
                   : "r"(mapa_u32(sm + r * T::kOutPitch + n, q)));
      v[0] += x.x, v[1] += x.y, v[2] += x.z, v[3] += x.w;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (n0 + n + e < N) C[static_cast<size_t>(m0 + r) * ldc + n0 + n + e] = v[e];
  }
  cluster_sync_all();  // the others have read this CTA's partial tile
}

// Parts of K: up to eight while there are fewer than about two CTAs per SM from N alone, each at least two steps of K.
static int f32_parts(int N, int K) {
  int parts = 1;
  while (parts < kFMaxParts && (N + 127) / 128 * parts * 2 <= 600 && K >= parts * 2 * 2 * kFK) parts *= 2;
  return parts;
}

template <int TM, int TN, int kWarpsM>
static int launch_gemm_f32(const float* A, const float* B, float* C, int M, int N, int K, int lda, int ldb, int ldc, cudaStream_t stream) {
  using T = F32Tile<TM, TN, kWarpsM>;
  const int parts = f32_parts(N, K), part = ((K + parts - 1) / parts + kFK - 1) / kFK * kFK;
  static bool configured[64] = {false};
  int dev = 0;
  B200_CHECK_CUDA(cudaGetDevice(&dev));
  if (!configured[dev & 63]) {
    B200_CHECK_CUDA(cudaFuncSetAttribute(gemm_f32_kernel<TM, TN, kWarpsM>, cudaFuncAttributeMaxDynamicSharedMemorySize, T::kSmem));
    configured[dev & 63] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((N + T::BN - 1) / T::BN * parts, (M + T::BM - 1) / T::BM);
  cfg.blockDim = dim3(kFThreads);
  cfg.dynamicSmemBytes = T::kSmem;
  cfg.stream = stream;
  B200_REQUIRE(cfg.gridDim.y <= 65535, "M (%d) is too large", M);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = parts;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  auto aligned = [](const float* p, int ld) { return ld % 4 == 0 && reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  B200_CHECK_CUDA(cudaLaunchKernelEx(&cfg, gemm_f32_kernel<TM, TN, kWarpsM>, A, B, C, M, N, K, parts, part, lda, ldb, ldc, aligned(A, lda),
                                     aligned(B, ldb)));
  return kOk;
}

}  // namespace b200

using namespace b200;

B200_API int b200_gemm_f32(const float* A, const float* B, float* C, int M, int N, int K, int lda, int ldb, int ldc,
                           void* stream) {
  B200_REQUIRE(M > 0 && N > 0 && K > 0, "empty problem %dx%dx%d", M, N, K);
  B200_REQUIRE(lda >= K && ldb >= K && ldc >= N, "leading dimensions are smaller than the rows");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (M <= 8) return launch_gemm_f32<2, 2, 1>(A, B, C, M, N, K, lda, ldb, ldc, s);     // 8 x 64
  if (M <= 16) return launch_gemm_f32<4, 2, 1>(A, B, C, M, N, K, lda, ldb, ldc, s);    // 16 x 64
  if (M <= 32) return launch_gemm_f32<4, 4, 2>(A, B, C, M, N, K, lda, ldb, ldc, s);    // 32 x 64
  const int tiles = (M + 63) / 64, rows = (M + tiles - 1) / tiles;                     // even tiles of up to 64 rows x 128
  if (rows <= 40) return launch_gemm_f32<5, 8, 2>(A, B, C, M, N, K, lda, ldb, ldc, s);
  if (rows <= 48) return launch_gemm_f32<6, 8, 2>(A, B, C, M, N, K, lda, ldb, ldc, s);
  if (rows <= 56) return launch_gemm_f32<7, 8, 2>(A, B, C, M, N, K, lda, ldb, ldc, s);
  return launch_gemm_f32<8, 8, 2>(A, B, C, M, N, K, lda, ldb, ldc, s);
}
