// Decode GEMM for at most 16 tokens whose tiles hold all of K: C[M, N] = X[M, K] W[N, K]^T, optionally
//   gamma      X is the residual stream h and the product is taken of RMSNorm(h) * gamma
//   residual   C = product + residual (the residual may be C itself)
//   dual       W = [gate; up], C = silu(X gate^T) * (X up^T)
//
// What bounds a decode step of a small layer is not the weights' bytes but what every kernel of its chain adds to them. The stream-K
// kernel of gemm_skinny_sm100.cu adds about 7 us: a tile's k-blocks lie on several SMs, so its sums meet in global memory (add and
// fence, ticket, re-read), behind the drain of the tensor core. Here a tile is a few rows of W and all of K: nothing meets outside the
// SM. Rows come in granules of eight, the narrow side of mma.m16n8k16 (the tokens are the 16), so that any N spreads over the SMs;
// a tcgen05 tile has 64 rows at least, which would leave most SMs of a 1280-row projection without one. The eight warps take
// the stages in turn, each with its own sums of all rows, which are added up once per tile through shared memory.
// The weights stream through a ring of TMA boxes of [k-blocks][rows][64] that starts to fill before the kernels in front are over.
// Every warp owns places of the ring and requests into them itself, which costs no second barrier and no producer: a producer thread for all
// warps took 270 clocks per stage (151936 x 4096, stages of 5 KB: 240 us for 189), and eight warps that share each stage 800 (370 us).
// What bounds it: from 4 K rows on the bytes in flight (150 KB of ring per SM), below that the start, the way of the
// activations into the SMs and the sums. 8 tokens, in a chain of such launches, us before (stream-K) and now: 1280 x 5120 7.7 -> 5.1, 5120 x
// 1024 8.0 -> 3.5, 3200 x 5120 gated 15.0 -> 11.7, 5120 x 3200 10.2 -> 7.3, 6144 x 4096 12.4 -> 9.9, 12288 x 4096 gated 35.2 -> 32.8,
// 4096 x 12288 19.1 -> 16.4, 151936 x 4096 190 -> 178 (7.0 TB/s). Fetching the next projections into L2 from here gained nothing.
//
// The norm costs no pass of its own: a warp multiplies the gain into its fragments of h (rounded once, as the separate kernel's
// result is), sums the squares of what it holds, and the row's factor is applied to the complete sums in fp32. The product with the gain must
// stay finite in the storage type, so this is for bf16.
//
// Role in the reference: F.linear, RMSNorm and the residual add of a decode step (python/triton_dist/layers/nvidia/tp_mlp.py:177-191,
// tp_attn.py:240-271, models/qwen.py:92-120).
#include "b200/elem.cuh"
#include "b200/host.h"
#include "b200/mma_sync.cuh"
#include "b200/primitives.cuh"
#include "b200/tcgen05.cuh"

#include <cstring>
#include <type_traits>

namespace b200 {

constexpr int kRowsBK = 64;            // elements of K per swizzled row
constexpr int kRowsWarps = 8;          // warps that multiply
constexpr int kRowsThreads = kRowsWarps * 32;
constexpr int kRowsMaxStages = 32;
constexpr int kRowsAhead = 2;          // fragments of W that are requested ahead of their products
constexpr int kRowsSmem = 204 * 1024;  // ring, sums and gain of a CTA; one CTA per SM

struct RowsParams {
  int M, N, K, ldc;
  int tiles, kbs, spans;     // tiles of rows; k-blocks per stage; stages per tile
  int stages, w_bytes, stage_bytes;
  int settled;               // W and gamma may be read before the kernels in front are over
  int out_f32;               // C is fp32 (of the values rounded to the storage type)
  float eps;
  const void* gamma;         // [K] or null
  const void* residual;      // [M, N], pitch ldc, or null
  void* C;
  uint32_t* status;          // raised when a wait expires; the tile's results are NaN then
};

__device__ __forceinline__ void ldmatrix_x2(uint32_t addr, uint32_t& r0, uint32_t& r1) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(addr));
}

// row pitch of the partial sums: 8 modulo 32 banks, so that the eight rows that a half warp writes lie side by side
constexpr int rows_pitch(int rows) { return (rows + 23) / 32 * 32 + 8; }
constexpr int rows_red_bytes(int mb, int rows) { return kRowsWarps * mb * rows_pitch(rows) * 4; }

// NG: granules of eight rows per tile and projection; MB: tokens, 8 or 16
template <bool BF16, int NG, int MB, bool kDual>
__global__ void __launch_bounds__(kRowsThreads)
gemm_rows_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const RowsParams p) {
  using T = typename std::conditional<BF16, __nv_bfloat16, __half>::type;
  constexpr int R = 8 * NG, kP = kDual ? 2 : 1, GT = kP * NG;
  constexpr int kPitch = rows_pitch(8 * GT);
  constexpr int kOut = (MB * R + 255) / 256;   // results per thread
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* red = reinterpret_cast<float*>(ring + p.stages * p.stage_bytes);               // [warps][MB][kPitch]
  uint32_t* s_gamma = reinterpret_cast<uint32_t*>(red + kRowsWarps * MB * kPitch);      // [K / 2] pairs
  __shared__ uint64_t full[kRowsMaxStages];
  __shared__ float s_sq[kRowsWarps][16];
  __shared__ int s_lost[kRowsWarps];   // stage whose wait a warp gave up
  __shared__ uint32_t abort_word;
  volatile uint32_t* abort_flag = &abort_word;
  const uint64_t timeout_ns = 4000000000ull;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int my_tiles = (p.tiles - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
  const int total = my_tiles * p.spans;   // stages of this CTA; warp w takes w, w + 8, ...
  griddep_launch_dependents();
  if (threadIdx.x == 0) abort_word = 0;
  // The first lane of a warp requests what the warp reads, into places that are the warp's own: at the start all of them (the
  // weights before the wait for the kernels in front), then each one again as soon as the warp has read it.
  int ask_tile = blockIdx.x, ask_span = warp, asked = warp;
  auto ask_next = [&]() {
    asked += kRowsWarps;
    ask_span += kRowsWarps;
    while (ask_span >= p.spans) { ask_span -= p.spans; ask_tile += gridDim.x; }
  };
  auto ask_w = [&](int slot, int tile, int span) {
    uint8_t* s = ring + slot * p.stage_bytes;
    mbar_expect_tx(full + slot, p.stage_bytes);
    tma_load_3d(s, &tmW, full + slot, 0, tile * R, span * p.kbs);
    if (kDual) tma_load_3d(s + p.w_bytes / 2, &tmW, full + slot, 0, p.N + tile * R, span * p.kbs);
  };
  auto ask_x = [&](int slot, int span) { tma_load_3d(ring + slot * p.stage_bytes + p.w_bytes, &tmX, full + slot, 0, 0, span * p.kbs); };
  while (ask_span >= p.spans) { ask_span -= p.spans; ask_tile += gridDim.x; }
  const int span0 = ask_span;
  if (lane == 0) {
    for (int slot = warp; slot < p.stages; slot += kRowsWarps) mbar_init(full + slot, 1);
    mbar_fence_init();
    if (!p.settled) {
      griddep_wait();
      fence_proxy_async();
    }
    for (int slot = warp; slot < p.stages && asked < total; slot += kRowsWarps, ask_next()) ask_w(slot, ask_tile, ask_span);
  }
  __syncwarp();
  if (p.gamma != nullptr) {
    if (!p.settled) griddep_wait();
    for (int i = threadIdx.x; i < p.K / 8; i += kRowsThreads) reinterpret_cast<uint4*>(s_gamma)[i] = static_cast<const uint4*>(p.gamma)[i];
  }
  if (lane == 0) {
    griddep_wait();
    fence_proxy_async();
    int span = span0;
    for (int slot = warp; slot < p.stages && slot < total; slot += kRowsWarps) {
      ask_x(slot, span);
      span += kRowsWarps;
      while (span >= p.spans) span -= p.spans;
    }
  }
  const int mi = lane >> 3, mr = lane & 7;
  __syncthreads();   // gamma, the abort word, and every warp's barriers
  // lane addresses inside a k-block of the activations and of a pair of granules (of the last one alone); chunks of 16 bytes
  // lie at their number xor the row's
  const uint32_t x_row = (MB == 16 ? (mi & 1) * 8 + mr : mr) * 128, x_chunk = MB == 16 ? mi >> 1 : mi & 1;
  const uint32_t w_row = ((mi >> 1) * 8 + mr) * 128, w_chunk = mi & 1;
  uint32_t x_at[4], w_at[4];   // of the four k16 steps of a k-block
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    x_at[i] = x_row + (((2 * i + x_chunk) ^ mr) << 4);
    w_at[i] = (((2 * i + w_chunk) ^ mr) << 4);
  }
  int at = warp, slot = warp;   // this warp's next stage, counted from the start of the CTA's work, and its place
  uint32_t phase = 0;
  bool ok = true;
  int first = 0;   // the tile's first stage
  for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x, first += p.spans) {
    float acc[GT][4];
#pragma unroll
    for (int g = 0; g < GT; ++g)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[g][e] = 0.f;
    float sq[2] = {0.f, 0.f};   // squares of tokens lane / 4 and eight further, this lane's channels
    for (; at < first + p.spans; at += kRowsWarps) {
      // After an expired wait the remaining rounds go by without work: all warps meet at the barriers below. One verdict per warp: the
      // fragment loads and products are instructions of all its lanes.
      if (ok) {
        const bool got = mbar_wait(full + slot, phase, abort_flag, timeout_ns);
        ok = __all_sync(0xffffffffu, got);
        if (!ok) s_lost[warp] = at;
      }
      if (ok) {
        uint32_t ws = smem_u32(ring + slot * p.stage_bytes), xs = ws + p.w_bytes;
        const uint32_t up = p.w_bytes / 2;
        int k = (at - first) * p.kbs * 32 + (lane & 3);   // pairs of channels
        for (int kb = 0; kb < p.kbs; ++kb, ws += R * 128, xs += MB * 128, k += 32) {
          constexpr int kPairs = (NG + 1) / 2, kUnits = kP * kPairs;   // per k16 step
          uint32_t x[4][4], b[kRowsAhead + 1][4];
          auto load_w = [&](int u) {
            const int step = u / kUnits, pr = u % kUnits / kPairs, g = u % kPairs * 2;
            uint32_t (&d)[4] = b[u % (kRowsAhead + 1)];
            if (g + 1 < NG) ldmatrix_x4(ws + pr * up + g * 1024 + w_row + w_at[step], d[0], d[1], d[2], d[3]);
            else ldmatrix_x2(ws + pr * up + g * 1024 + mr * 128 + w_at[step], d[0], d[1]);
          };
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            x[i][1] = x[i][3] = 0u;
            if (MB == 16) ldmatrix_x4(xs + x_at[i], x[i][0], x[i][1], x[i][2], x[i][3]);
            else ldmatrix_x2(xs + x_at[i], x[i][0], x[i][2]);
          }
#pragma unroll
          for (int u = 0; u < kRowsAhead; ++u) load_w(u);
          if (BF16 && p.gamma != nullptr && k < p.K / 2) {   // (behind K the activations are zero)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const __nv_bfloat162 g0 = reinterpret_cast<const __nv_bfloat162*>(s_gamma)[k + 8 * i];
              const __nv_bfloat162 g1 = reinterpret_cast<const __nv_bfloat162*>(s_gamma)[k + 8 * i + 4];
#pragma unroll
              for (int r = 0; r < 4; ++r) {
                if (MB == 8 && (r & 1)) continue;
                const float2 f = unpack_bf16x2(x[i][r]);
                sq[r & 1] = fmaf(f.x, f.x, fmaf(f.y, f.y, sq[r & 1]));
                const __nv_bfloat162 y = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&x[i][r]), r < 2 ? g0 : g1);
                x[i][r] = *reinterpret_cast<const uint32_t*>(&y);
              }
            }
          }
#pragma unroll
          for (int u = 0; u < 4 * kUnits; ++u) {
            if (u + kRowsAhead < 4 * kUnits) load_w(u + kRowsAhead);
            const int pr = u % kUnits / kPairs, g = u % kPairs * 2;
            const uint32_t (&d)[4] = b[u % (kRowsAhead + 1)];
            mma16816<BF16>(acc[pr * NG + g], x[u / kUnits], d[0], d[1]);
            if (g + 1 < NG) mma16816<BF16>(acc[pr * NG + (g + 1 < NG ? g + 1 : g)], x[u / kUnits], d[2], d[3]);
          }
        }
        __syncwarp();   // every lane has its fragments
        if (lane == 0 && asked < total) {
          ask_w(slot, ask_tile, ask_span);
          ask_x(slot, ask_span);
          ask_next();
        }
      }
      slot += kRowsWarps;
      if (slot >= p.stages) { slot = warp; phase ^= 1; }
    }
    // ---- sums of the eight warps
    const int row = lane >> 2, col = (lane & 3) * 2;
#pragma unroll
    for (int g = 0; g < GT; ++g) {
      float* sum = red + (warp * MB + row) * kPitch + g * 8 + col;
      *reinterpret_cast<float2*>(sum) = make_float2(acc[g][0], acc[g][1]);
      if (MB == 16) *reinterpret_cast<float2*>(sum + 8 * kPitch) = make_float2(acc[g][2], acc[g][3]);
    }
    if (p.gamma != nullptr) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        sq[h] += __shfl_xor_sync(0xffffffffu, sq[h], 1);
        sq[h] += __shfl_xor_sync(0xffffffffu, sq[h], 2);
        if ((lane & 3) == 0) s_sq[warp][row + 8 * h] = sq[h];
      }
    }
    griddep_wait();   // the residual, and what the kernels in front may still read where C lies
    float res[kOut];
#pragma unroll
    for (int j = 0; j < kOut; ++j) {
      const int i = threadIdx.x + j * 256, m = i / R, n = tile * R + i % R;
      res[j] = p.residual != nullptr && m < p.M && n < p.N ? to_float(static_cast<const T*>(p.residual)[static_cast<size_t>(m) * p.ldc + n]) : 0.f;
    }
    const bool whole = __syncthreads_and(ok);   // no warp gave up, or the sums lack its share
#pragma unroll
    for (int j = 0; j < kOut; ++j) {
      const int i = threadIdx.x + j * 256, m = i / R, n = tile * R + i % R;
      if (m >= p.M || n >= p.N) continue;
      float v = 0.f, u = 0.f;
#pragma unroll
      for (int w = 0; w < kRowsWarps; ++w) {
        const float* sum = red + (w * MB + m) * kPitch + i % R;
        v += sum[0];
        if (kDual) u += sum[R];
      }
      if (p.gamma != nullptr) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < kRowsWarps; ++w) s += s_sq[w][m];
        s = rsqrtf(s / static_cast<float>(p.K) + p.eps);
        v *= s;
        u *= s;
      }
      if (kDual) v = v / (1.f + __expf(-v)) * u;
      const T y = from_float<T>(whole ? v + res[j] : NAN);
      const size_t to = static_cast<size_t>(m) * p.ldc + n;
      if (p.out_f32) static_cast<float*>(p.C)[to] = to_float(y);
      else static_cast<T*>(p.C)[to] = y;
    }
    __syncthreads();   // the next tile's sums take the same place
  }
  if (!ok && lane == 0) {   // boxes that are on their way have to land before shared memory is given back
    volatile uint32_t never = 0;
    for (int i = s_lost[warp]; i < asked; i += kRowsWarps) {
      const int round = i / kRowsWarps, places = p.stages / kRowsWarps;   // of this warp
      mbar_wait(full + warp + round % places * kRowsWarps, round / places & 1, &never, timeout_ns);
    }
  }
  if (threadIdx.x == 0 && abort_word != 0u && p.status != nullptr) atomicMax(p.status, static_cast<uint32_t>(kStatusPipeTimeout));
}

using RowsKernel = void (*)(const CUtensorMap, const CUtensorMap, const RowsParams);
template <bool BF16, int MB, bool kDual>
static RowsKernel rows_kernel(int granules) {
  switch (granules) {
    case 1: return gemm_rows_kernel<BF16, 1, MB, kDual>;
    case 2: return gemm_rows_kernel<BF16, 2, MB, kDual>;
    case 3: return gemm_rows_kernel<BF16, 3, MB, kDual>;
    case 4: return gemm_rows_kernel<BF16, 4, MB, kDual>;
    case 5: return gemm_rows_kernel<BF16, 5, MB, kDual>;
    default: return gemm_rows_kernel<BF16, 6, MB, kDual>;
  }
}
constexpr int kRowsMaxGranules = 6;

}  // namespace b200

using namespace b200;

// X [M <= 16, K] (pitch ldx), W [N, K] or [2 N, K] (dual; pitch ldw), C [M, N] (pitch ldc) of the same type (fp32 with out_f32).
// gamma [K] (bf16 only) and residual [M, N] (pitch ldc) may be null. K must be a multiple of 64. dtype + kSettled: see host.h.
B200_API int b200_gemm_rows(const void* X, const void* W, void* C, int M, int N, int K, int ldx, int ldw, int ldc, int dual,
                            const void* gamma, float eps, const void* residual, int out_f32, int dtype, uint32_t* status, void* stream) {
  const bool settled = take_settled(dtype);
  B200_REQUIRE(dtype == kBF16 || dtype == kF16, "gemm_rows supports bf16/f16");
  B200_REQUIRE(M >= 1 && M <= 16 && N >= 1, "gemm_rows handles 1..16 tokens, got %d", M);
  B200_REQUIRE(K >= 64 && K % 64 == 0, "gemm_rows: K (%d) must be a multiple of 64", K);
  B200_REQUIRE(gamma == nullptr || (dtype == kBF16 && K <= 16384 && reinterpret_cast<uintptr_t>(gamma) % 16 == 0),
               "gemm_rows: the norm is for bf16, K <= 16384 and a gain on a 16-byte boundary");
  B200_REQUIRE(!(dual && residual), "gemm_rows: a gated product has no residual");
  RowsParams p;
  memset(&p, 0, sizeof(p));
  p.M = M; p.N = N; p.K = K; p.ldc = ldc;
  p.settled = settled; p.out_f32 = out_f32; p.eps = eps; p.gamma = gamma; p.residual = residual; p.C = C; p.status = status;
  const int mb = M <= 8 ? 8 : 16, proj = dual ? 2 : 1, sms = sm_count();
  // The tile height with the least rows on the busiest SM; a tile's sums and results take about as long as two rows, and a ring of
  // less than 140 KB keeps too little in flight. Measured at 8 tokens, all heights: 12288 x 4096 gated 31.6 .. 35.8 us (this rule 32.8),
  // 6144 x 4096 9.9 .. 14.8 (9.9), 151936 x 4096 176 .. 241 (178).
  const int budget = kRowsSmem - 1024 - (gamma ? K * 2 : 0), num_kb = K / kRowsBK;
  int granules = 1, units = 1;
  float best = 0.f;
  for (int g = 1; g <= kRowsMaxGranules; ++g) {
    const int rows = 8 * g * proj, unit = (rows + mb) * 128 * kRowsWarps;   // bytes of one k-block for every warp
    const int n = (budget - rows_red_bytes(mb, rows)) / unit;
    if (n < 1) break;
    const long long tiles = (N + 8 * g - 1) / (8 * g);
    const float flight = n * unit < 140 * 1024 ? static_cast<float>(n * unit) / (140 * 1024) : 1.f;
    const float cost = static_cast<float>((tiles + sms - 1) / sms * (8 * g + 2)) * (1.3f - 0.3f * flight);
    if (g == 1 || cost <= best) { best = cost; granules = g; units = n; }
  }
  const int R = 8 * granules;
  p.tiles = (N + R - 1) / R;
  // Two stages or more per warp (1280 x 5120, 150 KB in flight: 5.1 us with two, 6.3 with one), none longer than a warp's share of K
  const int even = (num_kb + kRowsWarps - 1) / kRowsWarps;
  p.kbs = units / 2 < 1 ? 1 : units / 2 > 8 ? 8 : units / 2;
  if (p.kbs > even) p.kbs = even;
  p.spans = (num_kb + p.kbs - 1) / p.kbs;
  p.w_bytes = p.kbs * R * 128 * proj;
  p.stage_bytes = p.w_bytes + p.kbs * mb * 128;
  const int grid = p.tiles < sms ? p.tiles : sms;
  const int rounds = (p.tiles + grid - 1) / grid * p.spans;
  p.stages = units / p.kbs * kRowsWarps;
  if (p.stages > kRowsMaxStages) p.stages = kRowsMaxStages;
  while (p.stages > kRowsWarps && p.stages - kRowsWarps >= rounds) p.stages -= kRowsWarps;
  const int smem = 1024 + p.stages * p.stage_bytes + rows_red_bytes(mb, R * proj) + (gamma ? K * 2 : 0);
  CUtensorMap tw, tx;
  int rc = make_tma_3d(&tw, W, dtype, kRowsBK, static_cast<uint64_t>(proj) * N, num_kb, ldw, kRowsBK, kRowsBK, R, p.kbs, true);
  if (rc != kOk) return rc;
  rc = make_tma_3d(&tx, X, dtype, kRowsBK, M, num_kb, ldx, kRowsBK, kRowsBK, mb, p.kbs, true);
  if (rc != kOk) return rc;
  RowsKernel kernel;
  if (dtype == kBF16)
    kernel = dual ? (mb == 8 ? rows_kernel<true, 8, true>(granules) : rows_kernel<true, 16, true>(granules))
                  : (mb == 8 ? rows_kernel<true, 8, false>(granules) : rows_kernel<true, 16, false>(granules));
  else
    kernel = dual ? (mb == 8 ? rows_kernel<false, 8, true>(granules) : rows_kernel<false, 16, true>(granules))
                  : (mb == 8 ? rows_kernel<false, 8, false>(granules) : rows_kernel<false, 16, false>(granules));
  // once per device and kernel, with what the largest launch needs (about 1 us of host time)
  static bool configured[64][2][2][2][kRowsMaxGranules] = {};
  int dev = 0;
  B200_CHECK_CUDA(cudaGetDevice(&dev));
  bool& done = configured[dev & 63][dtype == kBF16][dual != 0][mb == 16][granules - 1];
  if (!done) {
    B200_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowsSmem));
    done = true;
  }
  B200_CHECK_CUDA(launch_pdl(kernel, dim3(grid), dim3(kRowsThreads), static_cast<size_t>(smem), static_cast<cudaStream_t>(stream), tw, tx, p));
  return kOk;
}
