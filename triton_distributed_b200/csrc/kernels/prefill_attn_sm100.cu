// Causal (or full) variable-length prefill attention for sm_100a, GQA, bf16 / f16, query / key sizes up to 256, any value
// size, with an optional sink logit per head (one more term of the softmax denominator, without a value).
//
//   out[q, h, :] = softmax(scale * Q[q, h, :] . K[keys of q's sequence, kvh(h), :]^T) V[...]     (bottom-right causal mask)
//
// A CTA works on two tiles of 128 query rows at a time and walks the keys in steps of 128. The tiles are the same rows of two
// heads that share a KV head, or, where the group size is odd, two row blocks of one head: either way both tiles use the K and V
// tiles in shared memory. While the softmax of one tile runs, the tensor core computes the other tile's products (two tiles in
// turn: published as ping-pong scheduling, FlashAttention-3, Shah et al. 2024):
//   warps 0-3   softmax of tile 0, one thread per query row
//   warps 4-7   softmax of tile 1
//   warps 8-11  rescale O of either tile while the softmax warps compute the exponentials, and store the finished rows (not in small
//               calls, where the softmax warps do both: prefill_helped; the warps below are 8 to 10 then)
//   warp 12     TMA producer: both Q tiles of an item, then K and V tiles through their rings (128-byte swizzle)
//   warp 13     one elected thread issues tcgen05.mma, for each step and tile O += P V of this step, then S = Q K^T of the next
//   warp 14     asks the hardware for the next item (cluster launch control) while the current one is worked on
// Tensor memory: S of tile t at columns 128 t, O of tile t at 256 + 128 t. The softmax thread reads its row of S, keeps it in
// registers, and writes P as 16-bit pairs over the same columns: P is the A operand of the second product straight from tensor
// memory. O stays in tensor memory; the rows of a warp are rescaled when one of them has a new maximum. A reference that lags behind
// the maximum would do (by up to 2^8), but it costs precision: a row's largest weight is one, which
// 16 bits hold exactly, only while the reference is the maximum itself (error against 64 bits 2.07e-3 of the norm for 2.03e-3).
// The sum over all keys is the tensor core's running fp32 sum, which truncates where the former kernel added the sums of 128 keys to
// registers: no difference in the error of random values (2.03e-3 on the pack, 2.11e-3 over 16384 keys in bf16, 2.63e-4 in f16);
// with values of mean one, results over 16384 keys lie 3.8e-5 low, which shows in f16 alone (2.26e-4 for 2.22e-4).
// V is read in place, row-major, as an MN-major operand (b200_prefill_attention_vt reads V^T as a K-major one). Rows behind a
// sequence's last key belong to others: their scores are masked and their values are zeroed in shared memory, so nothing that
// stands there (not even NaN) reaches the output.
// The kernel is compiled for 1 to 4 column blocks of 64 in a query / key row; columns beyond the row are zero-filled by TMA. Up to
// two blocks the K and V rings have two stages, with three K has two, with four both have one, which is what shared memory holds.
// Every barrier wait is bounded; on expiry the CTA unwinds through an abort flag and reports a status.
//
// What bounds it: a tile's chain of softmax and both products (with nothing but the products the pack below takes 315 us, without the
// exponentials 370, without the rescaling 390), and in long calls the power cap. The special-function unit and the tensor core are busy 42 % of
// the time each. Rescaling and storing by the softmax warps themselves took 450 us where it is 424 now; stored row by row from the registers
// it was 525, since a warp that stores 32 rows at a time keeps the next item's rescaling waiting. Two threads per row (16 softmax warps)
// took 524 us for 508 over changing inputs, steps of 64 keys with the next step's scores in front of this step's product 565 for 500: products of
// 64 columns are slow.
// One query tile per CTA, P through shared memory, O in registers and a launch that transposed V
// before it took 769 us for five causal sequences of 1 K to 3 K tokens (64 / 8 heads, bf16) and 851 for one of 16384 (8 / 1 heads);
// the softmax warps rescaling 450 and 516.
//
// Role in the reference: flash_attn_with_kvcache in layers/nvidia/tp_attn.py:194-195 (prefill) and the Triton
// flash-attention consumer of the sequence-parallel all-gather path, kernels/nvidia/sp_ag_attention_intra_node.py:255-425.
#include "b200/host.h"
#include "b200/packed_f32.cuh"
#include "b200/primitives.cuh"
#include "b200/tcgen05.cuh"

#include <cstring>

namespace b200 {

constexpr int kPD = 128;                    // value columns per CTA
constexpr int kPM = 128, kPN = 128;         // query rows per tile, keys per step
constexpr int kPAtom = 128 * 64 * 2;        // one 128-row x 64-column 16-bit swizzle atom: 16 KB
constexpr int kPTile = 2 * kPAtom;          // a 128 x 128 tile: 32 KB
constexpr int prefill_k_stages(int dk_atoms) { return dk_atoms <= 3 ? 2 : 1; }
constexpr int prefill_v_stages(int dk_atoms) { return dk_atoms <= 2 ? 2 : 1; }
// Output rows go to memory through shared memory, a warp's 32 rows at once, where rows of Q and K leave 32 KB for it.
constexpr bool prefill_staged(int dk_atoms) { return dk_atoms <= 2; }
constexpr int prefill_smem(int dk_atoms, bool helped) {
  return 2 * dk_atoms * kPAtom /*Q*/ + prefill_k_stages(dk_atoms) * dk_atoms * kPAtom /*K*/ + prefill_v_stages(dk_atoms) * kPTile /*V*/ +
         1024 + 256 + (helped ? 2 * kPM * 4 /*factors*/ + (prefill_staged(dk_atoms) ? kPM * kPD * 2 : 0) : 0);
}
// 512 threads start with 128 registers each; 2 x 128 x softmax + 128 x rescaling + 128 x others is the same total. Who stores needs more.
// 384 threads (without the rescaling warps) start with 168: 2 x 128 x 216 + 128 x 72.
constexpr int prefill_threads(bool helped) { return helped ? 512 : 384; }
constexpr int prefill_softmax_regs(int dk_atoms, bool helped) { return !helped ? 216 : prefill_staged(dk_atoms) ? 176 : 184; }
constexpr int prefill_scale_regs(int dk_atoms) { return prefill_staged(dk_atoms) ? 88 : 72; }
constexpr int kPOtherRegs = 72;

struct PrefillParams {
  int Hq, Hkv, causal, bf16;
  int dk, dv;           // query / key and value sizes of a head
  int v_chunks;         // ceil(dv / 128): items per (query rows, head), each with up to 128 columns of the values
  int v_packed;         // V^T is given, [Hkv, dv, total_k], a sequence's keys at columns cu_k[b] ...; else V [total_k, Hkv, dv]
  int pair_heads;       // tiles are two heads of a KV head (even group size); else two row blocks of a head
  const float* sink;    // nullable [Hq]
  const void* gate;     // nullable [total_q, Hq] (row pitch ldg): every head's output is multiplied by sigmoid(gate)
  int ldg;
  const int* cu_q;      // [B + 1] first packed query row of every sequence
  const int* cu_k;      // [B + 1] first key row of every sequence (only [0, B) is read when k_lens is given)
  const int* k_lens;    // nullable [B]: keys of every sequence; null = cu_k[b + 1] - cu_k[b] (packed sequences)
  float scale_log2e;    // softmax scale * log2(e)
  void* out;            // [total_q, Hq, dv]
  uint32_t* status;     // nullable: set non-zero when a pipeline wait expired
};

// 2^x on the special-function unit (one instruction; -inf gives 0, which is what a masked score must contribute)
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// What a CTA works on at a time, from the block coordinates of the launch grid: x = (heads or head pairs) x value chunks, y = row
// blocks from the last one down (under the causal mask the long ones start first), z = sequence.
struct PrefillItem {
  int b, v_col0, kvh;
  int head[2], m_blk[2], steps[2];  // per tile; steps = 0: nothing to attend (or no such rows)
  int q_start, q_len, k_start, k_len;
  int n;  // max of steps
  // by a tile that is not known when compiling, without indexing (which would put the item into local memory)
  __device__ int steps_of(int t) const { return t == 0 ? steps[0] : steps[1]; }
  __device__ int head_of(int t) const { return t == 0 ? head[0] : head[1]; }
  __device__ int m_blk_of(int t) const { return t == 0 ? m_blk[0] : m_blk[1]; }
};
__device__ __forceinline__ PrefillItem prefill_item(const PrefillParams& p, uint3 at, int grid_y) {
  PrefillItem w;
  const int hx = at.x / p.v_chunks, y = grid_y - 1 - at.y;
  w.b = at.z;
  w.v_col0 = (at.x - hx * p.v_chunks) * kPD;
  w.q_start = p.cu_q[w.b];
  w.q_len = p.cu_q[w.b + 1] - w.q_start;
  w.k_start = p.cu_k[w.b];
  w.k_len = p.k_lens ? p.k_lens[w.b] : p.cu_k[w.b + 1] - w.k_start;
  w.kvh = (p.pair_heads ? 2 * hx : hx) / (p.Hq / p.Hkv);
  w.n = 0;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    w.head[t] = p.pair_heads ? 2 * hx + t : hx;
    w.m_blk[t] = p.pair_heads ? y : 2 * y + t;
    int kv_end = w.k_len;
    if (p.causal) kv_end = max(0, min(w.k_len, w.m_blk[t] * kPM + kPM + w.k_len - w.q_len));  // bottom-right alignment
    w.steps[t] = w.m_blk[t] * kPM < w.q_len ? (kv_end + kPN - 1) / kPN : 0;
    w.n = max(w.n, w.steps[t]);
  }
  return w;
}

// Stores a warp's 32 rows of a tile's output times inv. Staged: through 8 KB of shared memory, two whole rows per instruction;
// o_empty is signalled as soon as the rows have left tensor memory.
template <bool kStaged, bool BF16>
__device__ __forceinline__ void prefill_store(const PrefillParams& p, const PrefillItem& w, int t, int steps, uint32_t o_addr, float inv,
                                              uint8_t* stg, uint64_t* o_empty) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q_pos = w.m_blk_of(t) * kPM + (warp & 3) * 32 + lane;
  const bool store = q_pos < w.q_len;
  const size_t pitch = static_cast<size_t>(p.Hq) * p.dv * 2;   // from a token to the next
  uint8_t* dst = static_cast<uint8_t*>(p.out) + static_cast<size_t>(w.q_start + q_pos) * pitch + (static_cast<size_t>(w.head_of(t)) * p.dv + w.v_col0) * 2;
  // 16-byte chunk c of this thread's row lies at number c xor lane % 8 (opaque: the sixteen addresses would be kept, and spill)
  uint32_t mine = smem_u32(stg + lane * 256 + (lane & 7) * 16);
  asm volatile("" : "+r"(mine));
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t o[32];
    if (steps > 0) {
      tmem_ld_32x32(o_addr + c * 32, o);
      tmem_ld_wait();
    } else {
#pragma unroll
      for (int e = 0; e < 32; ++e) o[e] = 0u;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float a = __uint_as_float(o[q * 8 + 2 * e]) * inv, b = __uint_as_float(o[q * 8 + 2 * e + 1]) * inv;
        v[e] = BF16 ? pack_bf16x2(a, b) : pack_f16x2(a, b);
      }
      if (kStaged)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(mine ^ ((c * 4 + q) * 16)), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
      else if (store && w.v_col0 + c * 32 + q * 8 < p.dv)
        *reinterpret_cast<uint4*>(dst + c * 64 + q * 16) = make_uint4(v[0], v[1], v[2], v[3]);
    }
  }
  if (steps > 0) {
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) mbar_arrive(o_empty);
  }
  if (kStaged) {   // two whole rows per store
    __syncwarp();
    const int chunk = lane & 15;
    const bool in = w.v_col0 + chunk * 8 < p.dv;
    const uint8_t* from = stg + (lane >> 4) * 256;
    uint8_t* to = dst + chunk * 16 - (lane - (lane >> 4)) * pitch;   // of row lane / 16 of the warp
    int left = w.q_len - (q_pos - lane) - (lane >> 4);               // rows from there to the sequence's end
#pragma unroll 4
    for (int r = 0; r < 32; r += 2, left -= 2, to += 2 * pitch) {
      const uint4 v4 = *reinterpret_cast<const uint4*>(from + r * 256 + (chunk ^ ((r + (lane >> 4)) & 7)) * 16);
      if (in && left > 0) *reinterpret_cast<uint4*>(to) = v4;
    }
    __syncwarp();
  }
}

// kHelped: four more warps rescale and, where shared memory allows, store
template <int kDkAtoms, bool BF16, bool kHelped>
__global__ void __launch_bounds__(prefill_threads(kHelped), 1)
prefill_attn_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const PrefillParams p) {
  constexpr int kKSt = prefill_k_stages(kDkAtoms), kVSt = prefill_v_stages(kDkAtoms);
  constexpr int kQkTile = kDkAtoms * kPAtom;
  constexpr bool kStaged = kHelped && prefill_staged(kDkAtoms);
  constexpr int kProducer = kHelped ? 12 : 8;   // the first warp behind those of the rows
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                   // [2 tiles][atoms]
  uint8_t* sK = sQ + 2 * kQkTile;       // [stages][atoms]
  uint8_t* sV = sK + kKSt * kQkTile;    // [stages][2 atoms]: rows = keys (V) or value columns (V^T)
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + kVSt * kPTile);
  uint64_t* q_full = bars;          // [1]
  uint64_t* q_empty = bars + 1;     // [1]
  uint64_t* k_full = bars + 2;      // [2]
  uint64_t* k_empty = bars + 4;     // [2]
  uint64_t* v_full = bars + 6;      // [2]
  uint64_t* v_empty = bars + 8;     // [2]
  uint64_t* s_full = bars + 10;     // [2 tiles] scores are in tensor memory (and the tile's earlier products are done)
  uint64_t* p_full = bars + 12;     // [2 tiles] probabilities are in tensor memory, and the output has been rescaled
  uint64_t* o_full = bars + 14;     // [2 tiles] the item's last product is done
  uint64_t* o_empty = bars + 16;    // [2 tiles] the item's output has been read
  uint64_t* next_full = bars + 18;  // [1]
  uint64_t* next_empty = bars + 19; // [1]
  uint4* next_item = reinterpret_cast<uint4*>(bars + 20);  // 16-byte answer of the launch control
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 22);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  uint64_t* c_full = bars + 24;     // [2 tiles] a step's factors of the output have been written
  uint64_t* f_full = bars + 26;     // [2 tiles] an item's last factors have been written
  float* s_factor = reinterpret_cast<float*>(bars + 32);   // [2 tiles][128 rows]
  uint8_t* s_out = reinterpret_cast<uint8_t*>(s_factor + 2 * kPM);   // [4 warps][32 rows][256 bytes]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t timeout_ns = 4000000000ull;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(k_full + i, 1);
      mbar_init(k_empty + i, 1);
      mbar_init(v_full + i, 1);
      mbar_init(v_empty + i, 1);
      mbar_init(s_full + i, 1);
      mbar_init(p_full + i, kHelped ? 8 : 4);
      mbar_init(o_full + i, 1);
      mbar_init(o_empty + i, 4);
      mbar_init(c_full + i, 4);
      mbar_init(f_full + i, 4);
    }
    mbar_init(next_full, 1);
    mbar_init(next_empty, kProducer + 2);  // producer, MMA issuer and all warps in front of them
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == kProducer + 3) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  uint3 at = make_uint3(blockIdx.x, blockIdx.y, blockIdx.z);

  // Moves on to the next item (a single thread's or a whole warp's call); false when there is none. `i` counts this CTA's items.
  auto advance = [&](int i, bool warp_wide) -> bool {
    bool ok = mbar_wait(next_full, i & 1, abort_flag, timeout_ns);
    if (warp_wide) ok = __all_sync(0xffffffffu, ok);
    if (!ok) return false;
    const bool more = clc_read(next_item, at);
    fence_view_async_shared();  // the answer has been read before the next one may be written
    if (warp_wide) __syncwarp();
    if (!warp_wide || lane == 0) mbar_arrive(next_empty);
    return more;
  };

  if (warp >= kProducer) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kPOtherRegs));
    if (warp == kProducer) {
      // ---------------------------------------------------------------- TMA producer
      if (elect_one()) {
        int kc = 0, vc = 0, qc = 0;
        bool ok = true;
        for (int i = 0; ok; ++i) {
          const PrefillItem w = prefill_item(p, at, gridDim.y);
          if (w.n > 0) {
            ok = mbar_wait(q_empty, (qc & 1) ^ 1, abort_flag, timeout_ns);
            if (!ok) break;
            mbar_expect_tx(q_full, ((w.steps[0] > 0) + (w.steps[1] > 0)) * kQkTile);
            for (int t = 0; t < 2; ++t)
              if (w.steps_of(t) > 0)
#pragma unroll
                for (int a = 0; a < kDkAtoms; ++a)
                  tma_load_3d(sQ + t * kQkTile + a * kPAtom, &tmQ, q_full, 64 * a, w.head_of(t), w.q_start + w.m_blk_of(t) * kPM);
            ++qc;
            for (int j = 0; j < w.n; ++j) {
              const int ks = kc % kKSt, vs = vc % kVSt;
              ok = mbar_wait(k_empty + ks, ((kc / kKSt) & 1) ^ 1, abort_flag, timeout_ns);
              if (!ok) break;
              mbar_expect_tx(k_full + ks, kQkTile);
#pragma unroll
              for (int a = 0; a < kDkAtoms; ++a)
                tma_load_3d(sK + ks * kQkTile + a * kPAtom, &tmK, k_full + ks, 64 * a, w.kvh, w.k_start + j * kPN);
              ++kc;
              ok = mbar_wait(v_empty + vs, ((vc / kVSt) & 1) ^ 1, abort_flag, timeout_ns);
              if (!ok) break;
              mbar_expect_tx(v_full + vs, kPTile);
#pragma unroll
              for (int a = 0; a < 2; ++a) {
                if (p.v_packed) tma_load_3d(sV + vs * kPTile + a * kPAtom, &tmV, v_full + vs, w.k_start + j * kPN + 64 * a, w.v_col0, w.kvh);
                else tma_load_3d(sV + vs * kPTile + a * kPAtom, &tmV, v_full + vs, w.v_col0 + 64 * a, w.kvh, w.k_start + j * kPN);
              }
              ++vc;
            }
          }
          if (!ok || !advance(i, false)) break;
        }
        // after an abort nothing waits for the last copies any more: they have to land before shared memory is given back
        volatile uint32_t never = 0;
        if (*abort_flag != 0u) {
          if (qc > 0) mbar_wait(q_full, (qc - 1) & 1, &never, timeout_ns);
          for (int c = max(0, kc - kKSt); c < kc; ++c) mbar_wait(k_full + c % kKSt, (c / kKSt) & 1, &never, timeout_ns);
          for (int c = max(0, vc - kVSt); c < vc; ++c) mbar_wait(v_full + c % kVSt, (c / kVSt) & 1, &never, timeout_ns);
        }
      }
      __syncwarp();
    } else if (warp == kProducer + 1) {
      // ---------------------------------------------------------------- MMA issuer
      if (elect_one()) {
        const uint32_t idesc_s = umma_idesc_f16(kPM, kPN, BF16);
        const uint32_t idesc_o = idesc_s | (p.v_packed ? 0u : 1u << 16);  // V as it stands is an MN-major B operand
        // Descriptors differ in their low word, the address (and for V the distance between atoms). The compiler must not see that
        // the words below come from loop invariants: it would keep dozens of finished descriptors and spill.
        const uint64_t dk = umma_desc_sw128_kmajor(0), dv = p.v_packed ? dk : umma_desc_sw128_mnmajor(0, kPAtom);
        const uint32_t hi = static_cast<uint32_t>(dk >> 32), lo_k = static_cast<uint32_t>(dk), lo_v = static_cast<uint32_t>(dv);
        auto hide = [](uint32_t x) { asm volatile("" : "+r"(x)); return x; };
        auto desc = [&](uint32_t lo) { return static_cast<uint64_t>(hi) << 32 | lo; };
        int kc = 0, vc = 0, qc = 0;
        uint32_t p_phase = 0, o_phase = 0;  // bit t: parity of tile t's next phase
        bool ok = true;
        auto scores = [&](int t, int ks) {  // S_t = Q_t K^T
          const uint32_t a = hide(lo_k + (smem_u32(sQ + t * kQkTile) >> 4)), b = hide(lo_k + (smem_u32(sK + ks * kQkTile) >> 4));
#pragma unroll
          for (int kk = 0; kk < kDkAtoms * 4; ++kk) {
            const uint32_t step = ((kk >> 2) * kPAtom >> 4) + 2 * (kk & 3);
            umma_f16(tmem_base + t * kPN, desc(a + step), desc(b + step), idesc_s, kk != 0);
          }
          umma_commit(s_full + t);
        };
        for (int i = 0; ok; ++i) {
          const PrefillItem w = prefill_item(p, at, gridDim.y);
          if (w.n > 0) {
            ok = mbar_wait(q_full, qc & 1, abort_flag, timeout_ns) && mbar_wait(k_full + kc % kKSt, (kc / kKSt) & 1, abort_flag, timeout_ns);
            if (!ok) break;
            ++qc;
            tc_fence_after_sync();
            for (int t = 0; t < 2; ++t)
              if (w.steps_of(t) > 0) scores(t, kc % kKSt);
            umma_commit(k_empty + kc % kKSt);
            ++kc;
            if (w.n == 1) umma_commit(q_empty);
            for (int j = 0; j < w.n && ok; ++j) {
              const int vs = vc % kVSt;
              ok = mbar_wait(v_full + vs, (vc / kVSt) & 1, abort_flag, timeout_ns);
              for (int t = 0; t < 2 && ok; ++t) {
                const int steps = w.steps_of(t);
                if (j < steps) {  // O_t (+)= P_t V
                  if (j == 0) {
                    ok = mbar_wait(o_empty + t, (o_phase >> t & 1) ^ 1, abort_flag, timeout_ns);
                    o_phase ^= 1u << t;
                  }
                  ok = ok && mbar_wait(p_full + t, p_phase >> t & 1, abort_flag, timeout_ns);
                  p_phase ^= 1u << t;
                  if (!ok) break;
                  tc_fence_after_sync();
                  const uint32_t b = hide(lo_v + (smem_u32(sV + vs * kPTile) >> 4));
#pragma unroll
                  for (int kk = 0; kk < kPN / 16; ++kk) {
                    const uint32_t step = p.v_packed ? ((kk >> 2) * kPAtom >> 4) + 2 * (kk & 3) : kk * 16 * 128 >> 4;
                    umma_f16_ta(tmem_base + 2 * kPN + t * kPD, tmem_base + t * kPN + kk * 8, desc(b + step), idesc_o, j != 0 || kk != 0);
                  }
                  if (j == steps - 1) umma_commit(o_full + t);
                }
                if (j + 1 < steps) {
                  ok = mbar_wait(k_full + kc % kKSt, (kc / kKSt) & 1, abort_flag, timeout_ns);
                  if (!ok) break;
                  tc_fence_after_sync();
                  scores(t, kc % kKSt);
                }
              }
              if (!ok) break;
              umma_commit(v_empty + vs);
              ++vc;
              if (j + 1 < w.n) {
                umma_commit(k_empty + kc % kKSt);
                ++kc;
                if (j + 2 == w.n) umma_commit(q_empty);
              }
            }
          }
          if (!ok || !advance(i, false)) break;
        }
      }
      __syncwarp();
    } else if (warp == kProducer + 2) {
      // ---------------------------------------------------------------- next items
      if (elect_one()) {
        bool more = true;
        for (int i = 0; more; ++i) {
          if (!mbar_wait(next_empty, (i & 1) ^ 1, abort_flag, timeout_ns)) break;
          mbar_expect_tx(next_full, 16);
          clc_try_cancel(next_item, next_full);
          volatile uint32_t never = 0;  // the answer is on its way into shared memory: an abort does not end this wait
          if (!mbar_wait(next_full, i & 1, &never, timeout_ns)) {
            *abort_flag = 1u;
            break;
          }
          uint3 unused;
          more = clc_read(next_item, unused);
        }
      }
      __syncwarp();
    }
  } else if (kHelped && warp >= 8) {
    // ------------------------------------------------------------------ rescaling and output, one thread per query row of either tile
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(prefill_scale_regs(kDkAtoms)));
    const int row = (warp & 3) * 32 + lane;
    const uint32_t o_lanes = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + 2 * kPN;
    uint32_t c_phase = 0, f_phase = 0;   // bit t: parity of tile t's next phase
    bool ok = true;
    for (int i = 0; ok; ++i) {
      const PrefillItem w = prefill_item(p, at, gridDim.y);
      for (int j = 1; j < w.n && ok; ++j) {
        for (int t = 0; t < 2; ++t) {
          if (j < w.steps_of(t)) {
            ok = __all_sync(0xffffffffu, mbar_wait(c_full + t, c_phase >> t & 1, abort_flag, timeout_ns));
            c_phase ^= 1u << t;
            if (!ok) break;
            tc_fence_after_sync();
            const float corr = s_factor[t * kPM + row];
            if (__any_sync(0xffffffffu, corr != 1.f)) {
              // the scores of this step were issued after the tile's last product, so O is complete and nothing writes it now
              const uint32_t o_addr = o_lanes + t * kPD;
              uint32_t o[2][16];
              tmem_ld_32x16(o_addr, o[0]);
#pragma unroll
              for (int c = 0; c < 8; ++c) {
                tmem_ld_wait();
                if (c < 7) tmem_ld_32x16(o_addr + (c + 1) * 16, o[(c + 1) & 1]);
#pragma unroll
                for (int e = 0; e < 16; ++e) o[c & 1][e] = __float_as_uint(__uint_as_float(o[c & 1][e]) * corr);
                tmem_st_32x16(o_addr + c * 16, o[c & 1]);
              }
              tmem_st_wait();
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full + t);
          }
        }
      }
      // ---- the rows' output
      for (int t = 0; t < 2 && ok && kStaged; ++t) {
        const int steps = w.steps_of(t);
        float inv = 0.f;
        if (steps > 0) {
          ok = __all_sync(0xffffffffu, mbar_wait(f_full + t, f_phase >> t & 1, abort_flag, timeout_ns) &&
                                           mbar_wait(o_full + t, f_phase >> t & 1, abort_flag, timeout_ns));
          f_phase ^= 1u << t;
          if (!ok) break;
          tc_fence_after_sync();
          inv = s_factor[t * kPM + row];
        }
        prefill_store<kStaged, BF16>(p, w, t, steps, o_lanes + t * kPD, inv, s_out + (warp & 3) * 32 * 256, o_empty + t);
      }
      if (!ok || !advance(i, true)) break;
    }
  } else {
    // ------------------------------------------------------------------ softmax, one thread per query row
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(prefill_softmax_regs(kDkAtoms, kHelped)));
    const int t = warp >> 2;  // tile
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lanes = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const uint32_t s_addr = lanes + t * kPN, o_addr = lanes + 2 * kPN + t * kPD;
    int sc = 0, oc = 0, vc = 0;
    bool ok = true;
    for (int i = 0; ok; ++i) {
      const PrefillItem w = prefill_item(p, at, gridDim.y);
      const int steps = w.steps_of(t), head = w.head_of(t);
      const int q_pos = w.m_blk_of(t) * kPM + row;
      const int limit = p.causal ? min(q_pos + w.k_len - w.q_len + 1, w.k_len) : w.k_len;  // keys this row may attend: [0, limit)
      // the tile that zeroes what follows the last key in the last V tile, for both
      const bool cleans = !p.v_packed && w.n * kPN > w.k_len && (t == 0 ? steps == w.n : w.steps[0] < w.n);
      float ref = -INFINITY, sum = 0.f;  // the row's reference (of scaled scores) and the sum of 2^(score - reference)
      for (int j = 0; j < steps; ++j) {
        ok = __all_sync(0xffffffffu, mbar_wait(s_full + t, sc++ & 1, abort_flag, timeout_ns));
        if (!ok) break;
        tc_fence_after_sync();
        uint32_t r[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_32x32(s_addr + c * 32, r[c]);
        tmem_ld_wait();
        const int visible = limit - j * kPN;
        if (!__all_sync(0xffffffffu, visible >= kPN)) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (c * 32 + e >= visible) r[c][e] = __float_as_uint(-INFINITY);
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int e = 0; e < 32; ++e)
#pragma unroll
          for (int c = 0; c < 4; ++c) mx[c] = fmaxf(mx[c], __uint_as_float(r[c][e]));
        const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2e;
        if (j == 0) {
          ref = top;
        } else if (kHelped) {
          // (the factors of the step before have been used: this step's scores were issued behind that step's product)
          float corr = 1.f;
          if (top > ref) {
            corr = fast_exp2(ref - top);
            ref = top;
          }
          sum *= corr;
          s_factor[t * kPM + row] = corr;
          __syncwarp();
          if (lane == 0) mbar_arrive(c_full + t);
        } else if (__any_sync(0xffffffffu, top > ref)) {
          // the scores of this step were issued after the tile's last product, so O is complete and nothing writes it now
          float corr = 1.f;
          if (top > ref) {
            corr = fast_exp2(ref - top);
            ref = top;
          }
          sum *= corr;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t o[32];
            tmem_ld_32x32(o_addr + c * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * corr);
            tmem_st_32x32(o_addr + c * 32, o);
          }
          tmem_st_wait();
        }
        const float base = ref == -INFINITY ? 0.f : ref;
        const f32x2 scale2 = pack2(p.scale_log2e, p.scale_log2e), base2 = pack2(-base, -base);
        f32x2 sums[2] = {pack2(0.f, 0.f), pack2(0.f, 0.f)};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t packed[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            // 2^(s * scale - base): one fused multiply-add for two scores, one special-function instruction each
            const float2 x = unpack2(fma2(pack2(__uint_as_float(r[c][2 * e]), __uint_as_float(r[c][2 * e + 1])), scale2, base2));
            const float p0 = fast_exp2(x.x), p1 = fast_exp2(x.y);
            sums[e & 1] = add2(sums[e & 1], pack2(p0, p1));
            packed[e] = BF16 ? pack_bf16x2(p0, p1) : pack_f16x2(p0, p1);
          }
          tmem_st_32x16(s_addr + c * 16, packed);
        }
        sum += sum2(add2(sums[0], sums[1]));
        if (cleans && j == w.n - 1) {
          const int stage = (vc + j) % kVSt, valid = w.k_len - j * kPN;
          ok = __all_sync(0xffffffffu, mbar_wait(v_full + stage, ((vc + j) / kVSt) & 1, abort_flag, timeout_ns));
          if (!ok) break;
          for (int c = threadIdx.x & 127; c < (kPN - valid) * 16; c += 128) {  // 16 chunks of 16 bytes per key, 8 in each atom
            const int key = valid + (c >> 4), chunk = c & 15;
            *reinterpret_cast<uint4*>(sV + stage * kPTile + (chunk >> 3) * kPAtom + key * 128 + (chunk & 7) * 16) = make_uint4(0, 0, 0, 0);
          }
          fence_view_async_shared();
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(p_full + t);
          if (kHelped && j == 0) mbar_arrive(p_full + t);   // for the warp that rescales: nothing to do yet
        }
      }
      vc += w.n;
      if (!ok) break;
      float inv = 0.f;
      if (steps > 0) {   // the row's factor; whoever rescaled the output also stores it, if through shared memory
        if (p.sink != nullptr) sum += exp2f(p.sink[head] * 1.4426950408889634f - ref);  // the sink counts once, unscaled
        inv = sum > 0.f ? 1.f / sum : 0.f;
        if (q_pos < w.q_len && p.gate != nullptr) {
          const size_t g = static_cast<size_t>(w.q_start + q_pos) * p.ldg + head;
          const float z = BF16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p.gate)[g]) : __half2float(static_cast<const __half*>(p.gate)[g]);
          inv /= 1.f + expf(-z);
        }
        // The last step's factor may still be needed: it has been used once the item's last product is done.
        ok = __all_sync(0xffffffffu, mbar_wait(o_full + t, oc++ & 1, abort_flag, timeout_ns));
        if (!ok) break;
        if (kStaged) {
          s_factor[t * kPM + row] = inv;
          __syncwarp();
          if (lane == 0) mbar_arrive(f_full + t);
        }
      }
      if (!kStaged) {   // eight warps store faster than four
        tc_fence_after_sync();
        prefill_store<false, BF16>(p, w, t, steps, o_addr, inv, nullptr, o_empty + t);
      }
      if (!advance(i, true)) break;
    }
  }

  // ---------------------------------------------------------------------- teardown
  tc_fence_before_sync();
  __syncthreads();
  if (warp == kProducer + 3) tmem_dealloc(tmem_base, 512);
  if (threadIdx.x == 0 && *abort_flag != 0u && p.status != nullptr) atomicMax(p.status, static_cast<uint32_t>(kStatusPipeTimeout));
}

// Whether the rescaling warps pay: their hand-overs and the rows' way through shared memory add to the time of an item, which is all there is
// when the items run at once over few keys. us without them and with them (8 / 2 heads, causal, 128 columns): 16 tokens 7.8, 9.2; 300 tokens
// 12.3, 13.5; 3 x 389 14.7, 15.7; 2 x 700 19.3, 20.0; 1000 24.4, 24.2; 2000 41.6, 41.1; 8 x 16 tokens of 64 / 8 heads (256 items) 13.2, 14.5; 3 x 389
// tokens of 32 / 8 heads (192 items) 25.3, 23.8. Not causal: 100 tokens 8.8, 9.5; 300 tokens 13.6, 13.6. Rows of 64 columns, causal: 1000 tokens
// 22.4, 23.1; 1400 29.1, 29.1; 1400 of 32 / 8 heads (176 items, of which those of the first rows are short) 32.6, 33.8; not causal: 1000 tokens
// 22.6, 23.0; 1400 29.5, 29.3. Wider rows are no slower with them at any size (192 x 192, 3 x 389 tokens: 30.0, 27.6).
static bool prefill_helped(int dk_atoms, long long items, bool causal, int max_k) {
  if (!prefill_staged(dk_atoms)) return true;
  if (max_k <= kPN) return false;
  const int few = dk_atoms == 1 ? (causal ? 1536 : 1280) : (causal ? 768 : 0);
  return max_k > few || items > (dk_atoms == 1 && causal ? 3 * sm_count() / 2 : sm_count());
}

template <int kDkAtoms, bool kHelped>
static int launch_prefill_form(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const PrefillParams& p, dim3 grid, cudaStream_t s) {
  constexpr int kSmem = prefill_smem(kDkAtoms, kHelped), kThreads = prefill_threads(kHelped);
  static bool configured[64] = {false};
  int dev = 0;
  B200_CHECK_CUDA(cudaGetDevice(&dev));
  if (!configured[dev & 63]) {
    B200_CHECK_CUDA(cudaFuncSetAttribute(prefill_attn_kernel<kDkAtoms, true, kHelped>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    B200_CHECK_CUDA(cudaFuncSetAttribute(prefill_attn_kernel<kDkAtoms, false, kHelped>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    configured[dev & 63] = true;
  }
  if (p.bf16) prefill_attn_kernel<kDkAtoms, true, kHelped><<<grid, kThreads, kSmem, s>>>(tq, tk, tv, p);
  else prefill_attn_kernel<kDkAtoms, false, kHelped><<<grid, kThreads, kSmem, s>>>(tq, tk, tv, p);
  B200_CHECK_CUDA(cudaGetLastError());
  return kOk;
}

static int prefill_launch(const void* q, int64_t ldq, const void* k, const void* v, int v_packed, const int* cu_q,
                          const int* cu_k, const int* k_lens, int B, int total_q, int total_k, int max_q, int max_k, int Hq, int Hkv, int dk, int dv, float scale,
                          int causal, const float* sink, const void* gate, int ldg, void* out, int dtype, uint32_t* status, cudaStream_t s) {
  CUtensorMap tq, tk, tv;
  int rc = make_tma_3d(&tq, q, dtype, dk, Hq, total_q, dk, static_cast<uint64_t>(ldq), 64, 1, kPM, true);
  if (rc != kOk) return rc;
  rc = make_tma_3d(&tk, k, dtype, dk, Hkv, total_k, dk, static_cast<uint64_t>(Hkv) * dk, 64, 1, kPN, true);
  if (rc != kOk) return rc;
  if (v_packed) rc = make_tma_3d(&tv, v, dtype, total_k, dv, Hkv, total_k, static_cast<uint64_t>(dv) * total_k, 64, kPD, 1, true);
  else rc = make_tma_3d(&tv, v, dtype, dv, Hkv, total_k, dv, static_cast<uint64_t>(Hkv) * dv, 64, 1, kPN, true);
  if (rc != kOk) return rc;
  PrefillParams p;
  memset(&p, 0, sizeof(p));
  p.Hq = Hq; p.Hkv = Hkv; p.causal = causal; p.bf16 = dtype == kBF16;
  p.dk = dk; p.dv = dv; p.v_chunks = (dv + kPD - 1) / kPD; p.v_packed = v_packed; p.sink = sink; p.gate = gate; p.ldg = ldg;
  p.pair_heads = (Hq / Hkv) % 2 == 0;
  p.cu_q = cu_q; p.cu_k = cu_k; p.k_lens = k_lens;
  p.scale_log2e = scale * 1.4426950408889634f;
  p.out = out; p.status = status;
  const int rows = p.pair_heads ? kPM : 2 * kPM;
  const dim3 grid((p.pair_heads ? Hq / 2 : Hq) * p.v_chunks, (max_q + rows - 1) / rows, B);
  B200_REQUIRE(grid.y <= 65535 && grid.z <= 65535, "prefill attention grid is too large");
  const int atoms = (dk + 63) / 64;
  const bool helped = prefill_helped(atoms, static_cast<long long>(grid.x) * grid.y * grid.z, causal != 0, max_k);
  switch (atoms) {
    case 1: return helped ? launch_prefill_form<1, true>(tq, tk, tv, p, grid, s) : launch_prefill_form<1, false>(tq, tk, tv, p, grid, s);
    case 2: return helped ? launch_prefill_form<2, true>(tq, tk, tv, p, grid, s) : launch_prefill_form<2, false>(tq, tk, tv, p, grid, s);
    case 3: return launch_prefill_form<3, true>(tq, tk, tv, p, grid, s);
    default: return launch_prefill_form<4, true>(tq, tk, tv, p, grid, s);
  }
}

}  // namespace b200

using namespace b200;

// q [total_q, Hq, dk], k [total_k, Hkv, dk], v [total_k, Hkv, dv] (contiguous rows), cu_q / cu_k int32 [B + 1] on the device, out
// [total_q, Hq, dv]. Sequence b's keys are rows [cu_k[b], cu_k[b] + len) with len = k_lens[b], or cu_k[b + 1] - cu_k[b]
// when k_lens is null (packed sequences); with k_lens the key rows may sit anywhere in k / v, e.g. in the pages of a
// KV cache whose sequences own contiguous runs of slots. With causal != 0 query i of a sequence attends keys
// <= i + (k_len - q_len). gate: nullable [total_q, Hq] with row pitch ldg, every head's output times sigmoid(gate).
// q, k and v 16-byte aligned; dk, dv: multiples of 8, dk <= 256. dtype 0 = bf16, 1 = f16.
B200_API int b200_prefill_attention_direct(const void* q, const void* k, const void* v, const int* cu_q, const int* cu_k,
                                           const int* k_lens, int B,
                                           int total_q, int total_k, int max_q, int max_k, int Hq, int Hkv, int dk, int dv,
                                           float scale, int causal, const void* gate, int ldg, void* out, int dtype,
                                           uint32_t* status, void* stream) {
  B200_REQUIRE(dtype == kBF16 || dtype == kF16, "prefill attention supports bf16/f16");
  B200_REQUIRE(dk >= 8 && dk % 8 == 0 && dk <= 256 && dv >= 8 && dv % 8 == 0,
               "prefill attention needs head sizes in multiples of 8, keys up to 256; got %d and %d", dk, dv);
  B200_REQUIRE(Hkv > 0 && Hq % Hkv == 0, "Hq (%d) must be a multiple of Hkv (%d)", Hq, Hkv);
  B200_REQUIRE(B >= 1 && max_q >= 1 && max_k >= 1 && total_q >= 1 && total_k >= 1, "empty problem");
  B200_REQUIRE(scale > 0.f, "the score scale must be positive");
  return prefill_launch(q, static_cast<int64_t>(Hq) * dk, k, v, 0, cu_q, cu_k, k_lens, B, total_q, total_k, max_q, max_k, Hq, Hkv, dk, dv, scale,
                        causal, nullptr, gate, ldg, out, dtype, status, static_cast<cudaStream_t>(stream));
}

// The form of callers that bring a scratch for transposed values: b200_prefill_attention_scratch_bytes(...) bytes, which nothing is
// written to any more. Values that do not start on a 16-byte boundary are copied to one that does, in stream order.
B200_API long long b200_prefill_attention_scratch_bytes(int B, int Hkv, int dv, int max_k) {
  const long long s_pad = (static_cast<long long>(max_k) + 127) / 128 * 128;
  return static_cast<long long>(B) * Hkv * dv * s_pad * 2;
}
B200_API int b200_prefill_attention(const void* q, const void* k, const void* v, const int* cu_q, const int* cu_k,
                                    const int* k_lens, int B,
                                    int total_q, int total_k, int max_q, int max_k, int Hq, int Hkv, int dk, int dv,
                                    float scale, int causal, const void* gate, int ldg, void* vt_scratch, void* out, int dtype,
                                    uint32_t* status, void* stream) {
  B200_REQUIRE(vt_scratch != nullptr, "the transposed-V scratch is required");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  void* copy = nullptr;
  if (reinterpret_cast<uintptr_t>(v) % 16 != 0 && total_k > 0 && Hkv > 0 && dv > 0) {
    const size_t bytes = static_cast<size_t>(total_k) * Hkv * dv * 2;
    B200_CHECK_CUDA(cudaMallocAsync(&copy, bytes, s));
    const cudaError_t e = cudaMemcpyAsync(copy, v, bytes, cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) cudaFreeAsync(copy, s);
    B200_CHECK_CUDA(e);
  }
  const int rc = b200_prefill_attention_direct(q, k, copy != nullptr ? copy : v, cu_q, cu_k, k_lens, B, total_q, total_k, max_q, max_k, Hq, Hkv, dk,
                                               dv, scale, causal, gate, ldg, out, dtype, status, stream);
  if (copy != nullptr) B200_CHECK_CUDA(cudaFreeAsync(copy, s));
  return rc;
}

// As b200_prefill_attention_direct for values that are already transposed:
//   q [total_q, Hq, dk] with ldq elements between two tokens; k [total_k, Hkv, dk] contiguous; vt [Hkv, dv, total_k], the keys of
//   a sequence at columns cu_k[b] ... (multiples of 8). Whole tiles of 128 keys are read: what follows a sequence must be finite;
//   sink: nullable fp32 [Hq] on the device, a logit that joins every row's softmax denominator unscaled and has no value;
//   out [total_q, Hq, dv]. dk, dv, ldq and total_k are multiples of 8, dk <= 256.
B200_API int b200_prefill_attention_vt(const void* q, long long ldq, const void* k, const void* vt, const int* cu_q,
                                       const int* cu_k, const int* k_lens, int B, int total_q, int total_k, int max_q, int Hq,
                                       int Hkv, int dk, int dv, float scale, int causal, const float* sink, void* out, int dtype,
                                       uint32_t* status, void* stream) {
  B200_REQUIRE(dtype == kBF16 || dtype == kF16, "prefill attention supports bf16/f16");
  B200_REQUIRE(Hkv > 0 && Hq % Hkv == 0, "Hq (%d) must be a multiple of Hkv (%d)", Hq, Hkv);
  B200_REQUIRE(B >= 1 && max_q >= 1 && total_q >= 1 && total_k >= 1, "empty problem");
  B200_REQUIRE(dk >= 8 && dk % 8 == 0 && dk <= 256 && dv >= 8 && dv % 8 == 0 && ldq % 8 == 0 && total_k % 8 == 0,
               "prefill attention needs dk (%d) <= 256, and dk, dv (%d), ldq, total_k (%d) in multiples of 8", dk, dv, total_k);
  B200_REQUIRE(scale > 0.f, "the score scale must be positive");
  return prefill_launch(q, ldq, k, vt, 1, cu_q, cu_k, k_lens, B, total_q, total_k, max_q, total_k, Hq, Hkv, dk, dv, scale, causal, sink,
                        nullptr, 0, out, dtype, status, static_cast<cudaStream_t>(stream));
}
