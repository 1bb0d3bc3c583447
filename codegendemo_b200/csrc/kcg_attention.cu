// Fused attention forward, O = softmax(scale * Q K^T) V per head, for fp16 / bf16 with head dimension 64 or 128:
// the attention-shaped chain (two products around a row softmax, which the reference lists after batched GEMM
// among its next operators, doc/结果汇总.md) as ONE kernel in which scores and probabilities never leave the SM.
// The three-launch form (matmul_op.attention: batched Q K^T with fp32 scores, row softmax, batched P V) stays as
// the path whose parity is pinned to the composition; this kernel is checked against the same composition.
//
// Default form (AttnFwd2): one CTA per (head, 256 query rows) = two query tiles of 128 rows, 384 threads:
//   warp 0    TMA producer: both Q tiles once, then K and V tiles of 128 keys through two-stage rings, shared by
//             the two query tiles
//   warp 2    waits for K and V tiles in the issuer's place
//   warp 1    tcgen05.mma issuer and TMEM owner; per tile t: S_t = Q_t K_j^T (both K-major) into the tile's S
//             buffer, O_t += P_t V_j with P_t read from tensor memory and V as the MN-major operand
//   warps 4-7 softmax of tile 0, warps 8-11 of tile 1, one query row per thread: read S_t from TMEM, exponentials in
//             the exp2 domain against the running maximum, P_t as packed 16-bit pairs over the S columns just read, O_t
//             rescaled where that maximum has moved; at the end O / sum to global memory
// A tile's chain is serial (scores, softmax, P V, next scores) and the two tiles' chains take turns, so the tensor
// pipe works for one tile while the other is in its softmax. What bounds it is that chain, and the power cap: per step and tile
// 512 + 512 cycles of products (the scores' operands fill the shared-memory port, 128 bytes a cycle) and 1024 of
// exponentials; both tiles' steps take 2970 cycles against 2048 of the tensor pipe alone, of a tile's 100 to read the
// scores, 300 for the maximum, 1170 for 96 exponentials with the rescaling, 400 for the last 32, 640 of products and 260 of
// hand-offs. The issuer's waits are named barriers: with mbarriers a step took 3450, 32 heads x 4096 x 4096 x 128 239 us ->
// 223 (1230 TFLOP/s), 16 x 2048 x 2048 x 128 37.5 -> 34.0, 100 x 700 x 3000 x 128 127 -> 113, 8 x 300 x 16384 x 128 57.6 ->
// 53.9, 32 x 4096 x 4096 x 64 196 -> 191 (B200, bf16, graph replay in turn).
// Tried without gain since: two threads a row (241 -> 276 us: the maximum through shared memory, both tiles' exponentials at
// once), steps of 64 keys with two score buffers a tile (311: the rescaling waits for the product before), the first half of the
// next scores under the exponentials (289: products of 64 keys read Q twice as often).
// A key-split form of it (kKeySplit) shares a group's keys among the CTAs of a cluster where groups do not fill a wave.
// Tried without gain: exponentials of every eighth to third pair as a polynomial on the FMA pipe (2 to 8 % slower: one
// warp per scheduler and tile is bound by its own latencies, not by the exponential pipe).
// Four single-tile forms are kept for comparison
// (AttnFwd: one query tile per CTA with two S buffers, 64- or 128-key steps, one or two threads per row, P through
// shared or tensor memory; S issued one step ahead - two steps ahead, with a third buffer, measured slower).
// Few query rows per head (up to 64): a form of its own (kernels/attn_decode.cuh).
// Every wait is bounded (ptx_sm100.cuh); a wait that runs out records a code in a status word the host can read
// (kcg_attention_status), raises the CTA's abort flag and all roles fall through to the exit.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <mutex>
#include <string>

#include "../../include/kcg_b200.h"
#include "kernels/ptx_sm100.cuh"

extern "C" int kcg_internal_fail(int code, const char* msg);
extern "C" void kcg_internal_count_launch(void);

namespace {

using namespace kcg;

__device__ unsigned int g_attn_status[4];  // {code, block, detail, detail}; 0 = no wait ran out

// 3-D tiled load: {column, row, head}
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* tm, uint64_t* bar, int32_t c0,
                                            int32_t c1, int32_t c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

// The tile of a later load into L2 (allowed before griddep_wait(): see tma_prefetch_2d).
__device__ __forceinline__ void tma_prefetch_3d(const CUtensorMap* tm, int32_t c0, int32_t c1, int32_t c2) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global [%0, {%1, %2, %3}];"
               :
               : "l"(reinterpret_cast<uint64_t>(tm)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}

// Ties the registers of an earlier tmem_ld to the wait before it: no use of them may be scheduled ahead of this.
__device__ __forceinline__ void pin_32(uint32_t (&r)[32]) {
#pragma unroll
  for (int i = 0; i < 32; ++i) asm volatile("" : "+r"(r[i]));
}
// Two fp32 operations per instruction on register pairs (one rounding each, like the scalar forms).
__device__ __forceinline__ uint64_t f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 f32x2_split(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <bool kBf16>
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi) {
  if constexpr (kBf16) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  } else {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
}

struct AttnParams {
  CUtensorMap tmQ, tmK, tmV;  // {d, rows, heads}, boxes of {64, 128, 1}, 128-byte swizzle
  void* O;                    // heads x sq x d, contiguous
  int sq, sk;
  float scale_log2;           // scale * log2(e): the softmax runs on exp2
  int first_group;            // AttnFwd2: group of 256 rows of the first CTA (cluster)
  int splits;                 // AttnFwd2, key-split form: CTAs that share a group's keys
  int tail_follows;           // AttnFwd2: the groups after this launch's are run by a key-split launch right behind it
};

enum : uint32_t { ATTN_TIMEOUT_PRODUCER = 1, ATTN_TIMEOUT_MMA = 2, ATTN_TIMEOUT_SOFTMAX = 3 };

#include "kernels/attn_decode.cuh"

// kBC = keys per step (64 or 128); kSplit = threads per query row (1 or 2). With 64 keys per step and one
// thread per row a CTA needs 96 KB of shared memory (d = 128), 256 TMEM columns and 192 threads, so TWO CTAs
// share an SM and one's products fill the tensor pipe while the other is in its softmax.
// kPTmem = 1 keeps P in tensor memory: the softmax threads write it (packed pairs) over the columns of the S buffer
// they have just read, and P V takes its A operand from there, so P never crosses the shared-memory port (which
// carries every operand byte of both products and is what bounds this kernel).
template <int kD, bool kBf16, int kBC, int kSplit, int kPTmem>
struct AttnFwd {
  static constexpr int BR = 128;  // query rows per CTA (= TMEM lanes)
  static constexpr int BC = kBC;  // keys per step
  static constexpr int K_STAGES = 2;
  static constexpr int V_STAGES = (kBC == 64) ? 1 : 2;  // V_j is needed a whole softmax later than K_j
  static constexpr int NUM_SOFTMAX_THREADS = 128 * kSplit;
  static constexpr int NUM_THREADS = 64 + NUM_SOFTMAX_THREADS;  // producer, MMA issuer, softmax warps
  static constexpr int BOXES = kD / 64;             // 64 values = 128 bytes per box row
  static constexpr int QBOX_BYTES = BR * 128;       // Q: boxes of 128 rows x 128 bytes
  static constexpr int KVBOX_BYTES = BC * 128;      // K, V: boxes of BC rows x 128 bytes
  static constexpr int Q_BYTES = BR * kD * 2, KV_BYTES = BC * kD * 2, P_BYTES = kPTmem ? 0 : BR * BC * 2;
  static constexpr int OFF_K = Q_BYTES, OFF_V = OFF_K + K_STAGES * KV_BYTES, OFF_P = OFF_V + V_STAGES * KV_BYTES;
  static constexpr int RING_BYTES = OFF_P + P_BYTES;
  static constexpr int SMEM_BYTES = RING_BYTES + 3072;  // 1 KB alignment slack + 2 KB barriers and exchange slots
  static constexpr uint32_t COL_O = 2 * BC;             // S0 [0, BC), S1 [BC, 2 BC), O [2 BC, 2 BC + kD)
  static constexpr uint32_t TMEM_COLS = (2 * BC + kD <= 256) ? 256 : 512;
  static constexpr uint32_t FMT = kBf16 ? FMT_BF16 : FMT_F16;
  // S = Q K^T: both operands K-major (rows x d); O += P V: P K-major (rows x keys), V MN-major (keys x d)
  static constexpr uint32_t IDESC_S = make_instr_desc(FMT, 0u, 0u, 128u, BC);
  static constexpr uint32_t IDESC_O = make_instr_desc(FMT, 0u, 1u, 128u, kD);
  static_assert((kBC == 64 || kBC == 128) && (kSplit == 1 || kSplit == 2) && (kBC / kSplit) % 32 == 0, "shape");
  using T = typename std::conditional<kBf16, __nv_bfloat16, __half>::type;

  struct Barriers {
    uint64_t q_full;
    uint64_t k_full[K_STAGES], k_empty[K_STAGES], v_full[V_STAGES], v_empty[V_STAGES];
    uint64_t s_full[2], s_empty[2];
    uint64_t p_full;    // P_j is in shared memory and O is rescaled (every softmax warp arrives)
    uint64_t pv_done;   // P_j V_j has retired: P may be overwritten, O may be read
    uint32_t tmem_base;
    volatile uint32_t abort_flag;
    float exchange[2][128];  // row maxima (and, at the end, row sums) passed between the two threads of a row
  };
  static_assert(sizeof(Barriers) <= 2048, "barrier block exceeds its shared-memory slot");

  __device__ static __forceinline__ void report(Barriers* bars, uint32_t code, uint32_t d0, uint32_t d1) {
    bars->abort_flag = 1u;
    if (atomicCAS(&g_attn_status[0], 0u, code) == 0u) {
      g_attn_status[1] = blockIdx.x;
      g_attn_status[2] = d0;
      g_attn_status[3] = d1;
    }
  }

  __device__ static void run(const AttnParams& p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    Barriers* bars = reinterpret_cast<Barriers*>(smem + RING_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q_tiles = (p.sq + BR - 1) / BR;
    const int head = static_cast<int>(blockIdx.x) / q_tiles;
    const int q0 = (static_cast<int>(blockIdx.x) % q_tiles) * BR;
    const int nkv = (p.sk + BC - 1) / BC;

    if (threadIdx.x == 0) {
      tma_prefetch_desc(&p.tmQ);
      tma_prefetch_desc(&p.tmK);
      tma_prefetch_desc(&p.tmV);
      mbar_init(&bars->q_full, 1);
      for (int s = 0; s < K_STAGES; ++s) {
        mbar_init(&bars->k_full[s], 1);
        mbar_init(&bars->k_empty[s], 1);
      }
      for (int s = 0; s < V_STAGES; ++s) {
        mbar_init(&bars->v_full[s], 1);
        mbar_init(&bars->v_empty[s], 1);
      }
      for (int b = 0; b < 2; ++b) {
        mbar_init(&bars->s_full[b], 1);
        mbar_init(&bars->s_empty[b], 4 * kSplit);  // one arrival per softmax warp
      }
      mbar_init(&bars->p_full, 4 * kSplit);
      mbar_init(&bars->pv_done, 1);
      bars->abort_flag = 0u;
      fence_mbar_init();
      fence_proxy_async_smem();
    }
    if (warp == 1) {
      tmem_alloc(&bars->tmem_base, TMEM_COLS);
      tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = bars->tmem_base;

    if (warp == 0) {
      // ------------------------------------------------------------------ producer
      if (lane == 0) {
        mbar_expect_tx(&bars->q_full, Q_BYTES);
#pragma unroll
        for (int b = 0; b < BOXES; ++b) tma_load_3d(smem + b * QBOX_BYTES, &p.tmQ, &bars->q_full, b * 64, q0, head);
        for (int j = 0; j < nkv; ++j) {
          const int ks = j % K_STAGES, vs = j % V_STAGES;
          if (!mbar_wait(&bars->k_empty[ks], ((j / K_STAGES) & 1u) ^ 1u, &bars->abort_flag)) {
            report(bars, ATTN_TIMEOUT_PRODUCER, j, 0u);
            break;
          }
          mbar_expect_tx(&bars->k_full[ks], KV_BYTES);
#pragma unroll
          for (int b = 0; b < BOXES; ++b)
            tma_load_3d(smem + OFF_K + ks * KV_BYTES + b * KVBOX_BYTES, &p.tmK, &bars->k_full[ks], b * 64, j * BC, head);
          if (!mbar_wait(&bars->v_empty[vs], ((j / V_STAGES) & 1u) ^ 1u, &bars->abort_flag)) {
            report(bars, ATTN_TIMEOUT_PRODUCER, j, 1u);
            break;
          }
          mbar_expect_tx(&bars->v_full[vs], KV_BYTES);
#pragma unroll
          for (int b = 0; b < BOXES; ++b)
            tma_load_3d(smem + OFF_V + vs * KV_BYTES + b * KVBOX_BYTES, &p.tmV, &bars->v_full[vs], b * 64, j * BC, head);
        }
      }
    } else if (warp == 1) {
      // ---------------------------------------------------------------- MMA issuer
      if (lane == 0) {
        bool ok = mbar_wait(&bars->q_full, 0u, &bars->abort_flag);
        if (!ok) report(bars, ATTN_TIMEOUT_MMA, 0u, 0u);
        tc_fence_after_sync();
        const uint32_t sq_addr = smem_u32(smem);
        // S_i = Q K_i^T into S buffer i % 2
        auto issue_s = [&](int i) -> bool {
          const int s = i % K_STAGES, b = i & 1;
          if (!mbar_wait(&bars->k_full[s], (i / K_STAGES) & 1u, &bars->abort_flag) ||
              !mbar_wait(&bars->s_empty[b], ((i >> 1) & 1u) ^ 1u, &bars->abort_flag)) {
            report(bars, ATTN_TIMEOUT_MMA, 1u, static_cast<uint32_t>(i));
            return false;
          }
          tc_fence_after_sync();
          const uint32_t sk_addr = smem_u32(smem + OFF_K + s * KV_BYTES);
#pragma unroll
          for (int ks = 0; ks < kD / 16; ++ks) {
            // 16 values of d = 32 bytes of a 128-byte box row; the boxes of 64 values follow one another
            const uint32_t in_row = (ks * 32) % 128, box = (ks * 32) / 128;
            const uint64_t adesc = make_smem_desc(sq_addr + box * QBOX_BYTES + in_row, 16, 1024, SWZ_128B);
            const uint64_t bdesc = make_smem_desc(sk_addr + box * KVBOX_BYTES + in_row, 16, 1024, SWZ_128B);
            umma_ss<false>(tmem_base + b * BC, adesc, bdesc, IDESC_S, ks > 0 ? 1u : 0u);
          }
          umma_commit(&bars->k_empty[s]);
          umma_commit(&bars->s_full[b]);
          return true;
        };
        if (ok) ok = issue_s(0);
        for (int j = 0; j < nkv && ok; ++j) {
          if (j + 1 < nkv) ok = issue_s(j + 1);
          if (!ok) break;
          const int s = j % V_STAGES;
          if (!mbar_wait(&bars->p_full, j & 1u, &bars->abort_flag) ||
              !mbar_wait(&bars->v_full[s], (j / V_STAGES) & 1u, &bars->abort_flag)) {
            report(bars, ATTN_TIMEOUT_MMA, 2u, static_cast<uint32_t>(j));
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t sp_addr = smem_u32(smem + OFF_P);
          const uint32_t sv_addr = smem_u32(smem + OFF_V + s * KV_BYTES);
#pragma unroll
          for (int ks = 0; ks < BC / 16; ++ks) {
            // P: K-major, 128 rows x BC keys in boxes of 64 keys; V: BC keys x d, its 64-value column chunks
            // are boxes of BC key rows (leading-dimension offset = one box), a K step = 16 key rows
            const uint64_t bdesc = make_smem_desc(sv_addr + ks * 16 * 128, KVBOX_BYTES, 1024, SWZ_128B);
            if constexpr (kPTmem) {
              // 16 keys = 8 columns of packed pairs in the S buffer of this step
              umma_ts<false>(tmem_base + COL_O, tmem_base + (j & 1) * BC + ks * 8, bdesc, IDESC_O,
                          (j > 0 || ks > 0) ? 1u : 0u);
            } else {
              const uint32_t a_off = ((ks * 32) / 128) * (BR * 128) + ((ks * 32) % 128);  // boxes of 64 keys
              const uint64_t adesc = make_smem_desc(sp_addr + a_off, 16, 1024, SWZ_128B);
              umma_ss<false>(tmem_base + COL_O, adesc, bdesc, IDESC_O, (j > 0 || ks > 0) ? 1u : 0u);
            }
          }
          umma_commit(&bars->v_empty[s]);
          umma_commit(&bars->pv_done);
        }
      }
    } else {
      // ------------------------------------------------- softmax, correction, epilogue
      // kSplit threads per query row. With two, warps 2-5 take the first half of a step's keys and of O's
      // columns, warps 6-9 the second; the two warps that share a TMEM lane quarter meet on a named barrier
      // of their own to combine their row maxima (the sums stay separate until the end).
      const int q = warp & 3;                // TMEM lane quarter this warp may access
      const int h = (warp - 2) >> 2;         // which part of the keys / of O's columns (0 when kSplit = 1)
      const int row = q * 32 + lane;         // query row of this thread inside the tile
      const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
      constexpr int HC = BC / kSplit;        // keys per thread and step
      constexpr int OC = kD / kSplit;        // O columns per thread
      float m = -INFINITY, l = 0.f;
      bool ok = true;
      for (int j = 0; j < nkv; ++j) {
        const int b = j & 1;
        bool got = mbar_wait(&bars->s_full[b], (j >> 1) & 1u, &bars->abort_flag);
        if (!named_bar_all(2, NUM_SOFTMAX_THREADS, got)) {
          if (!got) report(bars, ATTN_TIMEOUT_SOFTMAX, 0u, static_cast<uint32_t>(j));
          ok = false;
          break;
        }
        tc_fence_after_sync();
        float s[HC];
#pragma unroll
        for (int c = 0; c < HC / 32; ++c) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(tmem_base + lane_addr + b * BC + h * HC + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) s[c * 32 + i] = __uint_as_float(r[i]);
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->s_empty[b]);  // the MMA warp may overwrite this S buffer
        const int valid = p.sk - j * BC - h * HC;       // keys of this thread's half that exist
        if (valid < HC) {
#pragma unroll
          for (int i = 0; i < HC; ++i)
            if (i >= valid) s[i] = -INFINITY;
        }
        // running maximum of the raw scores (the scale is positive: checked by the host), four chains
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < HC; i += 4) {
          mx4[0] = fmaxf(mx4[0], s[i]);
          mx4[1] = fmaxf(mx4[1], s[i + 1]);
          mx4[2] = fmaxf(mx4[2], s[i + 2]);
          mx4[3] = fmaxf(mx4[3], s[i + 3]);
        }
        float rowmax = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
        if constexpr (kSplit == 2) {
          bars->exchange[h][row] = rowmax;
          named_bar_sync(3 + q, 64);  // the two warps of this lane quarter
          rowmax = fmaxf(rowmax, bars->exchange[h ^ 1][row]);
          // (the slot is written again a step later, behind the vote of all softmax warps below: the partner
          // has read it by then)
        }
        const float mx = fmaxf(m, rowmax * p.scale_log2);
        const float alpha = ex2(m - mx);  // 0 on the first step (m = -inf)
        float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < HC; i += 4) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s[i + e] = ex2(fmaf(s[i + e], p.scale_log2, -mx));
            sum4[e] += s[i + e];
          }
        }
        l = l * alpha + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
        m = mx;
        // Does any row of this warp have a new maximum? Only then is O rescaled (alpha = 1 otherwise).
        const bool rescale = j > 0 && __any_sync(0xffffffffu, alpha != 1.f);
        if constexpr (kPTmem) {
          // P_j goes over the S columns this thread has read: no other step uses them, so it need not wait
          // for the previous product. Two keys per 32-bit column.
          static_assert(HC == 64, "one 32-column store per thread and step");
          uint32_t w[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            if constexpr (kBf16) {
              __nv_bfloat162 v2 = __floats2bfloat162_rn(s[2 * i], s[2 * i + 1]);
              w[i] = *reinterpret_cast<uint32_t*>(&v2);
            } else {
              __half2 v2 = __floats2half2_rn(s[2 * i], s[2 * i + 1]);
              w[i] = *reinterpret_cast<uint32_t*>(&v2);
            }
          }
          tmem_st_32x32b_x32(tmem_base + lane_addr + b * BC + h * (HC / 2), w);
        }
        // P_{j-1} V_{j-1} must have retired before O is touched - and, when P goes through shared memory, before
        // its one buffer is overwritten. (S_j is complete, so every product before P_{j-1} V_{j-1} has retired:
        // the barrier is at most one phase behind and the parity test is unambiguous even after skipped waits.)
        got = (kPTmem && !rescale) ? true : mbar_wait(&bars->pv_done, (j & 1u) ^ 1u, &bars->abort_flag);
        if (!named_bar_all(2, NUM_SOFTMAX_THREADS, got)) {
          if (!got) report(bars, ATTN_TIMEOUT_SOFTMAX, 1u, static_cast<uint32_t>(j));
          ok = false;
          break;
        }
        tc_fence_after_sync();
        if constexpr (!kPTmem) {
          // this thread's keys of its row of P: boxes of 64 keys, 16-byte units XOR-swizzled by the row
          constexpr int PBOX_BYTES = BR * 128;
          uint8_t* prow = smem + OFF_P + row * 128;
#pragma unroll
          for (int u = 0; u < HC / 8; ++u) {
            const int unit = (h * HC) / 8 + u;  // 16-byte unit inside the row of BC keys
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              if constexpr (kBf16) {
                __nv_bfloat162 v2 = __floats2bfloat162_rn(s[u * 8 + 2 * e], s[u * 8 + 2 * e + 1]);
                w[e] = *reinterpret_cast<uint32_t*>(&v2);
              } else {
                __half2 v2 = __floats2half2_rn(s[u * 8 + 2 * e], s[u * 8 + 2 * e + 1]);
                w[e] = *reinterpret_cast<uint32_t*>(&v2);
              }
            }
            *reinterpret_cast<uint4*>(prow + (unit / 8) * PBOX_BYTES + (((unit % 8) ^ (row & 7)) << 4)) =
                make_uint4(w[0], w[1], w[2], w[3]);
          }
          fence_proxy_async_smem();  // P visible to the tensor core's operand reads
        }
        if (rescale) {
          // O <- alpha * O for this thread's columns
#pragma unroll
          for (int c = 0; c < OC / 32; ++c) {
            uint32_t r[32];
            tmem_ld_32x32b_x32(tmem_base + lane_addr + COL_O + h * OC + c * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
            tmem_st_32x32b_x32(tmem_base + lane_addr + COL_O + h * OC + c * 32, r);
          }
        }
        tmem_st_wait();  // P (when it lives in tensor memory) and the rescaled O are written
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->p_full);
      }
      if (ok) {
        bool got = mbar_wait(&bars->pv_done, (nkv - 1) & 1u, &bars->abort_flag);
        if (!named_bar_all(2, NUM_SOFTMAX_THREADS, got)) {
          if (!got) report(bars, ATTN_TIMEOUT_SOFTMAX, 2u, 0u);
          ok = false;
        }
      }
      if (ok) {
        tc_fence_after_sync();
        if constexpr (kSplit == 2) {
          bars->exchange[h][row] = l;  // the row's sum = the two halves' sums (both relative to the same maximum)
          named_bar_sync(3 + q, 64);
          l += bars->exchange[h ^ 1][row];
        }
        const float inv = 1.f / l;
        const int grow = q0 + row;
        T* out = reinterpret_cast<T*>(p.O) + (static_cast<size_t>(head) * p.sq + grow) * kD + h * OC;
#pragma unroll
        for (int c = 0; c < OC / 32; ++c) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(tmem_base + lane_addr + COL_O + h * OC + c * 32, r);
          tmem_ld_wait();
          if (grow < p.sq) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              uint32_t w[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float a = __uint_as_float(r[u * 8 + 2 * e]) * inv, bb = __uint_as_float(r[u * 8 + 2 * e + 1]) * inv;
                if constexpr (kBf16) {
                  __nv_bfloat162 v2 = __floats2bfloat162_rn(a, bb);
                  w[e] = *reinterpret_cast<uint32_t*>(&v2);
                } else {
                  __half2 v2 = __floats2half2_rn(a, bb);
                  w[e] = *reinterpret_cast<uint32_t*>(&v2);
                }
              }
              *reinterpret_cast<uint4*>(out + c * 32 + u * 8) = make_uint4(w[0], w[1], w[2], w[3]);
            }
          }
        }
      }
    }

    // ---------------------------------------------------------------- common exit
    __syncwarp();
    if (bars->abort_flag != 0u) {
      // give loads / MMAs still in flight time to land before shared memory and TMEM are released
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
      tc_fence_after_sync();
      tmem_dealloc(tmem_base, TMEM_COLS);
    }
  }
};

// Two query tiles per CTA. Tile 0 (rows q0 .. q0 + 127) and tile 1 (the next 128 rows) share the K and V tiles in
// shared memory and take turns on the tensor pipe: while the softmax warps of one tile work on its scores, the
// products of the other run. Each tile owns one S buffer (P is written over it) and one O accumulator in tensor
// memory - S_t [128 t, 128 t + 128), O_t [256 + kD t, ...) - and four softmax warps, one thread per row and 128 keys
// per thread and step. A tile's chain is serial (S, softmax, P V, next S: the next scores overwrite P, and the
// tensor pipe runs its instructions in order), the two chains interleave. The MMA warp serves the tiles in a fixed
// order (serving whichever P is ready first measured no faster).
template <int kD, bool kBf16, bool kKeySplit>
struct AttnFwd2 {
  static constexpr int BR = 128, BC = 128, TILES = 2;
  static constexpr int K_STAGES = 2, V_STAGES = 2;
  static constexpr int NUM_THREADS = 128 + TILES * 128;  // whole warpgroups, for setmaxnreg
  static constexpr int BOXES = kD / 64;
  static constexpr int QBOX_BYTES = BR * 128, KVBOX_BYTES = BC * 128;
  static constexpr int Q_BYTES = BR * kD * 2, KV_BYTES = BC * kD * 2;
  static constexpr int OFF_K = TILES * Q_BYTES, OFF_V = OFF_K + K_STAGES * KV_BYTES;
  static constexpr int RING_BYTES = OFF_V + V_STAGES * KV_BYTES;
  static constexpr int SMEM_BYTES = RING_BYTES + 2048;  // 1 KB alignment slack + barriers
  // Keys of a step after which P V starts, and whether tile 1 starts half a step after tile 0 (the walk keeps the distance:
  // one tile's exponentials then run while the other waits for its products, not beside the other's). Measured, 32 heads x
  // 4096 x 4096: d = 128 after 64, 96, 112, 128 keys 236, 223, 230, 233 us, with the distance 230, 225 (its products alone keep
  // the tiles apart); d = 64 after 64, 96, 128 keys 198, 205, 208 us, with the distance 191, 203.
  static constexpr int P_PART = kD == 128 ? 96 : 64;
  static constexpr bool kApart = kD == 64;
  static constexpr uint32_t COL_O = TILES * BC, TMEM_COLS = 512;
  static constexpr uint32_t FMT = kBf16 ? FMT_BF16 : FMT_F16;
  static constexpr uint32_t IDESC_S = make_instr_desc(FMT, 0u, 0u, 128u, BC);
  static constexpr uint32_t IDESC_O = make_instr_desc(FMT, 0u, 1u, 128u, kD);
  using T = typename std::conditional<kBf16, __nv_bfloat16, __half>::type;

  struct Barriers {
    uint64_t q_full;
    uint64_t k_full[K_STAGES], k_empty[K_STAGES], v_full[V_STAGES], v_empty[V_STAGES];
    uint64_t s_full[TILES];   // S_t of the current step is complete
    uint64_t o_full[TILES];   // the last P_t V has retired
    uint32_t tmem_base;
    volatile uint32_t abort_flag;
  };

  // Named barriers, on which the issuer meets what its products wait for. They are not in shared memory: a look at an
  // mbarrier there takes 200 to 300 cycles while the products' operand reads fill the port, and an issuer that looked six
  // times a step (P_t twice, K and V) was on the critical path with 900 of 3450 cycles.
  // Every meeting takes place in every step whatever else happened: the issuer and warp 2 go on after a wait that ran out, and
  // so do the softmax warps, whose scores then come from whatever the operands hold. These wait for their scores without
  // looking at the abort flag, and four times as long as anybody else waits: should the scores never come, every other wait of
  // the CTA has ended long before, so the issuer has left the step before, and the warp only comes to the meetings that
  // are left (it must not come twice to one that the issuer has not come to).
  static constexpr uint32_t BAR_PART = 1;  // + t: the first P_PART keys of P_t are in tensor memory and O_t is rescaled
  static constexpr uint32_t BAR_FULL = 3;  // + t: all of P_t is (both: four softmax warps arrive, the issuer waits)
  static constexpr uint32_t BAR_KV = 5;    // the V tile of a step and the K tile of the next have landed (warp 2 and the issuer)
  static constexpr uint32_t PT_THREADS = 160, KV_THREADS = 64;

  __device__ static __forceinline__ void report(Barriers* bars, uint32_t code, uint32_t d0, uint32_t d1) {
    bars->abort_flag = 1u;
    if (atomicCAS(&g_attn_status[0], 0u, code) == 0u) {
      g_attn_status[1] = blockIdx.x;
      g_attn_status[2] = d0;
      g_attn_status[3] = d1;
    }
  }

  __device__ static void run(const AttnParams& p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    Barriers* bars = reinterpret_cast<Barriers*>(smem + RING_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q_groups = (p.sq + TILES * BR - 1) / (TILES * BR);
    const int rank = kKeySplit ? static_cast<int>(cluster_cta_rank()) : 0;
    const int group = p.first_group + static_cast<int>(blockIdx.x) / (kKeySplit ? p.splits : 1);
    const int head = group / q_groups;
    const int q0 = (group % q_groups) * (TILES * BR);
    // steps of this CTA: [key0 / BC, key0 / BC + nkv); splits <= steps, so every CTA has at least one
    const int steps = (p.sk + BC - 1) / BC;
    const int step0 = kKeySplit ? static_cast<int>(static_cast<long long>(steps) * rank / p.splits) : 0;
    const int nkv =
        (kKeySplit ? static_cast<int>(static_cast<long long>(steps) * (rank + 1) / p.splits) : steps) - step0;
    const int key0 = step0 * BC;
    if (!kKeySplit && p.tail_follows) griddep_launch_dependents();

    if (threadIdx.x == 0) {
      tma_prefetch_desc(&p.tmQ);
      tma_prefetch_desc(&p.tmK);
      tma_prefetch_desc(&p.tmV);
      mbar_init(&bars->q_full, 1);
      for (int s = 0; s < K_STAGES; ++s) {
        mbar_init(&bars->k_full[s], 1);
        mbar_init(&bars->k_empty[s], 1);
      }
      for (int s = 0; s < V_STAGES; ++s) {
        mbar_init(&bars->v_full[s], 1);
        mbar_init(&bars->v_empty[s], 1);
      }
      for (int t = 0; t < TILES; ++t) {
        mbar_init(&bars->s_full[t], 1);
        mbar_init(&bars->o_full[t], 1);
      }
      bars->abort_flag = 0u;
      fence_mbar_init();
      fence_proxy_async_smem();
    }
    if (warp == 1) {
      tmem_alloc(&bars->tmem_base, TMEM_COLS);
      tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = bars->tmem_base;

    // Registers: 384 threads are launched with 168 each; the control warpgroup keeps 56, the softmax warpgroups take
    // 224 (56 + 2 * 224 = 3 * 168), which a row's 128 scores need.
    if (warp < 4) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
      if (warp == 0) {
        // ------------------------------------------------------------------ producer
        if (lane == 0) {
          mbar_expect_tx(&bars->q_full, TILES * Q_BYTES);
  #pragma unroll
          for (int t = 0; t < TILES; ++t)
  #pragma unroll
            for (int b = 0; b < BOXES; ++b)
              tma_load_3d(smem + t * Q_BYTES + b * QBOX_BYTES, &p.tmQ, &bars->q_full, b * 64, q0 + t * BR, head);
          for (int j = 0; j < nkv; ++j) {
            const int ks = j % K_STAGES, vs = j % V_STAGES;
            if (!mbar_wait(&bars->k_empty[ks], ((j / K_STAGES) & 1u) ^ 1u, &bars->abort_flag)) {
              report(bars, ATTN_TIMEOUT_PRODUCER, j, 0u);
              break;
            }
            mbar_expect_tx(&bars->k_full[ks], KV_BYTES);
  #pragma unroll
            for (int b = 0; b < BOXES; ++b)
              tma_load_3d(smem + OFF_K + ks * KV_BYTES + b * KVBOX_BYTES, &p.tmK, &bars->k_full[ks], b * 64, key0 + j * BC, head);
            if (!mbar_wait(&bars->v_empty[vs], ((j / V_STAGES) & 1u) ^ 1u, &bars->abort_flag)) {
              report(bars, ATTN_TIMEOUT_PRODUCER, j, 1u);
              break;
            }
            mbar_expect_tx(&bars->v_full[vs], KV_BYTES);
  #pragma unroll
            for (int b = 0; b < BOXES; ++b)
              tma_load_3d(smem + OFF_V + vs * KV_BYTES + b * KVBOX_BYTES, &p.tmV, &bars->v_full[vs], b * 64, key0 + j * BC, head);
          }
        }
      } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer
        // The whole warp walks the loop and elects one lane for each batch of instructions: their descriptors are then
        // warp-uniform values. (With the loop inside an if (lane == 0) every tcgen05.mma took about 125 cycles to issue, twice
        // what a 128 x 128 x 16 product takes to run.) One issuer per tile was slower: the tiles' products then mix on the
        // pipe instead of taking turns, and both softmaxes wait and work at the same time. After a wait somewhere that ran
        // out the loop goes on, over whatever the operands hold.
        const bool q_there = mbar_wait(&bars->q_full, 0u, &bars->abort_flag);
        if (!q_there && lane == 0) report(bars, ATTN_TIMEOUT_MMA, 0u, 0u);
        __syncwarp();
        const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
        const uint64_t qdesc = make_smem_desc(smem_u32(smem), 16, 1024, SWZ_128B);
        const uint64_t kdesc = make_smem_desc(smem_u32(smem + OFF_K), 16, 1024, SWZ_128B);
        const uint64_t vdesc = make_smem_desc(smem_u32(smem + OFF_V), KVBOX_BYTES, 1024, SWZ_128B);
        // S_t of step i. Issued after P_t V of step i - 1 (program order), which is what has read the P that
        // these scores overwrite; the softmax warps of tile t have read the old scores before they wrote that P.
        auto issue_s = [&](int t, int i) {
          const uint64_t ad = qdesc + t * (Q_BYTES >> 4), bd = kdesc + (i % K_STAGES) * (KV_BYTES >> 4);
#pragma unroll
          for (int ks = 0; ks < kD / 16; ++ks) {
            const uint32_t in_row = (ks * 32) % 128, box = (ks * 32) / 128;
            umma_ss<false>(tmem + t * BC, ad + ((box * QBOX_BYTES + in_row) >> 4),
                           bd + ((box * KVBOX_BYTES + in_row) >> 4), IDESC_S, ks > 0 ? 1u : 0u);
          }
          umma_commit(&bars->s_full[t]);
          if (t == TILES - 1) umma_commit(&bars->k_empty[i % K_STAGES]);  // both tiles have read this K tile
        };
        auto issue_pv = [&](int t, int j, int ks0, int ks1) {
          const uint64_t vd = vdesc + (j % V_STAGES) * (KV_BYTES >> 4);
#pragma unroll
          for (int ks = 0; ks < BC / 16; ++ks)
            if (ks >= ks0 && ks < ks1)
              umma_ts<false>(tmem + COL_O + t * kD, tmem + t * BC + ks * 8, vd + ((ks * 16 * 128) >> 4), IDESC_O,
                          (j > 0 || ks > 0) ? 1u : 0u);
        };
        named_bar_sync(BAR_KV, KV_THREADS);  // the first K tile
        tc_fence_after_sync();
        if (elect_one()) {
          issue_s(0, 0);
          if (!kApart) issue_s(1, 0);
        }
        __syncwarp();
        for (int j = 0; j < nkv; ++j) {
          named_bar_sync(BAR_KV, KV_THREADS);
#pragma unroll
          for (int t = 0; t < TILES; ++t) {
            named_bar_sync(BAR_PART + t, PT_THREADS);
            tc_fence_after_sync();
            if (elect_one()) {
              if (kApart && j == 0 && t == 0) issue_s(1, 0);
              issue_pv(t, j, 0, P_PART / 16);
            }
            __syncwarp();
            named_bar_sync(BAR_FULL + t, PT_THREADS);
            tc_fence_after_sync();
            if (elect_one()) {
              issue_pv(t, j, P_PART / 16, BC / 16);
              if (t == TILES - 1) umma_commit(&bars->v_empty[j % V_STAGES]);
              if (j + 1 < nkv) {
                issue_s(t, j + 1);
              } else {
                umma_commit(&bars->o_full[t]);
              }
            }
            __syncwarp();
          }
        }
      } else if (warp == 2) {
        // ------------------------------------------- waits for K and V in the issuer's place
        bool ok = true;
        auto wait = [&](uint64_t* bar, uint32_t parity, uint32_t what, int i) {
          if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar, parity, &bars->abort_flag));
          if (!ok && lane == 0) report(bars, ATTN_TIMEOUT_MMA, what, static_cast<uint32_t>(i));
        };
        wait(&bars->k_full[0], 0u, 1u, 0);
        named_bar_sync(BAR_KV, KV_THREADS);
        for (int j = 0; j < nkv; ++j) {
          wait(&bars->v_full[j % V_STAGES], (j / V_STAGES) & 1u, 2u, j);
          if (j + 1 < nkv) wait(&bars->k_full[(j + 1) % K_STAGES], ((j + 1) / K_STAGES) & 1u, 1u, j + 1);
          named_bar_sync(BAR_KV, KV_THREADS);
        }
      }  // (warp 3 only gives its registers)
      if constexpr (kKeySplit) {  // the two meetings of the cluster that join the partial results
        __syncwarp();
        cluster_sync_all();
        cluster_sync_all();
      }
    } else {
      asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
      // ------------------------------------------------- softmax, correction, epilogue
      const int q = warp & 3;           // TMEM lane quarter this warp may access
      const int t = (warp - 4) >> 2;    // query tile of this warp
      const int row = q * 32 + lane;    // query row of this thread inside its tile
      const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
      const uint32_t col_s = tmem_base + lane_addr + t * BC, col_o = tmem_base + lane_addr + COL_O + t * kD;
      // m: the row's running maximum, which the exponentials of a step are taken against, in the exp2 domain. It has to
      // be the maximum itself: the largest probability is then exactly 1 and does not lose a bit to the 16-bit P. A
      // reference that lagged behind by up to 8 spared most rescaling (32 heads x 4096 x 4096 x 128: 230 against 238 us)
      // but cost 1 to 4 % of the error against 64 bits on normal scores and 15 to 25 % where few keys dominate.
      float m = -INFINITY;
      uint64_t sum2[2] = {f32x2(0.f, 0.f), f32x2(0.f, 0.f)};
      bool ok = true;
      const uint64_t scale2 = f32x2(p.scale_log2, p.scale_log2);
      int j = 0;
      for (; j < nkv; ++j) {
        const bool got = mbar_wait_for(&bars->s_full[t], j & 1u, 4 * KCG_WAIT_LIMIT_NS);
        if (!__all_sync(0xffffffffu, got)) {
          if (lane == 0) report(bars, ATTN_TIMEOUT_SOFTMAX, 0u, static_cast<uint32_t>(j));
          ok = false;
          break;
        }
        tc_fence_after_sync();
        uint32_t sr[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(col_s + c * 32, sr[c]);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 4; ++c) pin_32(sr[c]);
        const int valid = p.sk - key0 - j * BC;
        if (valid < BC) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i >= valid) sr[c][i] = __float_as_uint(-INFINITY);
        }
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        auto max_of = [&](int c) {
#pragma unroll
          for (int i = 0; i < 32; i += 2)
            mx4[(i >> 1) & 3] = max3(mx4[(i >> 1) & 3], __uint_as_float(sr[c][i]), __uint_as_float(sr[c][i + 1]));
        };
#pragma unroll
        for (int c = 0; c < 4; ++c) max_of(c);
        // (the scale is positive: checked by the host)
        const float mx = fmaxf(m, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2);
        // (without a finite score so far the probabilities are 0, not -inf - -inf: a CTA may see excluded keys only)
        const float base = mx == -INFINITY ? 0.f : mx;
        const float alpha = ex2(m - base);
        m = mx;
        const uint64_t alpha2 = f32x2(alpha, alpha), zero2 = f32x2(0.f, 0.f), base2 = f32x2(-base, -base);
        sum2[0] = fma_f32x2(sum2[0], alpha2, zero2);
        sum2[1] = fma_f32x2(sum2[1], alpha2, zero2);
        // Exponentials and P of 32 keys: packed pairs over the S columns this thread has read.
        auto exponentials = [&](int c) {
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float2 e = f32x2_split(fma_f32x2(f32x2(__uint_as_float(sr[c][2 * i]), __uint_as_float(sr[c][2 * i + 1])),
                                             scale2, base2));
            e.x = ex2(e.x);
            e.y = ex2(e.y);
            sum2[i & 1] = add_f32x2(sum2[i & 1], f32x2(e.x, e.y));
            w[i] = pack_pair<kBf16>(e.x, e.y);
          }
          tmem_st_32x32b_x16(col_s + c * 16, w);
        };
        // O_t <- alpha * O_t, where a row of the warp has a new maximum. The previous P_t V has retired: the scores just
        // read were issued behind it. The reads of O travel while the exponentials of the next piece are taken
        // (rescaling the second half of O behind them all: 243 us, a warpgroup of its own that rescales: 258 us).
        if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
          auto scale_store = [&](uint32_t (&o)[32], int c) {
            pin_32(o);
#pragma unroll
            for (int i = 0; i < 32; i += 2) {  // (pairs: 8 x 300 x 16384 x 128 60.3 -> 59.0 us, 32 x 4096 x 4096 x 64 199 -> 197)
              const float2 v = f32x2_split(mul_f32x2(f32x2(__uint_as_float(o[i]), __uint_as_float(o[i + 1])), alpha2));
              o[i] = __float_as_uint(v.x);
              o[i + 1] = __float_as_uint(v.y);
            }
            tmem_st_32x32b_x32(col_o + c * 32, o);
          };
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t o[32];
            tmem_ld_32x32b_x32(col_o + c * 32, o);
            exponentials(c);
            tmem_ld_wait();
            scale_store(o, c);
          }
          if constexpr (kD == 128) {
            static_assert(P_PART == 96, "the third piece of 32 keys comes before the publication");
            uint32_t o[2][32];
            tmem_ld_32x32b_x32(col_o + 64, o[0]);
            tmem_ld_32x32b_x32(col_o + 96, o[1]);
            exponentials(2);
            tmem_ld_wait();
            scale_store(o[0], 2);
            scale_store(o[1], 3);
          }
        } else {
          exponentials(0);
          exponentials(1);
          if constexpr (P_PART == 96) exponentials(2);
        }
        auto publish = [&](uint32_t bar) {
          tmem_st_wait();
          tc_fence_before_sync();
          named_bar_arrive(bar, PT_THREADS);
        };
        publish(BAR_PART + t);
        if constexpr (P_PART == 64) exponentials(2);
        exponentials(3);
        publish(BAR_FULL + t);
      }
      for (; j < nkv; ++j) {  // (given up)
        __syncwarp();
        named_bar_sync(BAR_PART + t, PT_THREADS);
        named_bar_sync(BAR_FULL + t, PT_THREADS);
      }
      const float2 s01 = f32x2_split(add_f32x2(sum2[0], sum2[1]));
      const float l = s01.x + s01.y;
      if (ok) {
        const bool got = mbar_wait(&bars->o_full[t], 0u, &bars->abort_flag);
        if (!__all_sync(0xffffffffu, got)) {
          if (lane == 0) report(bars, ATTN_TIMEOUT_SOFTMAX, 2u, 0u);
          ok = false;
        }
      }
      if constexpr (kKeySplit) {
        // Partial results: once the products of BOTH tiles have retired, the operand ring holds this CTA's O rows
        // (fp32, not normalised, 16-byte units XOR-swizzled by the row: a warp writes 32 rows at a time) and their
        // {maximum, sum}; then each CTA joins an equal share of the output over the cluster's shared memories.
        constexpr int UNITS = kD / 4;  // 16-byte units of a row
        constexpr int OFF_ML = TILES * BR * kD * 4;
        static_assert(OFF_ML + TILES * BR * 8 <= RING_BYTES, "the partial result must fit the ring");
        if (ok) {
          const bool got = mbar_wait(&bars->o_full[t ^ 1], 0u, &bars->abort_flag);
          if (!__all_sync(0xffffffffu, got)) {
            if (lane == 0) report(bars, ATTN_TIMEOUT_SOFTMAX, 3u, 0u);
            ok = false;
          }
        }
        if (ok) {
          tc_fence_after_sync();
          const int r = t * BR + row;
          uint8_t* mine = smem + r * kD * 4;
#pragma unroll
          for (int c = 0; c < kD / 32; ++c) {
            uint32_t o[32];
            tmem_ld_32x32b_x32(col_o + c * 32, o);
            tmem_ld_wait();
            pin_32(o);
#pragma unroll
            for (int u = 0; u < 8; ++u)
              *reinterpret_cast<uint4*>(mine + (((c * 8 + u) ^ (r & (UNITS - 1))) << 4)) =
                  make_uint4(o[4 * u], o[4 * u + 1], o[4 * u + 2], o[4 * u + 3]);
          }
          reinterpret_cast<float2*>(smem + OFF_ML)[r] = make_float2(m, l);
        }
        __syncwarp();
        cluster_sync_all();
        if (ok) {
          const int rows = p.sq - q0 < TILES * BR ? p.sq - q0 : TILES * BR;
          const int u0 = rows * UNITS * rank / p.splits, u1 = rows * UNITS * (rank + 1) / p.splits;
          const uint32_t base_addr = smem_u32(smem);
          T* out = reinterpret_cast<T*>(p.O) + (static_cast<size_t>(head) * p.sq + q0) * kD;
          for (int i = u0 + static_cast<int>(threadIdx.x) - 128; i < u1; i += TILES * 128) {
            const int r = i / UNITS, u = i % UNITS;
            const uint32_t ml_addr = base_addr + OFF_ML + r * 8;
            const uint32_t o_addr = base_addr + r * kD * 4 + ((u ^ (r & (UNITS - 1))) << 4);
            float top = -INFINITY;
            for (int c = 0; c < p.splits; ++c) top = fmaxf(top, ld_cluster_f2(map_to_cta(ml_addr, c)).x);
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
            float sum = 0.f;
#pragma unroll 4
            for (int c = 0; c < p.splits; ++c) {
              const float2 ml = ld_cluster_f2(map_to_cta(ml_addr, c));
              const float4 x = ld_cluster_f4(map_to_cta(o_addr, c));
              const float f = ml.x == -INFINITY ? 0.f : ex2(ml.x - top);
              a.x = fmaf(f, x.x, a.x);
              a.y = fmaf(f, x.y, a.y);
              a.z = fmaf(f, x.z, a.z);
              a.w = fmaf(f, x.w, a.w);
              sum = fmaf(f, ml.y, sum);
            }
            const float inv = 1.f / sum;
            *reinterpret_cast<uint2*>(out + 4 * static_cast<size_t>(i)) =
                make_uint2(pack_pair<kBf16>(a.x * inv, a.y * inv), pack_pair<kBf16>(a.z * inv, a.w * inv));
          }
        }
        __syncwarp();
        cluster_sync_all();  // the other CTAs read this one's shared memory until here
        griddep_wait();      // behind a launch of whole groups: complete after it, so that what follows waits for both
      } else {
        if (ok) {
          tc_fence_after_sync();
          const float inv = 1.f / l;
          const int grow = q0 + t * BR + row;
          T* out = reinterpret_cast<T*>(p.O) + (static_cast<size_t>(head) * p.sq + grow) * kD;
  #pragma unroll
          for (int c = 0; c < kD / 32; ++c) {
            uint32_t r[32];
            tmem_ld_32x32b_x32(col_o + c * 32, r);
            tmem_ld_wait();
            if (grow < p.sq) {
  #pragma unroll
              for (int u = 0; u < 4; ++u) {
                uint32_t w[4];
  #pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const float a = __uint_as_float(r[u * 8 + 2 * e]) * inv, bb = __uint_as_float(r[u * 8 + 2 * e + 1]) * inv;
                  if constexpr (kBf16) {
                    __nv_bfloat162 v2 = __floats2bfloat162_rn(a, bb);
                    w[e] = *reinterpret_cast<uint32_t*>(&v2);
                  } else {
                    __half2 v2 = __floats2half2_rn(a, bb);
                    w[e] = *reinterpret_cast<uint32_t*>(&v2);
                  }
                }
                *reinterpret_cast<uint4*>(out + c * 32 + u * 8) = make_uint4(w[0], w[1], w[2], w[3]);
              }
            }
          }
        }
      }
    }

    // ---------------------------------------------------------------- common exit
    __syncwarp();
    if (bars->abort_flag != 0u) {
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
      tc_fence_after_sync();
      tmem_dealloc(tmem_base, TMEM_COLS);
    }
  }
};

template <int kD, bool kBf16, bool kKeySplit>
__global__ void __launch_bounds__(384, 1) kcg_attention2_kernel(const __grid_constant__ AttnParams p) {
  AttnFwd2<kD, kBf16, kKeySplit>::run(p);
}

template <int kD, bool kBf16, int kBC, int kSplit, int kPTmem>
__global__ void __launch_bounds__(64 + 128 * kSplit, (kBC == 64 && kSplit == 1) ? 2 : 1)
kcg_attention_kernel(const __grid_constant__ AttnParams p) {
  AttnFwd<kD, kBf16, kBC, kSplit, kPTmem>::run(p);
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeFn g_encode = nullptr;
bool g_ready[16][36];  // [device][kernel instance]: dynamic shared memory opted in
std::mutex g_mutex;

int fail(int code, const std::string& msg) { return kcg_internal_fail(code, msg.c_str()); }
int cuda_fail(cudaError_t e, const char* what) {
  return fail(static_cast<int>(e), std::string(what) + ": " + cudaGetErrorString(e));
}

// KCG_PDL=0 turns programmatic dependent launch off (read once, at the first launch of the process).
bool pdl_on() {
  static const bool on = [] {
    const char* e = getenv("KCG_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}

struct DeviceGuard {
  int prev = -1;
  bool switched = false;
  cudaError_t enter(int device) {
    cudaError_t e = cudaGetDevice(&prev);
    if (e != cudaSuccess) return e;
    if (prev == device) return cudaSuccess;
    e = cudaSetDevice(device);
    switched = (e == cudaSuccess);
    return e;
  }
  ~DeviceGuard() {
    if (switched) cudaSetDevice(prev);
  }
};

// {d, rows, heads} view of a contiguous heads x rows x d tensor; boxes of 64 values x `box_rows` rows of one
// head. Rows past the end of a head read as zero.
int encode3(CUtensorMap* tm, bool bf16, uint64_t ptr, int d, int rows, int heads, int box_rows) {
  cuuint64_t gdim[3] = {static_cast<cuuint64_t>(d), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(heads)};
  cuuint64_t gstride[2] = {static_cast<cuuint64_t>(d) * 2, static_cast<cuuint64_t>(d) * 2 * static_cast<cuuint64_t>(rows)};
  cuuint32_t box[3] = {64, static_cast<cuuint32_t>(box_rows), 1};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = g_encode(tm, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3,
                              reinterpret_cast<void*>(ptr), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(static_cast<int>(r), "cuTensorMapEncodeTiled failed");
  return 0;
}

struct Problem {
  uint64_t Q, K, V, O;
  int heads, sq, sk, d;
  float scale;
  bool bf16;
};

template <int kD, bool kBf16, int kBC, int kSplit, int kPTmem>
int launch(int device, int slot, cudaStream_t st, const Problem& pb) {
  using Kern = AttnFwd<kD, kBf16, kBC, kSplit, kPTmem>;
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_ready[device][slot]) {
      const cudaError_t e = cudaFuncSetAttribute(kcg_attention_kernel<kD, kBf16, kBC, kSplit, kPTmem>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, Kern::SMEM_BYTES);
      if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(MaxDynamicSharedMemorySize)");
      g_ready[device][slot] = true;
    }
  }
  AttnParams p{};
  if (int r = encode3(&p.tmQ, kBf16, pb.Q, kD, pb.sq, pb.heads, 128)) return r;
  if (int r = encode3(&p.tmK, kBf16, pb.K, kD, pb.sk, pb.heads, kBC)) return r;
  if (int r = encode3(&p.tmV, kBf16, pb.V, kD, pb.sk, pb.heads, kBC)) return r;
  p.O = reinterpret_cast<void*>(pb.O);
  p.sq = pb.sq;
  p.sk = pb.sk;
  p.scale_log2 = pb.scale * 1.4426950408889634f;
  const int grid = pb.heads * ((pb.sq + 127) / 128);
  kcg_attention_kernel<kD, kBf16, kBC, kSplit, kPTmem><<<grid, Kern::NUM_THREADS, Kern::SMEM_BYTES, st>>>(p);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "attention launch");
  kcg_internal_count_launch();
  return 0;
}

// Clusters of 1 .. 16 CTAs of the few-row kernels that run at once (asked once per device, kernel and size; -1 = none).
int g_few_clusters[16][12][17];

// How many clusters of 2 .. 8 CTAs of the key-split kernel run at once (asked once per device and kernel), and SMs.
int g_clusters[16][4][9];
int g_sms[16];

// The largest number of CTAs, 2 to 8, that `groups` groups of 256 rows can share their keys among with every cluster
// running at once and at least four steps of 128 keys per CTA (joining costs what two steps do); 1 = none.
int key_splits(const int (&clusters)[9], long long groups, int sk) {
  const int steps = (sk + 127) / 128;
  for (int s = 8; s >= 2; --s)
    if (groups <= clusters[s] && steps >= 4 * s) return s;
  return 1;
}

template <int kD, bool kBf16>
int launch2(int device, int kind, cudaStream_t st, const Problem& pb) {
  using Kern = AttnFwd2<kD, kBf16, false>;
  using Split = AttnFwd2<kD, kBf16, true>;
  const auto whole = kcg_attention2_kernel<kD, kBf16, false>;
  const auto split = kcg_attention2_kernel<kD, kBf16, true>;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(Split::NUM_THREADS);
  cfg.dynamicSmemBytes = Split::SMEM_BYTES;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_ready[device][16 + kind]) {
      cudaError_t e = cudaFuncSetAttribute(whole, cudaFuncAttributeMaxDynamicSharedMemorySize, Kern::SMEM_BYTES);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(split, cudaFuncAttributeMaxDynamicSharedMemorySize, Split::SMEM_BYTES);
      if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(MaxDynamicSharedMemorySize)");
      for (int s = 2; s <= 8; ++s) {
        attr[0].val.clusterDim.x = s;
        cfg.gridDim = dim3(s);
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, split, &cfg) != cudaSuccess) {
          cudaGetLastError();  // not known: this size is not used
          n = 0;
        }
        g_clusters[device][kind][s] = n;
      }
      e = cudaDeviceGetAttribute(&g_sms[device], cudaDevAttrMultiProcessorCount, device);
      if (e != cudaSuccess) return cuda_fail(e, "cudaDeviceGetAttribute(MultiProcessorCount)");
      g_ready[device][16 + kind] = true;
    }
  }
  AttnParams p{};
  if (int r = encode3(&p.tmQ, kBf16, pb.Q, kD, pb.sq, pb.heads, 128)) return r;
  if (int r = encode3(&p.tmK, kBf16, pb.K, kD, pb.sk, pb.heads, 128)) return r;
  if (int r = encode3(&p.tmV, kBf16, pb.V, kD, pb.sk, pb.heads, 128)) return r;
  p.O = reinterpret_cast<void*>(pb.O);
  p.sq = pb.sq;
  p.sk = pb.sk;
  p.scale_log2 = pb.scale * 1.4426950408889634f;
  // A group of 256 rows keeps one SM for the whole walk over the keys, so a wave is one group per SM. What does not fill a
  // wave - the remainder of a large problem, all of a small one - shares its keys among the SMs that would stand idle:
  // (bf16) 32 heads x 4096 x 4096 x 128, 3.46 waves, then 246 -> 230 us; 8 x 300 x 16384 x 128, 16 groups: 224 -> 59 us; 8 x 65
  // x 16384 x 64, 8 groups: 33 us.
  // The remainder is a launch of its own right behind the whole groups, allowed to start as soon as all of those have.
  const long long groups = static_cast<long long>(pb.heads) * ((pb.sq + 255) / 256);
  const long long rest = groups % g_sms[device];
  const int s = rest ? key_splits(g_clusters[device][kind], rest, pb.sk) : 1;
  const long long full = s > 1 ? groups - rest : groups;
  if (full > 0) {
    p.tail_follows = s > 1 ? 1 : 0;
    whole<<<static_cast<unsigned>(full), Kern::NUM_THREADS, Kern::SMEM_BYTES, st>>>(p);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "attention launch");
    kcg_internal_count_launch();
  }
  if (s > 1) {
    p.first_group = static_cast<int>(full);
    p.splits = s;
    p.tail_follows = 0;
    attr[0].val.clusterDim.x = s;
    cfg.gridDim = dim3(static_cast<unsigned>(rest * s));
    cfg.numAttrs = full > 0 && pdl_on() ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, split, p);
    if (e != cudaSuccess) return cuda_fail(e, "attention launch");
    kcg_internal_count_launch();
  }
  return 0;
}

// CTAs that share a head's keys in the decode form (one cluster). Two CTAs of this size fit an SM, but a cluster has to
// fit one GPC: beyond about 264 CTAs some clusters wait for a second wave (32 heads x 8192 x 128: 8 CTAs per head
// 26 us, 9 35 us; 100 heads x 4096: 2 per head 37 us, 3 46 us), pairs alone pack all 296 places. More than 8 per head
// pay only where fewer heads leave SMs idle (8 heads x 16384: 8 per head 21.2 us, 12 19.5, 16 18.6; 20 heads x 8192:
// 8 23.9, 10 21.7, 16 33.9 us). At least two stages of 64 keys each: below that the joining costs what the walk saves.
// A cluster of more CTAs than any GPC can hold (`fits`: fewer SMs than a whole GPU's) is not asked for.
template <typename Fits>
int decode_splits(int heads, int sk, Fits&& fits) {
  const int tiles = (sk + 63) / 64;
  int s = heads <= 148 && heads > 132 ? 2 : 264 / heads;
  if (s > 8) s = 200 / heads > 8 ? 200 / heads : 8;
  if (s > 16) s = 16;
  if (s > tiles / 2) s = tiles / 2;
  while (s > 1 && !fits(s)) --s;
  return s < 1 ? 1 : s;
}

// Whether the few-row form takes a call. Up to 32 rows always: the 256-row kernel loses everywhere (32 heads x 1 x 8192 x
// 128: 148 against 26 us, 32 x 32 x 8192 x 128 38 / 28 us, 100 x 32 x 4096 61 / 40 us, 128 x 16 x 256 9.9 / 8.3 us). At 33
// to 64 rows each of its four warps reads all keys from shared memory, which costs most at d = 128. Measured on 8 to 128
// heads x 40 and 64 rows x 256 to 8192 keys, bf16, few-row time over that of the 256-row kernel:
//   d = 64   0.47 to 0.95 from 512 keys on, whatever the heads (32 x 64 x 4096 16 / 22 us, 128 x 64 x 8192 69 / 103 us);
//            at 256 keys 0.80 to 1.11 (7 us either way)
//   d = 128  up to 32 heads 0.66 to 1.04 from 512 to 1536 keys (8 x 64 x 1024 11 / 16 us), then 0.97 to 1.14 (with 8 heads
//            only from 3072 keys on); where at least three CTAs share a head (up to 88 heads) 0.77 to 1.02 from 1536 keys on
//            (48 x 64 x 4096 36 / 40 us, 80 x 64 x 4096 51 / 61 us) and 0.93 to 1.49 below; with 100 and 128 heads 1.00 to
//            1.45.
// At 65 rows the warps would have to walk the keys twice.
bool few_rows_form(int heads, int sq, int sk, int d) {
  if (sq <= 32) return true;
  if (sq > 64 || sk < 512) return false;
  if (d == 64) return true;
  if (heads <= 32) return sk < (heads <= 8 ? 3072 : 2048);
  return heads <= 88 && sk >= 1536;
}

template <int kD, bool kBf16, int kRowGroups>
int launch_decode(int device, int slot, cudaStream_t st, const Problem& pb) {
  using Kern = AttnDecode<kD, kBf16, kRowGroups>;
  const auto kernel = kcg_attention_decode_kernel<kD, kBf16, kRowGroups>;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(Kern::NUM_THREADS);
  cfg.dynamicSmemBytes = Kern::SMEM_BYTES;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  AttnDecodeParams p{};
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_ready[device][slot]) {
      cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Kern::SMEM_BYTES);
      if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(MaxDynamicSharedMemorySize)");
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(NonPortableClusterSizeAllowed)");
      g_ready[device][slot] = true;
    }
    p.splits = decode_splits(pb.heads, pb.sk, [&](int s) {
      int& known = g_few_clusters[device][slot - 20][s];
      if (known == 0) {
        attr[0].val.clusterDim.x = s;
        cfg.gridDim = dim3(s);
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&known, kernel, &cfg) != cudaSuccess) cudaGetLastError();
        if (known <= 0) known = -1;
      }
      return known > 0;
    });
  }
  if (int r = encode3(&p.tmK, kBf16, pb.K, kD, pb.sk, pb.heads, 64)) return r;
  if (int r = encode3(&p.tmV, kBf16, pb.V, kD, pb.sk, pb.heads, 64)) return r;
  p.Q = reinterpret_cast<const void*>(pb.Q);
  p.O = reinterpret_cast<void*>(pb.O);
  p.sq = pb.sq;
  p.sk = pb.sk;
  p.scale_log2 = pb.scale * 1.4426950408889634f;
  attr[0].val.clusterDim.x = p.splits;
  cfg.gridDim = dim3(static_cast<unsigned>(pb.heads) * p.splits);
  cfg.numAttrs = pdl_on() ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
  if (e != cudaSuccess) return cuda_fail(e, "attention launch");
  kcg_internal_count_launch();
  return 0;
}

template <int kRowGroups>
int launch_decode_shape(int device, int base_slot, cudaStream_t st, const Problem& pb) {
  if (pb.d == 128)
    return pb.bf16 ? launch_decode<128, true, kRowGroups>(device, base_slot, st, pb)
                   : launch_decode<128, false, kRowGroups>(device, base_slot + 1, st, pb);
  return pb.bf16 ? launch_decode<64, true, kRowGroups>(device, base_slot + 2, st, pb)
                 : launch_decode<64, false, kRowGroups>(device, base_slot + 3, st, pb);
}

template <int kBC, int kSplit, int kPTmem>
int launch_shape(int device, int base_slot, cudaStream_t st, const Problem& pb) {
  if (pb.d == 128)
    return pb.bf16 ? launch<128, true, kBC, kSplit, kPTmem>(device, base_slot, st, pb)
                   : launch<128, false, kBC, kSplit, kPTmem>(device, base_slot + 1, st, pb);
  return pb.bf16 ? launch<64, true, kBC, kSplit, kPTmem>(device, base_slot + 2, st, pb)
                 : launch<64, false, kBC, kSplit, kPTmem>(device, base_slot + 3, st, pb);
}

}  // namespace

// For tests of the host logic: 1 where kcg_attention_fwd takes the few-row form for a call, else 0.
extern "C" int kcg_internal_attention_few_rows(int heads, int sq, int sk, int d) {
  return few_rows_form(heads, sq, sk, d) ? 1 : 0;
}

// For tests of the host logic: the CTAs per head of the few-row form where bit s of `fitting` says that a cluster of s fits.
extern "C" int kcg_internal_attention_splits(int heads, int sk, unsigned int fitting) {
  return decode_splits(heads, sk, [&](int s) { return (fitting >> s & 1u) != 0u; });
}

extern "C" int kcg_attention_fwd(int device, uint64_t stream, uint64_t Q, uint64_t K, uint64_t V, uint64_t O, int dtype,
                                 int heads, int sq, int sk, int d, float scale) {
  if (!Q || !K || !V || !O) return fail(KCG_E_BAD_ARG, "null device pointer");
  if (heads <= 0 || sq <= 0 || sk <= 0) return fail(KCG_E_BAD_ARG, "empty shape");
  if (!(dtype == KCG_DTYPE_BFLOAT16 || dtype == KCG_DTYPE_FLOAT16))
    return fail(KCG_E_BAD_ARG, "the fused attention kernel takes float16 or bfloat16 data");
  if (!(d == 64 || d == 128)) return fail(KCG_E_BAD_CONFIG, "head dimension must be 64 or 128");
  if (!(scale > 0.f) || !std::isfinite(scale)) return fail(KCG_E_BAD_ARG, "scale must be positive and finite");
  if (device < 0 || device >= 16) return fail(KCG_E_BAD_ARG, "device index out of range");
  if (Q % 16 || K % 16 || V % 16 || O % 16) return fail(KCG_E_BAD_ARG, "operands must start on 16-byte boundaries");
  const long long tiles = static_cast<long long>(heads) * ((sq + 127) / 128);
  if (tiles > 0x7fffffffLL) return fail(KCG_E_TOO_LARGE, "too many query tiles for one launch");
  DeviceGuard guard;
  cudaError_t e = guard.enter(device);
  if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_encode) {
      void* fn = nullptr;
      cudaDriverEntryPointQueryResult qres;
      e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres);
      if (e != cudaSuccess || qres != cudaDriverEntryPointSuccess || !fn)
        return fail(KCG_E_NO_DRIVER, "cuTensorMapEncodeTiled not available from the driver");
      g_encode = reinterpret_cast<EncodeFn>(fn);
    }
  }
  Problem pb{Q, K, V, O, heads, sq, sk, d, scale, dtype == KCG_DTYPE_BFLOAT16};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // Default: two query tiles per CTA that alternate on the tensor pipe (AttnFwd2; the fastest form measured).
  // KCG_ATTN_FORM selects a comparison form with ONE query tile per CTA: 4 = 128-key steps, two threads per row,
  // P in tensor memory; 5 = 64-key steps, one thread per row, two CTAs per SM; 6 and 7 = the same two with P
  // through shared memory.
  static const int form = [] {
    const char* v = getenv("KCG_ATTN_FORM");
    return v ? atoi(v) & 15 : 0;
  }();
  // KCG_ATTN_FORM=8: the 256-row kernel for every number of queries.
  if (form == 0 && few_rows_form(heads, sq, sk, d)) {
    if (sq <= 16) return launch_decode_shape<1>(device, 20, st, pb);
    if (sq <= 32) return launch_decode_shape<2>(device, 24, st, pb);
    return launch_decode_shape<4>(device, 28, st, pb);
  }
  switch (form) {
    case 4: return launch_shape<128, 2, 1>(device, 0, st, pb);
    case 5: return launch_shape<64, 1, 1>(device, 4, st, pb);
    case 6: return launch_shape<128, 2, 0>(device, 8, st, pb);
    case 7: return launch_shape<64, 1, 0>(device, 12, st, pb);
    default:
      if (pb.d == 128) return pb.bf16 ? launch2<128, true>(device, 0, st, pb) : launch2<128, false>(device, 1, st, pb);
      return pb.bf16 ? launch2<64, true>(device, 2, st, pb) : launch2<64, false>(device, 3, st, pb);
  }
}

// Reads (and clears) the status word of the fused attention kernels on `device`: out = {code, block, detail,
// detail}; code 0 = no bounded wait has run out since the last call. Synchronises the device.
extern "C" int kcg_attention_status(int device, uint32_t out[4]) {
  if (!out) return fail(KCG_E_BAD_ARG, "null argument");
  DeviceGuard guard;
  cudaError_t e = guard.enter(device);
  if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
  e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return cuda_fail(e, "cudaDeviceSynchronize");
  e = cudaMemcpyFromSymbol(out, g_attn_status, sizeof(uint32_t) * 4);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyFromSymbol");
  if (out[0] != 0u) {
    const uint32_t zero[4] = {0u, 0u, 0u, 0u};
    e = cudaMemcpyToSymbol(g_attn_status, zero, sizeof(zero));
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyToSymbol");
    return fail(KCG_E_DEVICE_TIMEOUT, "a bounded wait of the attention kernel ran out");
  }
  return 0;
}
