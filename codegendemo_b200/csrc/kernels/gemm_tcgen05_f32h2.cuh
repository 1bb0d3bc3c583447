// fp32 GEMM with fp32-level accuracy from three fp16 products, CTA pairs. The operands arrive split: a kernel in front
// (csrc/kcg_f32split.cu) has written every value x as two fp16 parts,
//     x * 2^e = hi + 2^-12 lo,   hi = fp16(x * 2^e),  lo = fp16((x * 2^e - hi) * 2^12),
// where the values that share an exponent e - 64 values of K of a row of A, or of 64 columns of B, each column multiplied by
// a power of two of its own before - have their largest in [2^14, 2^15). hi and lo carry 22 bits between them, as the two
// TF32 parts of gemm_tcgen05_f32x3.cuh do, but hi is rounded where kind::tf32 truncates, so lo * lo, which both leave out, is
// below 2^-24 of the product instead of 2^-20; and kind::f16 multiplies twice as many values a cycle as kind::tf32 and reads
// half as many bytes for it. Error against 64 bits, uniform values: 1.4e-7 at K = 1024, 1.9e-7 at 4096, 2.6e-7 at 11008,
// where 3xTF32 has 1.0e-6 (normwise; largest 2e-6 and 5e-6).
// A chunk with a value so far (about 2^-30) below the largest one beside it that its parts would keep less than 21 bits has far
// parts: such values alone, under an exponent of their own, in one of a limited number of slots (kcg_f32split.cu). It is multiplied
// once more for them. What does not split at all - an infinity, a NaN, values whose largest is outside 2^+-50, more chunks with far
// parts than slots - sets a word, and this kernel then multiplies the fp32 operands as 3xTF32 (TcGemmF32x3, in the same launch):
// no input loses accuracy over that kernel. Values drawn from a normal distribution need far parts about once in thirty products of
// 4096 x 4096 operands. Times of a call with values that all split / with one far value / that fall back after the split (every
// value of A exp(8 x normal)) / of 3xTF32 alone, us: 1024x7936x768 48 / 57 / 86 / 66, 1536x5632x1024 56 / 65 / 105 / 84, 512x11008x4096
// 177 / 213 / 242 / 209, 2048x4096x4096 188 / 250 / 336 / 300, 4096^3 380 / 426 / 592 / 566, 2048x11008x11008 1350 / 1477 / 2073 / 2012 (calls in
// a row; without far parts one such value took 82, 96, 239, 349, 609, 2115).
//
// Each 64 values of K (a chunk) are multiplied into a fresh accumulator in tensor memory, the two correction products
// first; the first hi * hi product scales what they have summed by 2^-12 (scale-input-d). The accumulating warps add
// d * 2^-(eA + eB) to their registers (round to nearest) while the other accumulator fills: the tensor core adds with
// truncation, an error that grows with the length of such a sum.
//
// What bounds it: a chunk of a 256x256 tile takes 1536 cycles of the tensor pipe; through the shared-memory port go 64 KB
// from TMA and 144 KB to the products, 1625 cycles at 128 bytes each (256x128: 768 and 1152). Measured 1600 in the main loop
// (3xTF32: 3540 for the same), then the power cap; before and behind it about 3500 cycles to the first chunk, 4100 to store
// 128 KB, 2000 to leave. (With an exponent per column, spread over shared memory to every thread, 2300: a 16-byte broadcast
// takes the port for four cycles.) Both operands are read and written once more in memory for the split, 41 us at 4096 x 4096.
// 3xTF32 -> this, graph replay in turn: 4096^3 495 -> 350 us, 2048x4096x4096 269 -> 182, 2048x11008x11008 1994 -> 1316,
// 1536x5632x1024 79 -> 56, 512x11008x4096 190 -> 177, 1024^3 21.1 -> 20.4, 256x8704x2560 54 -> 69 (not chosen there).
//
// Warp roles (as many threads as the 3xTF32 kernel this one falls back to): warp 0 TMA producer, warp 1 MMA issuer (of
// the leader CTA) and TMEM owner, the last two warpgroups accumulate and store; the others only give their registers.
#pragma once
#include "epilogue.cuh"
#include "gemm_params.h"
#include "gemm_tcgen05_f32x3.cuh"
#include "ptx_sm100.cuh"
#include "work_iter.cuh"

namespace kcg {

template <int kBN, int kSplitK, int kGroup>
struct TcGemmF32H2 {
  static constexpr int kBM = 256, kBK = H2_BK, BNL = kBN / 2;
  static_assert(h2_config_error(kBM, kBN, kBK) == 0, "config not buildable by the split fp32 kernel");
  using Fallback = TcGemmF32x3<kBM, kBN, 32, h2_x3_stages(kBN), 0, kSplitK, kGroup, 4, 1>;
  static constexpr int NUM_THREADS = Fallback::NUM_THREADS;
  static constexpr int FIRST_ACC_WARP = Fallback::FIRST_ACC_WARP, NUM_EPI_THREADS = 256;
  // a stage: A, 128 rows of hi and 128 of lo (K-major, 128 bytes a row); B, for each 64 columns 64 values of K of hi and of
  // lo (columns contiguous, 128 bytes a row). One tensor map of 128-byte rows for both, boxes of 128 rows.
  static constexpr int BOX_BYTES = 128 * 128, A_BYTES = 2 * BOX_BYTES, STAGE_BYTES = A_BYTES + BNL / 64 * BOX_BYTES;
  static constexpr int kStages = h2_stages(kBN);
  static constexpr int RING_BYTES = kStages * STAGE_BYTES;
  static constexpr int STORE_BYTES = 8 * 32 * 128;  // a block of 32 x 32 results for each accumulating warp
  static constexpr uint32_t IDESC = make_instr_desc(FMT_F16, 0u, 1u, 256u, kBN);
  static constexpr int TMEM_COLS = 2 * kBN;
  static constexpr int KSTEPS = kBK / 16;
  static constexpr int HALF_COLS = kBN / 2, PIECES = HALF_COLS / 32, CHUNKS = HALF_COLS / 64;
  // registers of a thread after setmaxnreg (launched with 128 each of 512 threads, or 96 of 640)
  static constexpr int CTL_REGS = 48, IDLE_REGS = 24;
  static constexpr int ACC_REGS = NUM_THREADS == 512 ? 216 : 192;
  static_assert(CTL_REGS + (NUM_THREADS / 128 - 3) * IDLE_REGS + 2 * ACC_REGS <=
                    (NUM_THREADS == 512 ? 4 * 128 : 5 * 96), "register split");
  static constexpr int SMEM_BYTES = h2_smem_bytes(kBN);

  struct Barriers {
    uint64_t full[kStages], empty[kStages];
    uint64_t tmem_full[2], tmem_empty[2];
    uint32_t tmem_base;
    volatile uint32_t abort_flag;
    uint32_t last_flag;
  };
  static_assert(RING_BYTES + STORE_BYTES + sizeof(Barriers) + 1024 <= SMEM_BYTES && sizeof(Barriers) <= 1024, "shared memory");

  using Unit = WorkUnit;
  using Iter = WorkIter<kBM, kBN, kGroup, KCG_SERPENTINE>;

  __device__ static __forceinline__ void report(const KcgGemmParams& p, Barriers* bars, uint32_t code, uint32_t d0,
                                                uint32_t d1) {
    bars->abort_flag = 1u;
    if (atomicCAS(p.status, 0u, code) == 0u) {
      p.status[1] = blockIdx.x;
      p.status[2] = d0;
      p.status[3] = d1;
    }
  }

  // The chunks that a unit of a product with far parts multiplies, in order, as runs: of every K block the parts (what = 0) and, where
  // one of the tile's panels of A or chunks of B has far parts there, those of A with the parts of B (1), those of B with the parts
  // of A (2), both (3), each a run of one; panels and chunks that have none stand in with zeros. Every role walks the same sequence.
  // Without far parts a unit is one run: the roles' inner loops go over a run, by increments alone, and know nothing of all this.
  // (With the walk inside the accumulating loop 2048x4096x4096 took 248 us instead of 188, with that loop compiled twice 196.)
  struct Chunks {
    const KcgGemmParams& p;
    int m0, n0, kb, run, end;
    uint32_t what, left;  // left: bit `what` of the runs of this K block that are still to come
    int base;             // K blocks base .. base + 31: which of them have far parts of A, of B
    uint32_t with_a, with_b;
    __device__ __forceinline__ Chunks(const KcgGemmParams& p_, const Unit& w)
        : p(p_), m0(w.m0), n0(w.n0), kb(w.kb0), run(0), end(w.kb0 + w.kbn), what(0u), left(0u), base(w.kb0 - 32), with_a(0u), with_b(0u) {}
    // slots of far parts (0: none) of panel i of the tile's rows and of chunk i of its columns
    __device__ __forceinline__ int slot_a(int k, int i) const {
      if (m0 + i * 128 >= p.M) return 0;
      return __float_as_uint(__ldcg(p.scale_a + static_cast<size_t>(k) * p.scale_lda + m0 + i * 128)) & H2_SLOT_BITS;
    }
    __device__ __forceinline__ int slot_b(int k, int i) const {
      if (n0 + i * 64 >= p.N) return 0;
      return __float_as_uint(__ldcg(p.scale_b + static_cast<size_t>(k) * p.scale_ldb + (n0 >> 6) + i)) & H2_SLOT_BITS;
    }
    __device__ __forceinline__ bool any_a(int k) const { return (slot_a(k, 0) | slot_a(k, 1)) != 0; }
    __device__ __forceinline__ bool any_b(int k) const {
      int any = 0;
#pragma unroll
      for (int i = 0; i < kBN / 64; ++i) any |= slot_b(k, i);
      return any != 0;
    }
    // The next run; false: none. A whole warp looks up 32 K blocks together and walks those without far parts as one run; one
    // thread takes them one by one.
    template <bool kWarp>
    __device__ __forceinline__ bool next() {
      if (left == 0u) {
        kb += run;
        if (kb >= end) return false;
        if (kWarp) {
          if (kb >= base + 32) {
            base = kb;
            const int k = base + static_cast<int>(threadIdx.x & 31);
            with_a = __ballot_sync(0xffffffffu, k < end && any_a(k));
            with_b = __ballot_sync(0xffffffffu, k < end && any_b(k));
          }
        } else {
          base = kb;
          with_a = any_a(kb) ? 1u : 0u;
          with_b = any_b(kb) ? 1u : 0u;
        }
        const uint32_t a = with_a >> (kb - base), b = with_b >> (kb - base);
        const int clear = (a | b) != 0u ? __ffs(a | b) - 1 : 32;  // K blocks without far parts from here on
        const int rest = (kWarp && end - base > 32 ? base + 32 : end) - kb;
        run = !kWarp || clear == 0 ? 1 : clear < rest ? clear : rest;
        left = 1u | (clear != 0 ? 0u : (a & 1u) << 1 | (b & 1u) << 2 | (a & b & 1u) << 3);
      }
      what = __ffs(left) - 1;
      left &= left - 1u;
      return true;
    }
    __device__ __forceinline__ bool far_a() const { return (what & 1u) != 0u; }
    __device__ __forceinline__ bool far_b() const { return (what & 2u) != 0u; }
  };

  __device__ static __forceinline__ void roles(const KcgGemmParams& p, uint8_t* smem, Barriers* bars, uint32_t tmem_base, uint32_t rank,
                                               bool far) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_m = (p.M + kBM - 1) / kBM, tiles_n = (p.N + kBN - 1) / kBN;
    const int num_kb = (p.K + kBK - 1) / kBK;
    const int unit0 = static_cast<int>(blockIdx.x >> 1), unit_stride = static_cast<int>(gridDim.x >> 1);
    if (warp < 4) {
      Fallback::template reg_dec<CTL_REGS>();
      if (warp == 1) tmem_relinquish_pair();
      if (warp == 0 && lane == 0) {
        // ---------------------------------------------------------- producer
        uint32_t it = 0;
        bool ok = true;
        Iter units(p, unit0, unit_stride, tiles_m, tiles_n, num_kb);
        Unit w;
        while (ok && units.next(w)) {
          const int a_row0 = ((w.m0 >> 7) + static_cast<int>(rank)) * num_kb;
          const int b_chunk0 = (w.n0 + static_cast<int>(rank) * BNL) >> 6;
          int a_row, b_row[BNL / 64];
          auto rows_of = [&](int kb) {
            // (chunks of columns past the problem, and those without far parts, lie past the map or are read as something for
            // results that are not stored, as are panels of rows past it)
            a_row = (a_row0 + kb) * 256;
#pragma unroll
            for (int j = 0; j < BNL / 64; ++j) b_row[j] = p.parts_b_row + ((b_chunk0 + j) * num_kb + kb) * 128;
          };
          auto load = [&](int run) {
            for (int i = 0; i < run; ++i, ++it) {
              const uint32_t s = it % kStages;
              if (!mbar_wait(&bars->empty[s], ((it / kStages) & 1u) ^ 1u, &bars->abort_flag)) {
                report(p, bars, KCG_ST_TIMEOUT_PRODUCER, it, s);
                ok = false;
                break;
              }
              // completion bytes of both CTAs land on the leader's barrier
              const uint32_t full_leader = map_to_cta(smem_u32(&bars->full[s]), 0u);
              if (rank == 0u) mbar_expect_tx(&bars->full[s], static_cast<uint32_t>(2 * STAGE_BYTES));
              uint8_t* sa = smem + s * STAGE_BYTES;
#pragma unroll
              for (int j = 0; j < 2; ++j) tma_load_2d_pair(sa + j * BOX_BYTES, &p.tmWs, full_leader, 0, a_row + j * 128);
#pragma unroll
              for (int j = 0; j < BNL / 64; ++j) tma_load_2d_pair(sa + A_BYTES + j * BOX_BYTES, &p.tmWs, full_leader, 0, b_row[j]);
              a_row += 256;
#pragma unroll
              for (int j = 0; j < BNL / 64; ++j) b_row[j] += 128;
            }
          };
          if (!far) {
            rows_of(w.kb0);
            load(w.kbn);
            continue;
          }
          for (Chunks ch(p, w); ok && ch.template next<false>();) {
            rows_of(ch.kb);
            if (ch.far_a()) {
              const int slot = ch.slot_a(ch.kb, static_cast<int>(rank));
              a_row = slot > 0 ? p.far_a_row + (slot - 1) * 256 : p.parts_rows;
            }
            if (ch.far_b()) {
#pragma unroll
              for (int j = 0; j < BNL / 64; ++j) {
                const int slot = ch.slot_b(ch.kb, static_cast<int>(rank) * (BNL / 64) + j);
                b_row[j] = slot > 0 ? p.far_b_row + (slot - 1) * 128 : p.parts_rows;
              }
            }
            load(1);
          }
        }
        griddep_launch_dependents();  // every load is issued: the stream's next kernel may be brought in
      } else if (warp == 1 && rank == 0u) {
        // ------------------------------------- MMA issuer: whole warp, one elected lane per chunk
        const uint32_t tmem_base_u = __shfl_sync(0xffffffffu, tmem_base, 0);
        const uint64_t ring_a = make_smem_desc(smem_u32(smem), 16, 1024, SWZ_128B);
        const uint64_t ring_b = make_smem_desc(smem_u32(smem) + A_BYTES, BOX_BYTES, 1024, SWZ_128B);
        uint32_t it = 0;
        bool ok = true;
        Iter units(p, unit0, unit_stride, tiles_m, tiles_n, num_kb);
        Unit w;
        while (ok && units.next(w)) {
          Chunks ch(p, w);
          for (bool more = true; more && ok; more = far) {  // (one run without far parts)
            if (far && !ch.template next<true>()) break;
            const int run = far ? ch.run : w.kbn;
            for (int i = 0; i < run; ++i, ++it) {
              const uint32_t s = it % kStages, ab = it & 1u;
              if (!mbar_wait_warp(&bars->tmem_empty[ab], ((it >> 1) & 1u) ^ 1u, &bars->abort_flag) ||
                  !mbar_wait_warp(&bars->full[s], (it / kStages) & 1u, &bars->abort_flag)) {
                report(p, bars, KCG_ST_TIMEOUT_MMA, it, s);
                ok = false;
                break;
              }
              tc_fence_after_sync();
              if (elect_one()) {
                const uint64_t a_hi = ring_a + s * (STAGE_BYTES >> 4), a_lo = a_hi + (128 * 128 >> 4);
                const uint64_t b_hi = ring_b + s * (STAGE_BYTES >> 4), b_lo = b_hi + (kBK * 128 >> 4);
                const uint32_t d = tmem_base_u + ab * kBN;
#pragma unroll
                for (int ks = 0; ks < KSTEPS; ++ks) {  // 16 values of K: 32 bytes of a row of A, 16 rows of B
                  umma_ss_pair<false>(d, a_lo + ks * 2, b_hi + ks * 128, IDESC, ks > 0 ? 1u : 0u);
                  umma_ss_pair<false>(d, a_hi + ks * 2, b_lo + ks * 128, IDESC, 1u);
                }
                umma_ss_pair_f16_scaled_d<12>(d, a_hi, b_hi, IDESC);
#pragma unroll
                for (int ks = 1; ks < KSTEPS; ++ks) umma_ss_pair<false>(d, a_hi + ks * 2, b_hi + ks * 128, IDESC, 1u);
                umma_commit_pair(smem_u32(&bars->empty[s]));
                umma_commit_pair(map_to_cta(smem_u32(&bars->empty[s]), 1u));
                umma_commit_pair(smem_u32(&bars->tmem_full[ab]));
                umma_commit_pair(map_to_cta(smem_u32(&bars->tmem_full[ab]), 1u));
              }
              __syncwarp();
            }
          }
        }
      }
    } else if (warp < FIRST_ACC_WARP) {
      Fallback::template reg_dec<IDLE_REGS>();
    } else {
      // --------------------------------------------------- accumulate + epilogue
      Fallback::template reg_inc<ACC_REGS>();
      const int q = warp & 3, half = (warp - FIRST_ACC_WARP) >> 2;
      const int epi_tid = threadIdx.x - 32 * FIRST_ACC_WARP;
      const int row_in_acc = q * 32 + lane, col_half0 = half * HALF_COLS;
      uint8_t* staging = smem + RING_BYTES + (warp - FIRST_ACC_WARP) * 32 * 128;
      uint32_t it = 0;
      bool ok = true;
      Iter units(p, unit0, unit_stride, tiles_m, tiles_n, num_kb);
      Unit w;
      while (ok && units.next(w)) {
        float acc[PIECES * 32];
#pragma unroll
        for (int i = 0; i < PIECES * 32; ++i) acc[i] = 0.f;
        // the factors of this warp's columns, PIECES of them in a lane (those past the edge are read, not used)
        float columns[PIECES];
#pragma unroll
        for (int i = 0; i < PIECES; ++i) columns[i] = __ldcg(p.columns + w.n0 + col_half0 + lane * PIECES + i);
        float next_a = 0.f, next_b[CHUNKS];
        int at_a = 0, at_b[CHUNKS];  // where the factors of the next chunk lie
        auto fetch = [&]() {     // them, one chunk ahead of its products, without the slots of far parts
          auto power = [](float factor) { return __uint_as_float(__float_as_uint(factor) & ~H2_SLOT_BITS); };
          next_a = power(__ldcg(p.scale_a + at_a));
          at_a += p.scale_lda;
#pragma unroll
          for (int i = 0; i < CHUNKS; ++i) {
            next_b[i] = power(__ldcg(p.scale_b + at_b[i]));
            at_b[i] += p.scale_ldb;
          }
        };
        Chunks ch(p, w);
        for (bool more = w.kbn > 0; more; more = far) {
          if (far && !ch.template next<true>()) break;
          const int run = far ? ch.run : w.kbn;
          const int kb0 = far ? ch.kb : w.kb0;
          at_a = kb0 * p.scale_lda + w.m0 + static_cast<int>(rank) * 128 + row_in_acc;
#pragma unroll
          for (int i = 0; i < CHUNKS; ++i) at_b[i] = kb0 * p.scale_ldb + ((w.n0 + col_half0) >> 6) + i;
          if (ch.far_a()) {
            const int slot = ch.slot_a(kb0, static_cast<int>(rank));
            at_a = slot > 0 ? p.far_scale_a + (slot - 1) * 128 + row_in_acc : p.far_zero_a;
          }
          if (ch.far_b()) {
#pragma unroll
            for (int i = 0; i < CHUNKS; ++i) {
              const int slot = ch.slot_b(kb0, (col_half0 >> 6) + i);
              at_b[i] = slot > 0 ? p.far_scale_b + slot - 1 : p.far_zero_b;
            }
          }
          fetch();
          for (int j = 0; j < run; ++j, ++it) {
            const uint32_t ab = it & 1u;
            float f[CHUNKS];
#pragma unroll
            for (int i = 0; i < CHUNKS; ++i) f[i] = next_a * next_b[i];
            if (j + 1 < run) fetch();
            // A warp whose wait ran out stops reading tensor memory but keeps walking the unit's chunks (their waits return
            // at once under the abort flag), so that all eight reach the vote below together.
            if (ok) {
              const bool got = mbar_wait(&bars->tmem_full[ab], (it >> 1) & 1u, &bars->abort_flag);
              if (!__all_sync(0xffffffffu, got)) {
                if (lane == 0) report(p, bars, KCG_ST_TIMEOUT_EPILOGUE, it, ab);
                ok = false;
              }
            }
            if (!ok) continue;
            tc_fence_after_sync();
            const uint32_t tmem_acc = tmem_base + ab * kBN + col_half0 + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll
            for (int c = 0; c < PIECES; ++c) {
              uint32_t r[32];
              tmem_ld_32x32b_x32(tmem_acc + c * 32, r);
              tmem_ld_wait();
              const float2 f2 = make_float2(f[c / 2], f[c / 2]);
#pragma unroll
              for (int i = 0; i < 32; i += 2) {  // (the factor is a power of two: its product is exact)
                float* x = acc + c * 32 + i;
                const float2 y = __ffma2_rn(make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), f2,
                                            make_float2(x[0], x[1]));
                x[0] = y.x, x[1] = y.y;
              }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster_cta(map_to_cta(smem_u32(&bars->tmem_empty[ab]), 0u));  // (the reads are complete)
          }
        }
        // The accumulating warps leave a unit as one: the store meets on a named barrier.
        ok = named_bar_all(2, NUM_EPI_THREADS, ok);
        if (!ok) break;
        const int row0 = w.m0 + static_cast<int>(rank) * 128 + q * 32;  // of this warp's rows
        bool reduce = false;
        const float4* parts = nullptr;
        if (w.nsplit > 1) {
          // A K range's partial tile, laid out [16-byte piece of a thread][thread] so that every warp store and load is 512
          // contiguous bytes; the last contributor to arrive sums them in the order of the ranges.
          float4* tile = reinterpret_cast<float4*>(p.splitk_ws + (static_cast<size_t>(w.slot - w.split) * kBM + rank * 128) * kBN) + epi_tid;
          float4* mine = tile + static_cast<size_t>(w.split) * (kBM * kBN / 4);
#pragma unroll
          for (int i = 0; i < PIECES * 8; ++i)
            __stcg(mine + i * NUM_EPI_THREADS, make_float4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]));
          const int ctr = (w.tile - p.split_first_tile) * 2 + static_cast<int>(rank);  // per CTA half
          __threadfence();
          named_bar_sync(1, NUM_EPI_THREADS);
          if (epi_tid == 0) {
            const unsigned int old = atomicAdd(&p.tile_counters[ctr], 1u);
            bars->last_flag = (old == static_cast<unsigned int>(w.nsplit - 1)) ? 1u : 0u;
            if (old == static_cast<unsigned int>(w.nsplit - 1)) p.tile_counters[ctr] = 0u;
          }
          named_bar_sync(1, NUM_EPI_THREADS);
          reduce = bars->last_flag != 0u;
          named_bar_sync(1, NUM_EPI_THREADS);  // the flag has been read
          if (!reduce) continue;
          __threadfence();
          parts = tile;
        }
        // The result, 32 columns at a time, through blocks of shared memory (16-byte units XORed with the row, the swizzle of
        // the tensor map) and TMA stores. In a CTA's last unit the operand ring is idle and holds all blocks of a warp;
        // before, a warp has one block and waits for its last store to have read it. (An SM writes about 32 bytes a cycle:
        // the 128 KB of a 256-column tile take 4100 cycles whatever is done before them; 16-byte pieces of rows straight from
        // the registers, or whole 128-byte lines after a transposition, took 9500 and 11000.)
        const bool idle_ring = w.last != 0;
#pragma unroll
        for (int c = 0; c < PIECES; ++c) {
          const int col = w.n0 + col_half0 + c * 32;
          if (row0 >= p.M || col >= p.N) break;
          float v[32];
          if (reduce) {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0.f;
#pragma unroll 1
            for (int s = 0; s < w.nsplit; ++s) {
              const float4* src = parts + static_cast<size_t>(s) * (kBM * kBN / 4) + c * 8 * NUM_EPI_THREADS;
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const float4 x = __ldcg(src + i * NUM_EPI_THREADS);
                v[4 * i] += x.x, v[4 * i + 1] += x.y, v[4 * i + 2] += x.z, v[4 * i + 3] += x.w;
              }
            }
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = acc[c * 32 + i];
          }
#pragma unroll
          for (int i = 0; i < 32; ++i)  // (a column's factor is a power of two)
            v[i] *= __shfl_sync(0xffffffffu, columns[i % PIECES], (c * 32 + i) / PIECES);
          if (p.epi_flags != 0u && row0 + lane < p.M) epi_span<float, 32>(p, v, row0 + lane, col);
          uint8_t* block = staging;
          if (idle_ring) {
            block = smem + ((warp - FIRST_ACC_WARP) * PIECES + c) * 4096;
          } else {
            if (lane == 0) tma_store_wait_read<0>();
            __syncwarp();
          }
#pragma unroll
          for (int u = 0; u < 8; ++u)
            *reinterpret_cast<float4*>(block + lane * 128 + ((u ^ (lane & 7)) << 4)) =
                make_float4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&p.tmC, block, col, row0);
            tma_store_commit();
          }
        }
      }
      if (lane == 0) tma_store_wait_read<0>();  // shared memory outlives the stores' reads
      __syncwarp();
    }
  }

  // What the split found; with H2_UNSPLIT nothing was computed.
  __device__ static __forceinline__ uint32_t multiply(const KcgGemmParams& p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    Barriers* bars = reinterpret_cast<Barriers*>(smem + RING_BYTES + STORE_BYTES);
    const int warp = threadIdx.x >> 5;

    if (threadIdx.x == 0) {
      for (int s = 0; s < kStages; ++s) {
        mbar_init(&bars->full[s], 1);
        mbar_init(&bars->empty[s], 1);
      }
      for (int a = 0; a < 2; ++a) {
        mbar_init(&bars->tmem_full[a], 1);
        mbar_init(&bars->tmem_empty[a], 16);  // one arrival per accumulating warp of each CTA
      }
      bars->abort_flag = 0u;
      bars->last_flag = 0u;
      fence_mbar_init();
      fence_proxy_async_smem();
      tma_prefetch_desc(&p.tmWs);
    }
    if (warp == 1) tmem_alloc_pair(&bars->tmem_base, TMEM_COLS);
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();  // the peer's barriers exist before anyone signals them
    tc_fence_after_sync();
    const uint32_t tmem_base = bars->tmem_base;
    const uint32_t rank = cluster_cta_rank();  // 0 = leader

    griddep_wait();  // the parts, their exponents and the words are written by the kernel before this one
    const uint32_t found = __ldcg(p.h2_words + H2_FOUND);
    const bool unsplit = (found & H2_UNSPLIT) != 0u;

    if (unsplit) {
      // (no role runs; the right to allocate tensor memory is kept for the other kernel)
    } else {
      roles(p, smem, bars, tmem_base, rank, (found & H2_FAR) != 0u);
    }

    // ------------------------------------------------------------ common exit
    __syncwarp();
    if (bars->abort_flag != 0u) {
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_before_sync();
    __syncthreads();
    __syncwarp();
    cluster_sync_all();  // the peer's shared memory and TMEM stay valid until both CTAs are done
    if (warp == 1) {
      __syncwarp();
      tc_fence_after_sync();
      tmem_dealloc_pair(tmem_base, TMEM_COLS);
    }
    if (unsplit) {  // the other kernel lays its ring over these barriers
      if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
          mbar_inval(&bars->full[s]);
          mbar_inval(&bars->empty[s]);
        }
        for (int a = 0; a < 2; ++a) {
          mbar_inval(&bars->tmem_full[a]);
          mbar_inval(&bars->tmem_empty[a]);
        }
      }
      __syncthreads();
    }
    return found;
  }

  __device__ static void run(const KcgGemmParams& p) {
    // No words: the launch had no memory for the parts and no kernel before it has written any.
    const uint32_t found = p.h2_words == nullptr ? H2_UNSPLIT : multiply(p);
    if (found & H2_UNSPLIT) Fallback::run(p);
    // Every CTA has read the word: the last one clears them all for the stream's next launch.
    if (p.h2_words != nullptr && threadIdx.x == 0) {
      if (atomicAdd(p.h2_words + H2_DONE, 1u) == gridDim.x - 1) {
        p.h2_words[H2_DONE] = 0u;
        if (found != 0u) {
          p.h2_words[H2_FOUND] = 0u;
          for (int i = H2_LINE; i < H2_WORDS; i += H2_LINE) p.h2_words[i] = 0u;
        }
      }
    }
  }
};

}  // namespace kcg
