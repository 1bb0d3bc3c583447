// fp32 GEMM on the tensor cores with fp32-level accuracy: 3xTF32 split plus
// chunked promotion of the TMEM accumulator into fp32 registers.
//
// Why two extra mechanisms on top of the plain tcgen05 pipeline:
//  * kind::tf32 reads fp32 words and ignores the low 13 mantissa bits, so
//    hi = x needs no work; splitter warps write lo = tf32_rn(x - trunc_tf32(x)) into a
//    twin of every landed stage - for A, where tensor memory has room beside the
//    accumulators, hi and lo into tensor memory instead - and each K step issues
//    lo*hi + hi*lo + hi*hi (lo*lo, ~2^-22 relative, is dropped).
//  * The tensor core adds into its fp32 accumulator with truncation, a bias that
//    grows linearly with the number of accumulated K steps (measured: 3e-5
//    normwise at K = 4096). So the MMA warp restarts a fresh accumulator every
//    kChunk K blocks, alternating between two TMEM buffers, and the epilogue
//    warps add each finished chunk into register accumulators with ordinary
//    round-to-nearest FADDs while the next chunk is being multiplied.
//
// What bounds it. Every K block crosses the shared-memory port (~128 bytes a cycle) several times: written by TMA, read
// and its lo twin written by the splitter, read by three products. With A in shared memory a CTA's half of a
// 256x256x32 pair block moves about 230 KB and takes 1770 cycles against 1536 of the tensor pipe. A through registers
// into tensor memory (hi and lo; 2 x BK columns a block) takes its lo twin and its reads by the products off the port:
// 104 KB for 256x128 (1060 cycles measured against 768 of the pipe), 140 KB for 256x192. Tiles of 256 columns, whose two
// accumulator buffers fill all 512 columns, and two-accumulator CTAs keep A in shared memory.
// What the splitter cost before it was written like this, 256x256x32 pair block: rounding by cvt.rna.tf32 15 cycles per
// warp instruction, arrivals at the leader with release at cluster scope 950 cycles, loads that waited for the stores
// before them; 2500 cycles in all. 4096^3 578 -> 488 us, 2048x4096x4096 338 -> 278, 512x11008x4096 220 -> 191,
// 640x2624x1024 34.6 -> 26.6, 6272x640x6144 252 -> 221 (graph replay in turn, B200), 1024^3 23.2 -> 20.2 per call.
// Spills (-Xptxas -v, bytes stored / loaded per thread): 256x256x32 124 / 180, 128x256x16 104 / 188, 256x192x32 24 / 44, the
// narrower tiles none.
//
// Warp roles (512 threads, 640 in the pair form with A in tensor memory; whole warpgroups so that setmaxnreg can move
// registers from the control warps to the accumulating warps):
//   WG0  warp 0 TMA producer, warp 1 MMA issuer + TMEM owner, warps 2-3 idle
//   WG1 (and WG2)  splitter (lo twin of each stage; A through registers into tensor memory)
//   the last two  accumulate + epilogue; warp w reads TMEM lane quarter w%4, column half by warpgroup;
//         MT*BN/2 fp32 register accumulators per thread
//
// Same work decomposition, raster, split-K reduction and bounded waits as
// gemm_tcgen05.cuh.
#pragma once
#include "epilogue.cuh"
#include "gemm_params.h"
#include "ptx_sm100.cuh"
#include "work_iter.cuh"

namespace kcg {

// kPair = 1 runs the same pipeline on clusters of two CTAs sharing each MMA
// (tcgen05 cta_group::2, M = 256): a CTA then holds kBM/2 rows of the tile and loads and
// splits only half of the B tile (kBN/2 columns); the leader CTA (even rank) issues the
// MMAs once the splitters of BOTH CTAs have arrived, and frees stages / publishes
// accumulators in both CTAs with one commit each. Halving the B operand traffic per SM
// lifts the shared-memory bound of the single-CTA form.
template <int kBM, int kBN, int kBK, int kStages, int kATrans, int kSplitK, int kGroup, int kChunk,
          int kPair = 0>
struct TcGemmF32x3 {
  static constexpr int kDType = KCG_DT_F32;
  static constexpr int NCTA = kPair ? 2 : 1;
  static constexpr int R = kBM / NCTA;     // rows of the tile held by one CTA
  static constexpr int BNL = kBN / NCTA;   // B columns loaded by one CTA
  static constexpr int X3 = kPair ? 2 : 1;
  static_assert(tc_config_error(kDType, R, BNL, kBK, kStages, X3) == 0,
                "config not buildable by the 3xTF32 kernel");
  static constexpr TcLayout L = make_tc_layout(kDType, R, BNL, kBK, kATrans);
  static constexpr int UMMA_K = 8;
  static constexpr int MT = R / 128;
  static constexpr int ACC_COLS = MT * kBN;
  static_assert(2 * ACC_COLS <= 512, "two accumulator buffers must fit the 512 TMEM columns");
  static_assert(kBN % 64 == 0, "each epilogue warp drains whole 32-column pieces of its column half");
  // K blocks of A in tensor memory, behind the accumulators: [hi: kBK columns][lo: kBK columns] each
  static constexpr int TA = tc_x3_tmem_a(R, BNL, kBK, kStages, X3);
  static constexpr uint32_t COL_A = 2 * ACC_COLS;
  static constexpr int TMEM_COLS = kc_pow2_ceil(2 * ACC_COLS + TA * 2 * kBK);
  static_assert(TMEM_COLS <= 512, "accumulators and A blocks must fit the 512 TMEM columns");
  static constexpr int STAGE_HI = L.stage_hi_bytes;
  // Two rings: kStages stages of TMA-landed hi operands (deep, to cover the load latency) and
  // LO_STAGES stages of their lo twins, written just in time by the splitter warps: lo stage
  // it % LO_STAGES is free again as soon as the MMAs of K block it - LO_STAGES have retired.
  static constexpr int LO_STAGES = tc_lo_stages(kStages);
  static constexpr int LO_RING = kStages * STAGE_HI;  // byte offset of the lo ring
  static constexpr int LO_BYTES = TA > 0 ? L.b_bytes : STAGE_HI;  // a lo stage: without A where that is in TMEM
  static constexpr int LO_A_BYTES = TA > 0 ? 0 : L.a_bytes;
  static constexpr int RING_BYTES = kStages * STAGE_HI + LO_STAGES * LO_BYTES;
  static constexpr int KSTEPS = kBK / UMMA_K;
  // Splitter warpgroups; two take every other K block each. One, at about 1200 cycles a block, is slower than the products
  // of a pair tile's block with A in tensor memory (768 for 128 columns).
  static constexpr int NUM_THREADS = tc_x3_threads(TA, X3);
  static constexpr int SPLIT_WGS = NUM_THREADS / 128 - 3;
  static constexpr int FIRST_ACC_WARP = 4 + 4 * SPLIT_WGS;
  static constexpr int FIRST_KS = kBN > 64 ? KSTEPS - 1 : 0;  // K steps issued before the next block is asked for
  static constexpr int NUM_SPLIT_THREADS = 128;  // of one warpgroup
  static constexpr int NUM_EPI_THREADS = 256;
  // registers of a thread after setmaxnreg; the CTA is launched with 96 each (640 threads) or 128 (512)
  static constexpr int CTL_REGS = SPLIT_WGS == 2 ? 48 : 56, SPLIT_REGS = TA > 0 && SPLIT_WGS == 1 ? 104 : 72;
  static constexpr int ACC_REGS = SPLIT_WGS == 2 ? 144 : TA > 0 ? 176 : 192;
  static_assert(CTL_REGS + SPLIT_WGS * SPLIT_REGS + 2 * ACC_REGS == (SPLIT_WGS == 2 ? 5 * 96 : 4 * 128), "register split");
  static constexpr int HALF_COLS = kBN / 2;
  static constexpr int PIECES = HALF_COLS / 32;
  static constexpr int ACC_PER_THREAD = MT * HALF_COLS;
  static_assert(ACC_PER_THREAD <= 128, "register accumulators per thread");
  static constexpr int SMEM_BYTES = tc_smem_bytes(kDType, R, BNL, kBK, kStages, X3);
  static constexpr uint32_t IDESC =
      make_instr_desc(FMT_TF32, kATrans && TA == 0 ? 1u : 0u, 1u, kPair ? 256u : 128u, kBN);

  struct Barriers {
    uint64_t full[kStages];
    uint64_t empty[kStages];
    uint64_t split_full[LO_STAGES];
    uint64_t tmem_full[2];
    uint64_t tmem_empty[2];
    uint32_t tmem_base;
    volatile uint32_t abort_flag;
    uint32_t last_flag;
  };
  static_assert(sizeof(Barriers) <= 1024, "barrier block exceeds its shared-memory slot");

  using Unit = WorkUnit;
  using Iter = WorkIter<kBM, kBN, kGroup, KCG_SERPENTINE>;  // units of this CTA (pair), in order: work_iter.cuh

  __device__ static __forceinline__ void report(const KcgGemmParams& p, Barriers* bars,
                                                uint32_t code, uint32_t d0, uint32_t d1) {
    bars->abort_flag = 1u;
    if (atomicCAS(p.status, 0u, code) == 0u) {
      p.status[1] = blockIdx.x;
      p.status[2] = d0;
      p.status[3] = d1;
    }
  }

  template <int REGS>
  __device__ static __forceinline__ void reg_dec() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS));
  }
  template <int REGS>
  __device__ static __forceinline__ void reg_inc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS));
  }

  __device__ static void run(const KcgGemmParams& p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    Barriers* bars = reinterpret_cast<Barriers*>(smem + RING_BYTES);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int tiles_m = (p.M + kBM - 1) / kBM;
    const int tiles_n = (p.N + kBN - 1) / kBN;
    const int num_kb = (p.K + kBK - 1) / kBK;
    const int first_split = p.split_first_tile;

    if (threadIdx.x == 0) {
      for (int s = 0; s < kStages; ++s) {
        mbar_init(&bars->full[s], 1);
        mbar_init(&bars->empty[s], 1);
      }
      for (int s = 0; s < LO_STAGES; ++s)
        mbar_init(&bars->split_full[s], 4 * NCTA);  // one arrival per splitter warp of each CTA
      for (int a = 0; a < 2; ++a) {
        mbar_init(&bars->tmem_full[a], 1);
        mbar_init(&bars->tmem_empty[a], 8 * NCTA);  // one arrival per accumulating warp of each CTA
      }
      bars->abort_flag = 0u;
      bars->last_flag = 0u;
      fence_mbar_init();
      fence_proxy_async_smem();
    }
    if (warp == 1) {
      if constexpr (kPair) {
        tmem_alloc_pair(&bars->tmem_base, TMEM_COLS);
        tmem_relinquish_pair();
      } else {
        tmem_alloc(&bars->tmem_base, TMEM_COLS);
        tmem_relinquish();
      }
    }
    tc_fence_before_sync();
    __syncthreads();
    if constexpr (kPair) cluster_sync_all();  // the peer's barriers exist before anyone signals them
    tc_fence_after_sync();
    const uint32_t tmem_base = bars->tmem_base;
    const uint32_t rank = kPair ? cluster_cta_rank() : 0u;  // 0 = leader
    const int unit0 = kPair ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x);
    const int unit_stride = kPair ? static_cast<int>(gridDim.x >> 1) : static_cast<int>(gridDim.x);
    const int row_base = static_cast<int>(rank) * R;     // this CTA's first row inside the tile
    const int bcol_base = static_cast<int>(rank) * BNL;  // this CTA's first B column inside the tile

    if (warp < 4) {
      reg_dec<CTL_REGS>();
      if (warp == 0 && lane == 0) {
        // ---------------------------------------------------------- producer
        tma_prefetch_desc(&p.tmA);
        tma_prefetch_desc(&p.tmB);
        griddep_wait();  // the kernel before this one in the stream may have written A or B
        uint32_t it = 0;
        bool ok = true;
        Iter units(p, unit0, unit_stride, tiles_m, tiles_n, num_kb);
        Unit w;
        while (ok && units.next(w)) {
          for (int kb = 0; kb < w.kbn; ++kb, ++it) {
            const uint32_t s = it % kStages;
            const uint32_t ph = (it / kStages) & 1u;
            if (!mbar_wait(&bars->empty[s], ph ^ 1u, &bars->abort_flag)) {
              report(p, bars, KCG_ST_TIMEOUT_PRODUCER, it, s);
              ok = false;
              break;
            }
            uint8_t* sa = smem + s * STAGE_HI;
            uint8_t* sb = sa + L.a_bytes;
            mbar_expect_tx(&bars->full[s], static_cast<uint32_t>(STAGE_HI));
            const int k0 = (w.kb0 + kb) * kBK;
#pragma unroll
            for (int j = 0; j < L.a_boxes; ++j) {
              if constexpr (kATrans) {  // K x M storage: the batch selects K rows, M counts inside it
                tma_load_2d(sa + j * L.a_box_bytes, &p.tmA, &bars->full[s], w.mcol + row_base + j * L.atom,
                            k0 + w.kofs);
              } else {
                tma_load_2d(sa + j * L.a_box_bytes, &p.tmA, &bars->full[s],
                            k0 + j * L.a_box_inner, w.m0 + row_base);
              }
            }
#pragma unroll
            for (int j = 0; j < L.b_boxes; ++j) {
              tma_load_2d(sb + j * L.b_box_bytes, &p.tmB, &bars->full[s], w.n0 + bcol_base + j * L.atom,
                          k0 + w.kofs);
            }
          }
        }
        griddep_launch_dependents();  // every load is issued: the stream's next kernel may be brought in
      } else if (warp == 1 && rank == 0u) {
        // ---------------------------- MMA issuer (in a pair: the leader CTA only)
        // whole warp, one elected lane per batch of instructions (see elect_one)
        const uint32_t tmem_base_u = __shfl_sync(0xffffffffu, tmem_base, 0);
        uint32_t it = 0, chunk_it = 0;
        bool ok = true, ready = false;  // ready: block `it` has been waited for
        // the lo twin is written after the hi stage has landed (in both CTAs of a pair)
        auto wait_split = [&](uint32_t i) -> bool {
          const bool got = mbar_wait_warp(&bars->split_full[i % LO_STAGES], (i / LO_STAGES) & 1u, &bars->abort_flag);
          if (!got) report(p, bars, KCG_ST_TIMEOUT_MMA, i, i % kStages);
          return got;
        };
        Iter units(p, unit0, unit_stride, tiles_m, tiles_n, num_kb);
        Unit w;
        while (ok && units.next(w)) {
          for (int kb0 = 0; kb0 < w.kbn && ok; kb0 += kChunk, ++chunk_it) {
            const uint32_t ab = chunk_it & 1u;
            const uint32_t aph = (chunk_it >> 1) & 1u;
            if (!mbar_wait_warp(&bars->tmem_empty[ab], aph ^ 1u, &bars->abort_flag)) {
              report(p, bars, KCG_ST_TIMEOUT_MMA, 0x100u + ab, chunk_it);
              ok = false;
              break;
            }
            tc_fence_after_sync();
            const uint32_t tmem_acc = tmem_base_u + ab * ACC_COLS;
            const int kb1 = (kb0 + kChunk < w.kbn) ? kb0 + kChunk : w.kbn;
            for (int kb = kb0; kb < kb1; ++kb, ++it) {
              if (!ready && !(ok = wait_split(it))) break;
              ready = false;
              tc_fence_after_sync();
              const uint32_t s = it % kStages;
              const uint32_t sl = it % LO_STAGES;
              const uint32_t sa = smem_u32(smem + s * STAGE_HI);
              const uint32_t sb = sa + L.a_bytes;
              const uint32_t sa_lo = smem_u32(smem + LO_RING + sl * LO_BYTES);
              const uint32_t sb_lo = sa_lo + LO_A_BYTES;
              const uint32_t ta = tmem_base_u + COL_A + it % (TA > 0 ? TA : 1) * 2 * kBK;
              auto issue = [&](int ks) {  // the products of one K step
                const uint32_t b_off = ks * UMMA_K * 128;
                const uint32_t first = (kb > kb0 || ks > 0) ? 1u : 0u;
                const uint64_t bdesc = make_smem_desc(sb + b_off, L.b_lbo, L.b_sbo, L.b_desc_swizzle);
                const uint64_t bdesc_lo = make_smem_desc(sb_lo + b_off, L.b_lbo, L.b_sbo, L.b_desc_swizzle);
                if constexpr (TA > 0) {
                  umma_ts<true, NCTA>(tmem_acc, ta + kBK + ks * UMMA_K, bdesc, IDESC, first);
                  umma_ts<true, NCTA>(tmem_acc, ta + ks * UMMA_K, bdesc_lo, IDESC, 1u);
                  umma_ts<true, NCTA>(tmem_acc, ta + ks * UMMA_K, bdesc, IDESC, 1u);
                } else {
                  uint32_t a_off;
                  if constexpr (kATrans) {
                    a_off = ks * UMMA_K * 128;
                  } else {
                    constexpr int swb = (kBK * 4 < 128) ? kBK * 4 : 128;
                    a_off = ((ks * 32) / swb) * L.a_box_bytes + ((ks * 32) % swb);
                  }
#pragma unroll
                  for (int t = 0; t < MT; ++t) {
                    const uint32_t a_t = kATrans ? t * (128 / L.atom) * L.a_box_bytes
                                                 : t * 128 * (L.a_box_bytes / R);
                    const uint64_t adesc =
                        make_smem_desc(sa + a_t + a_off, L.a_lbo, L.a_sbo, L.a_desc_swizzle);
                    const uint64_t adesc_lo = make_smem_desc(sa_lo + a_t + a_off, L.a_lbo,
                                                             L.a_sbo, L.a_desc_swizzle);
                    const uint32_t d = tmem_acc + t * kBN;
                    if constexpr (kPair) {
                      umma_ss_pair<true>(d, adesc_lo, bdesc, IDESC, first);
                      umma_ss_pair<true>(d, adesc, bdesc_lo, IDESC, 1u);
                      umma_ss_pair<true>(d, adesc, bdesc, IDESC, 1u);
                    } else {
                      umma_ss<true>(d, adesc_lo, bdesc, IDESC, first);
                      umma_ss<true>(d, adesc, bdesc_lo, IDESC, 1u);
                      umma_ss<true>(d, adesc, bdesc, IDESC, 1u);
                    }
                  }
                }
              };
              if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < FIRST_KS; ++ks) issue(ks);
              }
              __syncwarp();
              // Is the next block there? Asked here, while the tensor pipe still has products to run, and not after the
              // last of them: where loads and splitter keep ahead, the question costs the pipe nothing (pair tiles 3 to
              // 5 %). Blocks of 64 columns are through before it pays: 128x64 tiles are 4 % faster without it.
              if (FIRST_KS > 0 && kb + 1 < w.kbn)
                ready = mbar_test_warp(&bars->split_full[(it + 1) % LO_STAGES], ((it + 1) / LO_STAGES) & 1u);
              if (elect_one()) {
#pragma unroll
                for (int ks = FIRST_KS; ks < KSTEPS; ++ks) issue(ks);
                // the hi stage, and with it the lo stage of this K block, is free in both CTAs
                // once these MMAs retire
                if constexpr (kPair) {
                  umma_commit_pair(smem_u32(&bars->empty[s]));
                  umma_commit_pair(map_to_cta(smem_u32(&bars->empty[s]), 1u));
                } else {
                  umma_commit(&bars->empty[s]);
                }
              }
              __syncwarp();
            }
            if (ok && elect_one()) {
              if constexpr (kPair) {
                umma_commit_pair(smem_u32(&bars->tmem_full[ab]));
                umma_commit_pair(map_to_cta(smem_u32(&bars->tmem_full[ab]), 1u));
              } else {
                umma_commit(&bars->tmem_full[ab]);
              }
            }
            __syncwarp();
          }
        }
      }
    } else if (warp < FIRST_ACC_WARP) {
      // --------------------------------------------------------------- splitter
      reg_dec<SPLIT_REGS>();
      const int stid = threadIdx.x & 127;
      const uint32_t turn = static_cast<uint32_t>(warp >> 2) - 1u;  // of this warpgroup among the K blocks
      uint32_t it = 0;
      bool ok = true;
      Iter units(p, unit0, unit_stride, tiles_m, tiles_n, num_kb);
      Unit w;
      while (ok && units.next(w)) {
        for (int kb = 0; kb < w.kbn; ++kb, ++it) {
          if (it % SPLIT_WGS != turn) continue;
          const uint32_t s = it % kStages;
          const uint32_t ph = (it / kStages) & 1u;
          const uint32_t sl = it % LO_STAGES;
          // lo stage sl was last read by the MMAs of K block it - LO_STAGES; their retirement is
          // what completes that block's phase of its hi stage's `empty` barrier. The MMA warp
          // never runs ahead of this loop, so that barrier cannot be a whole phase further on.
          bool got = true;
          // (with rings of equal depth the landed hi stage already implies it)
          if (LO_STAGES < kStages && it >= static_cast<uint32_t>(LO_STAGES)) {
            const uint32_t prev = it - LO_STAGES;
            got = mbar_wait(&bars->empty[prev % kStages], (prev / kStages) & 1u, &bars->abort_flag);
          }
          if (got) got = mbar_wait(&bars->full[s], ph, &bars->abort_flag);
          got = __all_sync(0xffffffffu, got);
          constexpr int FIRST = TA > 0 ? L.a_bytes : 0;  // the part of the stage that gets a twin in shared memory
          constexpr int PER_THREAD = (STAGE_HI - FIRST) / 16 / NUM_SPLIT_THREADS;
          constexpr int BATCH = PER_THREAD % 8 == 0 ? 8 : PER_THREAD % 6 == 0 ? 6 : PER_THREAD % 4 == 0 ? 4 : 1;
          static_assert(PER_THREAD % BATCH == 0 && (STAGE_HI - FIRST) % (16 * NUM_SPLIT_THREADS) == 0, "whole batches");
          if (got) {
            const uint4* hi = reinterpret_cast<const uint4*>(smem + s * STAGE_HI + FIRST) + stid;
            uint4* lo = reinterpret_cast<uint4*>(smem + LO_RING + sl * LO_BYTES) + stid;
            // (a batch's loads are all in flight before its first store: the compiler may not move a load above a store)
#pragma unroll
            for (int b = 0; b < PER_THREAD; b += BATCH) {
              uint4 x[BATCH];
#pragma unroll
              for (int u = 0; u < BATCH; ++u) x[u] = hi[(b + u) * NUM_SPLIT_THREADS];
#pragma unroll
              for (int u = 0; u < BATCH; ++u)
                lo[(b + u) * NUM_SPLIT_THREADS] =
                    make_uint4(lo_part(x[u].x), lo_part(x[u].y), lo_part(x[u].z), lo_part(x[u].w));
            }
            fence_proxy_async_smem();
          }
          if constexpr (TA > 0) {
            uint32_t a[kBK];
            if (got) load_a_row(smem + s * STAGE_HI, (warp & 3) * 32 + lane, a);
            // TMEM block it % TA was last read by the MMAs of K block it - TA (as above, their stage's `empty`). The
            // stores to tensor memory are made by whole warps, which therefore leave the loop as one.
            if (got && TA < kStages && it >= static_cast<uint32_t>(TA)) {
              const uint32_t prev = it - TA;
              got = mbar_wait(&bars->empty[prev % kStages], (prev / kStages) & 1u, &bars->abort_flag);
            }
            got = __all_sync(0xffffffffu, got);
            if (got) {
              tc_fence_after_sync();
              const uint32_t ta =
                  tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + COL_A + (it % TA) * 2 * kBK;
#pragma unroll
              for (int k0 = 0; k0 < kBK; k0 += 16) {
                uint32_t h[16], l[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                  h[i] = a[k0 + i];
                  l[i] = lo_part(a[k0 + i]);
                }
                tmem_st_32x32b_x16(ta + k0, h);
                tmem_st_32x32b_x16(ta + kBK + k0, l);
              }
              tmem_st_wait();
              tc_fence_before_sync();
            }
          }
          if (!got) {
            if (lane == 0) report(p, bars, KCG_ST_TIMEOUT_SPLITTER, it, s);
            ok = false;
            break;
          }
          __syncwarp();
          if (lane == 0) {
            if constexpr (kPair) {
              mbar_arrive_cluster_cta(map_to_cta(smem_u32(&bars->split_full[sl]), 0u));
            } else {
              mbar_arrive(&bars->split_full[sl]);
            }
          }
        }
      }
    } else {
      // --------------------------------------------------- accumulate + epilogue
      reg_inc<ACC_REGS>();
      griddep_wait();  // C, the workspace and the counters may still be in use by the kernel before
      const int q = warp & 3;
      const int half = (warp - FIRST_ACC_WARP) >> 2;
      const int epi_tid = threadIdx.x - 32 * FIRST_ACC_WARP;
      const int row_in_acc = q * 32 + lane;
      const int col_half0 = half * HALF_COLS;
      float* Cout = reinterpret_cast<float*>(p.C);
      uint32_t chunk_it = 0;
      bool ok = true;
      Iter units(p, unit0, unit_stride, tiles_m, tiles_n, num_kb);
      Unit w;
      while (ok && units.next(w)) {
        float acc[ACC_PER_THREAD];
#pragma unroll
        for (int i = 0; i < ACC_PER_THREAD; ++i) acc[i] = 0.f;
        for (int kb0 = 0; kb0 < w.kbn; kb0 += kChunk, ++chunk_it) {
          const uint32_t ab = chunk_it & 1u;
          const uint32_t aph = (chunk_it >> 1) & 1u;
          // A warp whose wait ran out stops reading TMEM but keeps walking the unit's chunks (their
          // waits return at once under the abort flag), so that all eight accumulating warps reach
          // the vote below together.
          if (ok) {
            const bool got = mbar_wait(&bars->tmem_full[ab], aph, &bars->abort_flag);
            if (!__all_sync(0xffffffffu, got)) {
              if (lane == 0) report(p, bars, KCG_ST_TIMEOUT_EPILOGUE, chunk_it, ab);
              ok = false;
            }
          }
          if (!ok) continue;
          tc_fence_after_sync();
          const uint32_t tmem_acc =
              tmem_base + ab * ACC_COLS + col_half0 + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll
          for (int t = 0; t < MT; ++t) {
#pragma unroll
            for (int c = 0; c < PIECES; ++c) {
              uint32_t r[32];
              tmem_ld_32x32b_x32(tmem_acc + t * kBN + c * 32, r);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i)
                acc[(t * PIECES + c) * 32 + i] += __uint_as_float(r[i]);
            }
          }
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) {
            if constexpr (kPair) {
              mbar_arrive_cluster_cta(map_to_cta(smem_u32(&bars->tmem_empty[ab]), 0u));  // (the reads above are complete)
            } else {
              mbar_arrive(&bars->tmem_empty[ab]);
            }
          }
        }
        // The accumulating warps leave a unit as one (named barrier 2 ANDs their outcomes): the
        // store path below meets on named barrier 1, where a warp that had given up alone would
        // leave the others waiting for its threads for ever.
        ok = named_bar_all(2, NUM_EPI_THREADS, ok);
        if (!ok) break;
        // ---- tile (or split partial) complete in registers: store. A launch with a fused
        // epilogue sends whole-K tiles through the workspace too and applies the epilogue in
        // the reduction loop below, where the accumulators are dead: with all of them live
        // there are no registers left for the bias / C operands.
        const bool via_ws = w.nsplit > 1 || p.epi_flags != 0u;
        // the tile's first contributor's, or the one that all whole tiles of this CTA (pair) take in turn
        const int slot0 = w.nsplit > 1 ? w.slot - w.split : p.whole_slot0 + unit0;
#pragma unroll
        for (int t = 0; t < MT; ++t) {
          const int row = w.m0 + row_base + t * 128 + row_in_acc;
#pragma unroll
          for (int c = 0; c < PIECES; ++c) {
            const int col = w.n0 + col_half0 + c * 32;
            if (row < p.M && col < p.N) {
              // A partial is private to this kernel, so it is not stored as a matrix: the CTA's
              // R x kBN floats are laid out [16-byte piece of a thread][thread], which makes every
              // warp store (and the reducer's loads) 512 contiguous bytes. Row-major partials, 16
              // bytes per lane at a 1 KB stride, made L2 merge every sector.
              float4* d4 = via_ws ? reinterpret_cast<float4*>(p.splitk_ws +
                                                             (static_cast<size_t>(slot0 + w.split) * kBM + row_base) * kBN) +
                                        (t * PIECES + c) * 8 * NUM_EPI_THREADS + epi_tid
                                  : reinterpret_cast<float4*>(Cout + static_cast<size_t>(row) * p.ldc + col);
              const int step = via_ws ? NUM_EPI_THREADS : 1;
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const int b = (t * PIECES + c) * 32 + 4 * i;
                d4[i * step] = make_float4(acc[b], acc[b + 1], acc[b + 2], acc[b + 3]);
              }
            }
          }
        }
        if (via_ws) {
          bool reduce_here = true;  // a one-way split reads back what this same thread just wrote
          if (w.nsplit > 1) {
            const int ctr = (w.tile - first_split) * NCTA + static_cast<int>(rank);  // per CTA half
            __threadfence();
            named_bar_sync(1, NUM_EPI_THREADS);
            if (epi_tid == 0) {
              const unsigned int old = atomicAdd(&p.tile_counters[ctr], 1u);
              bars->last_flag = (old == static_cast<unsigned int>(w.nsplit - 1)) ? 1u : 0u;
              if (old == static_cast<unsigned int>(w.nsplit - 1)) p.tile_counters[ctr] = 0u;
            }
            named_bar_sync(1, NUM_EPI_THREADS);
            reduce_here = bars->last_flag != 0u;
          }
          if (reduce_here) {
            __threadfence();
            // One partial at a time: the accumulating warps have no registers to spare for
            // deeper prefetch (more loads in flight made ptxas spill inside the main loop).
#pragma unroll 1
            for (int t = 0; t < MT; ++t) {
              const int row = w.m0 + row_base + t * 128 + row_in_acc;
              if (row >= p.M) continue;
#pragma unroll 1
              for (int c = 0; c < PIECES; ++c) {
                const int col = w.n0 + col_half0 + c * 32;
                if (col >= p.N) continue;
                float v[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = 0.f;
#pragma unroll 1
                for (int s = 0; s < w.nsplit; ++s) {
                  const float4* src =
                      reinterpret_cast<const float4*>(
                          p.splitk_ws + (static_cast<size_t>(slot0 + s) * kBM + row_base) * kBN) +
                      (t * PIECES + c) * 8 * NUM_EPI_THREADS + epi_tid;
#pragma unroll
                  for (int i = 0; i < 8; ++i) {
                    const float4 x = __ldcg(src + i * NUM_EPI_THREADS);
                    v[4 * i] += x.x;
                    v[4 * i + 1] += x.y;
                    v[4 * i + 2] += x.z;
                    v[4 * i + 3] += x.w;
                  }
                }
                if (p.epi_flags != 0u) epi_span<float, 32>(p, v, row, col);
                float4* d4 = reinterpret_cast<float4*>(Cout + static_cast<size_t>(row) * p.ldc + col);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                  d4[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
              }
            }
          }
          named_bar_sync(1, NUM_EPI_THREADS);
        }
      }
    }

    // ------------------------------------------------------------ common exit
    // The producer and MMA roles run in one lane; the other lanes of those warps come straight here.
    // Reconverge every warp first: the block-wide barrier below must be executed by whole warps.
    __syncwarp();
    if (bars->abort_flag != 0u) {
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_before_sync();
    __syncthreads();
    if constexpr (kPair) {
      __syncwarp();
      cluster_sync_all();  // the peer's shared memory and TMEM stay valid until both CTAs are done
    }
    if (warp == 1) {
      __syncwarp();
      tc_fence_after_sync();
      if constexpr (kPair) {
        tmem_dealloc_pair(tmem_base, TMEM_COLS);
      } else {
        tmem_dealloc(tmem_base, TMEM_COLS);
      }
    }
  }

  // One thread's row of a landed A block.
  __device__ static __forceinline__ void load_a_row(const uint8_t* a, int row, uint32_t (&x)[kBK]) {
    if constexpr (kATrans) {
      // boxes of 32 rows x kBK values of K, 128 bytes per value; 32-byte units XORed with K mod 4
      const uint8_t* col = a + (row >> 5) * L.a_box_bytes + (row & 7) * 4;
#pragma unroll
      for (int k = 0; k < kBK; ++k)
        x[k] = *reinterpret_cast<const uint32_t*>(col + k * 128 + ((((row >> 3) & 3) ^ (k & 3)) << 5));
    } else {
      // boxes of `swb` bytes of K x R rows; 16-byte units XORed with the row's number within the swizzle's repeat
      constexpr int swb = (kBK * 4 < 128) ? kBK * 4 : 128;
      const int flip = (row * swb / 128) & (swb / 16 - 1);
#pragma unroll
      for (int u = 0; u < kBK / 4; ++u) {
        const uint8_t* line = a + (u * 16 / swb) * L.a_box_bytes + row * swb;
        const uint4 v = *reinterpret_cast<const uint4*>(line + (((u % (swb / 16)) ^ flip) << 4));
        x[4 * u] = v.x;
        x[4 * u + 1] = v.y;
        x[4 * u + 2] = v.z;
        x[4 * u + 3] = v.w;
      }
    }
  }

  // tf32_rna(x - trunc_tf32(x)) on raw bits, in its upper 19 bits: half of the last bit kept is added and kind::tf32
  // ignores the rest. The subtraction is exact in fp32; x * 0 turns the lo part of an infinite or NaN x into NaN (the
  // integer sum would wrap). cvt.rna.tf32.f32 - same bits - takes 15 cycles per warp instruction.
  __device__ static __forceinline__ uint32_t lo_part(uint32_t xbits) {
    const float x = __uint_as_float(xbits);
    const float hi = __uint_as_float(xbits & 0xffffe000u);
    return __float_as_uint(__fmaf_rn(x, 0.f, __uint_as_float(__float_as_uint(x - hi) + 0x1000u)));
  }
};

}  // namespace kcg
