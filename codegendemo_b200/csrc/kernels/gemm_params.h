// Kernel-argument block and compile-time layout rules shared by the device
// kernels and the host shim. Plain C++ (no torch, no CUDA runtime types beyond
// CUtensorMap), so the host library and every JIT-compiled cubin agree on the
// byte layout of one `__grid_constant__` parameter.
#pragma once
#include <cuda.h>
#include <stdint.h>

// DATATYPE_* values of the tuning config. 2/4/8 are the reference's
// EnumKernelDType byte-size codes (Runtime/python/kcg/Utils.py:198-203);
// 62 is this library's bfloat16 (62 % 30 == 2 bytes keeps the reference's
// sizeof() rule, Utils.py:219-221).
#define KCG_DT_F16 2
#define KCG_DT_F32 4
#define KCG_DT_F64 8
#define KCG_DT_BF16 62

// KERNEL_VARIANT
#define KCG_VARIANT_AUTO 0
#define KCG_VARIANT_SIMT 1     // FFMA register-tiled kernel (fp32)
#define KCG_VARIANT_TCGEN05 2  // TMA + tcgen05/TMEM kernel (bf16, fp16, fp32 as 3xTF32)
#define KCG_VARIANT_TF32X1 3   // tcgen05 single-pass TF32 (fp32 in, reduced accuracy; comparison only)

#define KCG_VARIANT_TCGEN05_PAIR 4  // tcgen05 cta_group::2 on clusters of two CTAs (fp16 / bf16)
// K split over a thread-block cluster of LOCAL_SPLIT_U CTAs, partial tiles reduced through
// distributed shared memory (fp16 / bf16, 128-row tiles, or 256-row tiles on CTA pairs): no workspace, no counters
#define KCG_VARIANT_TCGEN05_CLUSTERK 5

// fp32 through two fp16 parts per value, split in memory before the product (CTA pairs; 3xTF32 where the parts cannot
// carry a value)
#define KCG_VARIANT_F32H2 6

#define KCG_MAX_PEERS 7  // other GPUs of one NVSwitch domain of eight

// epi_flags bits
#define KCG_EPI_SCALE 1u  // alpha / beta differ from 1 / 0
#define KCG_EPI_BIAS 2u   // add bias[col]
#define KCG_EPI_RELU 4u   // max(x, 0) last

// Device status word values (status[0]); 0 = ok.
#define KCG_ST_OK 0u
#define KCG_ST_TIMEOUT_PRODUCER 1u
#define KCG_ST_TIMEOUT_MMA 2u
#define KCG_ST_TIMEOUT_EPILOGUE 3u
#define KCG_ST_TIMEOUT_SPLITTER 4u
#define KCG_ST_BAD_SHAPE 5u
#define KCG_ST_TIMEOUT_PUSHER 6u

struct alignas(64) KcgGemmParams {
  CUtensorMap tmA;  // tcgen05 variants: tiled map of A (or of A^T when IS_ATRANS=1)
  CUtensorMap tmB;  // tiled map of B (K x N row-major)
  CUtensorMap tmC;  // C as 32-row x 128-byte boxes (128B swizzle): the TMA-store epilogue
  CUtensorMap tmWs;  // K-split workspace as one tall fp32 matrix of BN columns, 32 x 32 boxes
  const void* A;
  const void* B;
  void* C;
  float* splitk_ws;             // fp32 partial tiles, [slot][BM][BN]; slot = unit - split_first_tile
  unsigned int* tile_counters;  // one per split tile (tile - split_first_tile), zero between launches
  unsigned int* status;         // 4 words: code, blockIdx.x, detail0, detail1
  int M, N, K;
  int lda, ldb, ldc;  // leading dimensions in elements (row-major storage)
  // K splitting over CTAs: tiles [0, split_first_tile) are computed whole, every tile from
  // split_first_tile on is cut into split_factor K ranges. LOCAL_SPLIT_U = S splits every tile
  // (first = 0, factor = S); with LOCAL_SPLIT_U = 1 the launcher splits only the tiles of the last,
  // partially filled wave of the persistent grid (or nothing: factor = 1).
  int split_first_tile, split_factor;
  // Stream-K over the tiles from split_first_tile on (instead of the even split) when > 0: their
  // K blocks, laid end to end, are cut into one contiguous range of sk_per blocks per CTA (pair);
  // the grid then has exactly as many CTAs (pairs) as there are ranges (work_iter.cuh).
  int sk_per;
  // Batched product when > 0: M counts the rows of all batches (A and C stacked by rows), K is one
  // batch's, B holds the batches' K x N matrices one under the other (an A stored K x M likewise),
  // and batch_rows is the M of one batch, a multiple of the tile height.
  int batch_rows;
  // Order of a CTA's units when a launch has both whole tiles and K-split tiles: 1 = the split
  // units (even split or stream-K ranges) come first and the whole tiles after them, so that the
  // partial tiles are written, summed and stored by the epilogue warps while the whole tiles' main
  // loops run, and a CTA ends with an ordinary tile; 0 = whole tiles first, split units last.
  int split_units_first;
  // Fused epilogue, in force when epi_flags != 0: D = act(alpha * (A.B) + beta * C + bias[col]),
  // computed in fp32 before the rounding to C's type. beta * C reads C in place (skipped when
  // beta == 0, so C may then hold anything); bias has N values of C's type.
  float alpha, beta;
  const void* bias;
  unsigned int epi_flags;  // KCG_EPI_*
  // fp32 kernels: workspace slots of whole tiles that go through the workspace (fused epilogue), one per CTA (pair) from
  // this on.
  int whole_slot0;
  // KERNEL_VARIANT 6 (gemm_tcgen05_f32h2.cuh): the factors of the parts' products, [K block][rows of A] and [K block][64
  // columns of B] with these pitches, those of the finished columns, and the words (H2_WORDS below); no words: 3xTF32
  // throughout. tmWs maps the parts, those of B from row parts_b_row on.
  const float* scale_a;
  const float* scale_b;
  const float* columns;
  int scale_lda, scale_ldb, parts_b_row;
  unsigned int* h2_words;
  // Fused all-gather of an M-sharded product: besides C, every finished tile is also written
  // to the same rows / columns of n_peers more matrices with C's pitch — this rank's slab inside
  // the full C of every other GPU, mapped into this process (coalesced 16-byte stores over NVLink
  // by the kernel's push warps, or by the reducer of a K-split tile; no remote loads, no multicast,
  // no flags between GPUs: the data is in place when every rank's kernel has completed).
  int n_peers;
  void* peerC[KCG_MAX_PEERS];
  // KERNEL_VARIANT 6: rows of tmWs; far parts, in slots of a chunk each: their first rows there; their factors, [slot][128 rows of
  // A] and [slot], as places from scale_a and from scale_b on, and the place of a zero from each.
  int parts_rows, far_a_row, far_b_row, far_scale_a, far_scale_b, far_zero_a, far_zero_b;
};

namespace kcg {

constexpr int kc_min(int a, int b) { return a < b ? a : b; }
constexpr int kc_pow2_ceil(int v) {
  int p = 32;
  while (p < v) p <<= 1;
  return p;
}

// Shared-memory / TMA layout of one pipeline stage of the tcgen05 kernels.
// Host (tensor-map construction) and device (descriptors) both derive it from
// the same five config values.
struct TcLayout {
  int eb;          // element bytes
  int umma_k;      // K extent of one MMA instruction
  int atom;        // elements per 128-byte swizzle row
  // A operand
  int a_box_inner, a_box_outer;  // TMA box in elements {contiguous, strided}
  int a_boxes, a_box_bytes, a_bytes;
  int a_tma_swizzle;   // CUtensorMapSwizzle value
  int a_desc_swizzle;  // UMMA descriptor layout type
  int a_lbo, a_sbo;
  // B operand (always MN-major: K x N row-major)
  int b_box_inner, b_box_outer;
  int b_boxes, b_box_bytes, b_bytes;
  int b_tma_swizzle, b_desc_swizzle;
  int b_lbo, b_sbo;
  int stage_hi_bytes;  // one copy of A+B
};

// `btrans` = B is stored N x K row-major (the "NT" product C = A * Bt^T): its tile is then a K-major
// operand laid out exactly like a K-major A tile; 16-bit types only.
constexpr TcLayout make_tc_layout(int dtype, int BM, int BN, int BK, int atrans, int btrans = 0) {
  TcLayout L{};
  L.eb = (dtype == KCG_DT_F32) ? 4 : 2;
  L.umma_k = 32 / L.eb;
  L.atom = 128 / L.eb;
  // MN-major operands: boxes of {atom elements along MN, BK rows of K}.
  // 16-bit: 128B swizzle of 16B units, 8-row repeat; 32-bit: 128B swizzle of
  // 32B units, 4-row repeat (the only MN-major form kind::tf32 accepts).
  const int mn_tma = (L.eb == 4) ? 4 /*128B_ATOM_32B*/ : 3 /*128B*/;
  const int mn_desc = (L.eb == 4) ? 1 : 2;
  const int mn_sbo = (L.eb == 4) ? 512 : 1024;
  if (atrans) {
    L.a_box_inner = L.atom;
    L.a_box_outer = BK;
    L.a_boxes = BM / L.atom;
    L.a_box_bytes = BK * 128;
    L.a_tma_swizzle = mn_tma;
    L.a_desc_swizzle = mn_desc;
    L.a_lbo = BK * 128;
    L.a_sbo = mn_sbo;
  } else {
    const int swb = kc_min(128, BK * L.eb);  // swizzle span = bytes of one K row
    L.a_box_inner = swb / L.eb;
    L.a_box_outer = BM;
    L.a_boxes = (BK * L.eb) / swb;
    L.a_box_bytes = BM * swb;
    L.a_tma_swizzle = (swb == 128) ? 3 : (swb == 64) ? 2 : 1;
    L.a_desc_swizzle = (swb == 128) ? 2 : (swb == 64) ? 4 : 6;
    L.a_lbo = 16;
    L.a_sbo = 8 * swb;
  }
  L.a_bytes = BM * BK * L.eb;
  L.b_box_inner = L.atom;
  L.b_box_outer = BK;
  L.b_boxes = BN / L.atom;
  L.b_box_bytes = BK * 128;
  L.b_bytes = BN * BK * L.eb;
  L.b_tma_swizzle = mn_tma;
  L.b_desc_swizzle = mn_desc;
  L.b_lbo = BK * 128;
  L.b_sbo = mn_sbo;
  if (btrans) {
    const int swb = kc_min(128, BK * L.eb);
    L.b_box_inner = swb / L.eb;
    L.b_box_outer = BN;
    L.b_boxes = (BK * L.eb) / swb;
    L.b_box_bytes = BN * swb;
    L.b_tma_swizzle = (swb == 128) ? 3 : (swb == 64) ? 2 : 1;
    L.b_desc_swizzle = (swb == 128) ? 2 : (swb == 64) ? 4 : 6;
    L.b_lbo = 16;
    L.b_sbo = 8 * swb;
  }
  L.stage_hi_bytes = L.a_bytes + L.b_bytes;
  return L;
}

// Epilogue staging of the single-pass kernel: each of its four epilogue warps owns two
// 32-row x 128-byte buffers from which C leaves through TMA stores. The 3xTF32 kernel
// stores from registers and has none. `x3` only has a meaning for fp32 data: 16-bit data always
// runs on the single-pass kernel.
constexpr int tc_staging_bytes(int dtype, int x3) {
  return (dtype == KCG_DT_F32 && x3) ? 0 : 4 * 2 * 32 * 128;
}

// 3xTF32 kernel: depth of the ring of lo twins beside `stages` TMA-fed hi stages. The kernel
// supports a shorter lo ring, but the splitter has to run several K blocks ahead of the MMAs
// (hand-offs plus two passes over a stage of shared memory), which only equally deep rings give:
// every shorter lo ring measured slower. So the lo ring is as deep as the hi ring.
constexpr int tc_lo_stages(int stages) { return stages; }

// `x3` of the rules below: 0 = single-pass kernel, 1 = 3xTF32 kernel, 2 = 3xTF32 on CTA pairs, whose BN here is one
// CTA's half of the tile's columns.
//
// 3xTF32 kernel: K blocks of A (hi and lo parts, BK columns each) that tensor memory holds beside the two accumulator
// buffers, or 0 where fewer than two fit (tiles of 256 columns, two accumulators): A then stays in shared memory.
constexpr int tc_x3_tmem_a(int BM, int BN, int BK, int stages, int x3) {
  if (x3 == 0 || BM != 128 || !(BK == 16 || BK == 32)) return 0;
  const int fit = (512 - 2 * BN * x3) / (2 * BK);
  const int n = kc_min(kc_min(fit, stages), 4);
  return n >= 2 ? n : 0;
}

// Threads of a 3xTF32 CTA: control, splitter (two warpgroups in the pair form with A in tensor memory) and two
// accumulating warpgroups.
constexpr int tc_x3_threads(int tmem_a, int x3) { return tmem_a > 0 && x3 == 2 ? 640 : 512; }

// Bytes of the operand rings: single-pass kernel stages * (A + B tile); 3xTF32 adds the lo ring, without A where that
// goes through tensor memory.
constexpr int tc_ring_bytes(int dtype, int BM, int BN, int BK, int stages, int x3) {
  const int eb = (dtype == KCG_DT_F32) ? 4 : 2;
  const int stage = (BM + BN) * BK * eb;
  if (!(eb == 4 && x3)) return stage * stages;
  const int lo = tc_x3_tmem_a(BM, BN, BK, stages, x3) > 0 ? BN * BK * eb : stage;
  return stage * stages + lo * tc_lo_stages(stages);
}

// Shape rules of the tcgen05 kernels; returns 0 when the config is buildable.
constexpr int tc_config_error(int dtype, int BM, int BN, int BK, int stages, int x3) {
  const int eb = (dtype == KCG_DT_F32) ? 4 : 2;
  if (!(dtype == KCG_DT_F32 || dtype == KCG_DT_F16 || dtype == KCG_DT_BF16)) return 1;
  if (!(BM == 128 || BM == 256)) return 2;
  if (BN < 128 / eb || BN > 256 || (BN % (128 / eb)) != 0 || (BN % 16) != 0) return 3;
  if ((BM / 128) * BN > 512) return 4;
  // 3xTF32: two TMEM accumulator buffers and MT*BN/2 register accumulators per epilogue thread
  if (eb == 4 && x3 && ((BM / 128) * BN > 256 || ((BN % 64) != 0 && !(x3 == 2 && BN == 96)))) return 9;
  const int rowb = BK * eb;
  if (!(rowb == 32 || rowb == 64 || (rowb % 128) == 0) || rowb > 512) return 5;
  if ((BK % (32 / eb)) != 0 || (BK % 8) != 0) return 6;
  if (eb == 2 && (BK % 16) != 0) return 6;
  if (stages < 2 || stages > 12) return 7;
  if (tc_ring_bytes(dtype, BM, BN, BK, stages, x3) + 2048 + tc_staging_bytes(dtype, x3) > 227 * 1024) return 8;
  return 0;
}

// Cluster split-K kernel (gemm_tcgen05_clusterk.cuh): a 128 x BN tile per cluster of `split` CTAs.
// The operand ring doubles as the exchange buffers of the reduction (a staging copy of the fp32
// accumulator, 128 x BN x 4 bytes, plus a receive slot per other CTA), so it must be at least that
// large; no TMA-store staging. `pair`: a 256 x BN tile per cluster of 2 * split CTAs, each loading half of B's columns;
// clusters of more than four such CTAs do not run side by side on enough of the GPU.
constexpr int ck_ring_bytes(int BN, int BK, int stages, int pair) { return (128 + BN / (pair ? 2 : 1)) * BK * 2 * stages; }
constexpr int ck_config_error(int dtype, int BN, int BK, int stages, int split, int pair = 0) {
  if (!(dtype == KCG_DT_F16 || dtype == KCG_DT_BF16)) return 1;
  if (split < 2 || split > (pair ? 2 : 4)) return 2;  // larger clusters do not fit the exchange buffers (nor the GPU: few run at once)
  if (BN < 64 || BN > 256 || (BN % (pair ? 128 : 64)) != 0 || BN / 32 < split) return 3;
  const int rowb = BK * 2;
  if (!(rowb == 32 || rowb == 64 || (rowb % 128) == 0) || rowb > 512 || (BK % 16) != 0) return 5;
  if (stages < 2 || stages > 12) return 7;
  const int ring = ck_ring_bytes(BN, BK, stages, pair);
  if (ring + 2048 > 227 * 1024) return 8;
  // the ring doubles as exchange buffers: a receive slot per other CTA plus a staging copy of the accumulator
  // of the blocks that belong to other CTAs
  if (ring < ((split - 1) * ((BN / 32 + split - 1) / split) + (BN / 32 - BN / 32 / split)) * 128 * 128) return 10;
  return 0;
}
constexpr int ck_smem_bytes(int BN, int BK, int stages, int pair = 0) { return ck_ring_bytes(BN, BK, stages, pair) + 2048; }

// fp32 through fp16 parts (gemm_tcgen05_f32h2.cuh): 256-row tiles on CTA pairs; the kernel it falls back to is the 3xTF32
// pair kernel of the same tile with K blocks of 32 and h2_x3_stages stages.
constexpr int H2_BK = 64;  // K block = chunk of one exponent
// Words between the split and the product, zero between launches: what the split found (H2_UNSPLIT | H2_FAR) and, on the same line,
// the CTAs of the product that are done; slots taken for far parts of A, of B; and H2_FLAGS flags that a value does not split, for
// the CTAs of the split itself. These lie on lines of their own: a thousand CTAs that set one word while others asked for it
// took 30 us.
constexpr unsigned int H2_UNSPLIT = 1u, H2_FAR = 2u;
constexpr int H2_LINE = 32, H2_FOUND = 0, H2_DONE = 1, H2_FAR_A = H2_LINE, H2_FAR_B = 2 * H2_LINE, H2_FLAG = 3 * H2_LINE, H2_FLAGS = 32;
constexpr int H2_WORDS = H2_FLAG + H2_FLAGS * H2_LINE;
// A factor is a power of two: those of a chunk of B and of the first row of a panel of A carry the chunk's slot of far parts
// (from 1 on, 0: none) in the bits below.
constexpr unsigned int H2_SLOT_BITS = 0x7fffffu;
constexpr int h2_config_error(int BM, int BN, int BK) {
  if (BM != 256) return 2;
  if (BN != 128 && BN != 256) return 3;
  return BK == H2_BK ? 0 : 5;
}
constexpr int h2_x3_stages(int BN) { return BN == 256 ? 3 : 6; }
constexpr int h2_stages(int BN) { return BN == 256 ? 3 : 4; }

constexpr int tc_smem_bytes(int dtype, int BM, int BN, int BK, int stages, int x3) {
  // +1024 alignment slack, +1024 barriers / TMEM holder / flags, + epilogue staging
  return tc_ring_bytes(dtype, BM, BN, BK, stages, x3) + 2048 + tc_staging_bytes(dtype, x3);
}

constexpr int h2_smem_bytes(int BN) {
  // ring, staging of the store, barriers, alignment slack; at least what the fallback takes
  const int own = h2_stages(BN) * (128 + BN / 2) * H2_BK * 4 + 8 * 32 * 128 + 2048;
  const int x3 = tc_smem_bytes(KCG_DT_F32, 128, BN / 2, 32, h2_x3_stages(BN), 2);
  return own > x3 ? own : x3;
}

}  // namespace kcg
