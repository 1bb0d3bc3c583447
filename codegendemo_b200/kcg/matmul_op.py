"""Convenience wrappers over the reference-style flow
``KernelArgMatmul -> KCGCompiler.compileKernel -> UserInputs -> CompiledKernelFactory.getKernel``
(the sequence of SerialCompileTask._task_compile_kernel, Runtime/python/kcg/KCGTask.py:275-297)."""
import math

from codegendemo_b200 import _lib
from codegendemo_b200.kcg.CudaLauncher import CudaLauncher
from codegendemo_b200.kcg.CompiledKernelFactory import CompiledKernelFactory, EnumOperator, UserInputs
from codegendemo_b200.kcg.KCGCompiler import KCGCompiler
from codegendemo_b200.kcg.Operators.matmul import KernelArgMatmul
from codegendemo_b200.kcg.Utils import DeviceInfo, EnumKernelDType, FromTorchType


def default_config(M: int, N: int, K: int, dtype: EnumKernelDType, out_dtype=None, **keys) -> KernelArgMatmul:
    """A tensor-core config for the NN case (A is M x K row-major) with sensible B200 defaults;
    any tuning key can be overridden by keyword (attribute names of KernelArgMatmul). ``out_dtype`` =
    float32 with fp16 / bf16 operands stores the fp32 accumulators unrounded."""
    kpm = KernelArgMatmul(M, N, K, dtype, dtype, dtype if out_dtype is None else out_dtype)
    eb = int(dtype) % 30
    kpm.BLOCK_SIZE_M = 128
    kpm.BLOCK_SIZE_N = 256 if N % 256 == 0 else 128 if N % 128 == 0 else 64
    kpm.BLOCK_SIZE_K = 128 // eb
    kpm.THREAD_SIZE_M, kpm.THREAD_SIZE_N = 8, kpm.BLOCK_SIZE_N // 16
    kpm.WARP_SIZE = 32
    kpm.WARP_LAYOUT_M, kpm.WARP_LAYOUT_N = 4, 8
    kpm.BLOCK_LAYOUT_M, kpm.BLOCK_LAYOUT_N = 4, 2
    kpm.isATranspose = 0
    kpm.LOCAL_SPLIT_U = 1
    kpm.BLOCK_MAPPING = 8
    kpm.SHARED_PREFETCH = 1
    kpm.REG_PREFETCH = 1
    kpm.GLOB_LOAD_WIDTH_A = kpm.GLOB_LOAD_WIDTH_B = kpm.GLOB_STORE_WIDTH = 4
    kpm.WARP_SCATTER_WIDTH_A = kpm.THREAD_SCATTER_WIDTH_A = kpm.THREAD_SIZE_M
    kpm.WARP_SCATTER_WIDTH_B = kpm.THREAD_SCATTER_WIDTH_B = kpm.THREAD_SIZE_N
    kpm.UNROLL_NUM = 4
    for k, v in keys.items():
        if not hasattr(kpm, k):
            raise KeyError(f"unknown tuning key {k}")
        setattr(kpm, k, v)
    return kpm


# Tiles of the 16-bit kernels the rule below chooses from: (KERNEL_VARIANT, BLOCK_SIZE_M, N, K) -> microseconds
# {fixed, per K block, per tile beyond its K blocks}. For the cluster split-K kernel the third figure is one per LOCAL_SPLIT_U
# of 2, 3, 4; its 256-row tiles run on CTA pairs, two K ranges only. Fitted to 4 900 device timings (CUDA-graph replay,
# operands rotating) of 36 tiles on 127 single products of 128..32768 x 512..16384 x 256..16384, B stored either way - the two
# 256-row cluster tiles later, to 12 shapes, and the KERNEL_VARIANT 4 rows are from before pairs released accumulators
# without waiting for their stores. On 56 other shapes of that range what the rule picks is now 4 % behind the best measured tile
# on average; more than 10 % on six, worst 10368 x 5568 x 320, 57 us against 38 with 256x256x64 pairs, whose row is too high
# at short K. (The rule of tiles that divide the problem was 22 % behind: 1664 x 2752 x 1472 33 -> 12.9 us, 11136 x 7488 x
# 1792 608 -> 205, 128 x 1344 x 3072 17.3 -> 7.7.) No batched products are among the fit's shapes: their times are 4 to 26 %,
# on average 15 %, above the estimate (24 x 384x768x640 11.5 estimated, 15.6 a call), the picks 2 % behind on 12 shapes, worst
# 10 %. The 256-row cluster tiles against the best 128-row choice: 512 x 4096 x 11008 41.3 -> 36.4 us, 1024 x 2048 x 8192
# 29.5 -> 27.5, 256 x 4096 x 4096 14.9 -> 13.0, 640 x 1280 x 2560 10.2 -> 9.6; behind it where K is short, 512 x 1024 x 1024
# 5.4 / 5.8, or most SMs idle, 256 x 2048 x 16384 23 / 30.
_TILE_COST = {
    (2, 128, 64, 128): (2.85, 0.433, 0.54),
    (2, 128, 128, 128): (2.94, 0.499, 0.53),
    (2, 128, 192, 64): (3.03, 0.344, 0.78),
    (2, 128, 256, 64): (2.81, 0.384, 1.28),
    (2, 256, 192, 64): (2.30, 0.57, 2.70),
    (2, 256, 256, 64): (1.77, 0.645, 4.13),
    (4, 256, 128, 128): (3.38, 0.469, 1.04),
    (4, 256, 256, 64): (3.37, 0.35, 1.58),
    (4, 256, 256, 128): (3.21, 0.663, 1.68),
    (4, 512, 256, 64): (2.02, 0.62, 5.45),
    (5, 128, 64, 128): (1.0, 0.45, (3.10,)),
    (5, 128, 128, 128): (1.0, 0.505, (4.24, 4.65, 4.69)),
    (5, 128, 192, 64): (1.0, 0.322, (5.15, 5.60, 6.32)),
    (5, 128, 256, 64): (1.0, 0.379, (5.77, 6.37, 6.61)),
    (5, 256, 128, 128): (1.0, 0.56, (3.20,)),
    (5, 256, 256, 64): (1.0, 0.35, (5.20,)),
}
# clusters of 2, 3, 4 CTAs at 200 KB of shared memory each that run at once on the GPU the table is fitted to (148 SMs).
# Of 44 or 45 clusters of three some start late, and the product with them, by about 4 us whatever K and the tile: 128 x
# N x 4096 with 128 columns 13.5, 14.1, 16.2, 17.6 us at 42 to 45 tiles; 256x4224x11008 with 192 columns in three ranges
# 31.9, with 128 in two 28.8; 512x2112x4480 18.2 / 14.8. More clusters than run at once take a second wave: 256x4608x4096 in
# 36 clusters of four 26.4, in 72 of two 14.6.
_CLUSTERS = {2: 74, 3: 45, 4: 33}
_LATE_CLUSTERS, _LATE_US = 43, 4.0


def _tile_us(tile, split, M, N, K, batch=1, sms=148):
    """Estimated time of a 16-bit product with one of the tiles above, in microseconds."""
    variant, bm, bn, bk = tile
    fixed, per_block, per_tile = _TILE_COST[tile]
    tiles, blocks = batch * -(-M // bm) * -(-N // bn), -(-K // bk)
    stream = 2.0 + 2e-6 * batch * (M * K + K * N + M * N) / 5.5  # operands and result through HBM at 5.5 TB/s
    if variant == 5:
        ctas = split * bm // 128
        late = _LATE_US if ctas == 3 and _LATE_CLUSTERS < tiles <= _CLUSTERS[3] else 0.0
        waves = -(-tiles // _CLUSTERS[ctas])
        return max(stream, fixed + waves * (-(-blocks // split) * per_block + per_tile[split - 2]) + late)
    at_once = sms // 2 if variant == 4 else sms
    waves, rest = -(-tiles // at_once), tiles % at_once
    f = min(8, at_once // rest) if rest else 0
    while f >= 2 and -(-blocks // f) * (f - 1) >= blocks:
        f -= 1
    if tiles > at_once and f >= 2:  # the launcher cuts the remainder tiles into f K ranges when that pays
        rows = bm // 2 if variant == 4 else bm
        tile_us = 2e-7 * rows * bn * K
        if tile_us * (1.0 - 1.0 / f) > 1.25 * (3.0 + max(0.0, 1.5 + 0.14 * rows * bn / 256 - tile_us)):
            waves = tiles // at_once + 1.0 / f + 3.0 / tile_us
    return max(stream, fixed + waves * (blocks * per_block + per_tile))


def _cheapest_tile(M, N, K, batch=1, single_pass=False):
    """(estimate, tile, split) of the tile with the smallest estimate. Tiles may hang over the edges of the problem,
    except over M and K of a batched one, past whose matrices the next batch lies. ``single_pass``: without the cluster
    split-K kernel."""
    best = None
    for tile in _TILE_COST:
        variant, bm, bn, bk = tile
        if batch > 1 and (M % bm or K % bk) or single_pass and variant == 5:
            continue
        for split in (2, 3, 4) if variant == 5 else (1,):
            if variant == 5 and (split > len(_TILE_COST[tile][2]) + 1 or -(-K // bk) < 2 * split or
                                 batch * -(-M // bm) * -(-N // bn) > _CLUSTERS[split * bm // 128]):
                continue
            # CTA pairs from four whole K blocks a range on. Below, the estimate leaves out up to 0.8 us of theirs (their
            # loads wait for the cluster's start) and 64 columns a CTA are ahead: K = 704 to 768 5.8-6.1 us against 6.1-6.9
            # on 17 shapes, K = 960 6.6-7.0 / 6.4-7.5. At 1024 they replace 128 columns, 7.2-8.0 / 6.5-7.6.
            if variant == 5 and bm == 256 and K // bk < 4 * split:
                continue
            us = _tile_us(tile, split, M, N, K, batch)
            if best is None or us < best[0]:
                best = (us, tile, split)
    return best


# Tiles of the 3xTF32 kernels the rule below chooses from: (KERNEL_VARIANT, BLOCK_SIZE_M, N, K) -> (microseconds
# {fixed, per 1000 values of K, per tile beyond them, per cut into K ranges}, stages). Fitted to 180 device timings
# (graph replay, rotating operands) on 18 shapes of 128..6272 x 512..11008 x 256..11008, plain and with every tile cut
# into 2 to 8 ranges: the tile the fit picks is 2.5 % behind the best measured one on average. The pair tiles of 128 and
# 192 columns, whose A goes through tensor memory, are ahead on the middling shapes (640x2624x1024 25 us against 31 with
# the best of the others, 896x1536x6144 80 / 83, 6272x640x6144 223 / 281 with 256 columns), 128 rows by 256 columns on
# few rows and long K (128x11008x11008 170 / 226), 256 by 256 on the largest (4096^3 488 / 510 with 192 columns).
_TILE_COST_F32 = {
    (2, 128, 64, 32): (2.88, 17.2, 1.44, 4.62, 6),
    (2, 128, 128, 32): (2.46, 20.2, 3.48, 6.14, 4),
    (2, 128, 256, 16): (1.65, 40.0, 7.11, 12.14, 4),
    (4, 256, 128, 32): (2.48, 17.3, 3.49, 6.43, 6),
    (4, 256, 192, 32): (2.32, 21.4, 6.75, 7.64, 5),
    (4, 256, 256, 32): (1.55, 30.4, 7.85, 10.70, 3),
}


def _tile_us_f32(tile, split, M, N, K, sms=148):
    """Estimated time of an fp32 product with one of the tiles above, in microseconds."""
    variant, bm, bn, bk = tile
    fixed, per_k, per_tile, per_cut, _ = _TILE_COST_F32[tile]
    tiles, k_us = -(-M // bm) * -(-N // bn), per_k * K / 1000
    at_once = sms // 2 if variant == 4 else sms
    if split > 1:
        return fixed + -(-tiles * split // at_once) * (k_us / split + per_tile) + per_cut
    us = fixed + -(-tiles // at_once) * (k_us + per_tile)
    f = min(8, at_once // (tiles % at_once)) if tiles % at_once else 0
    if f >= 2:  # the launcher cuts the remainder tiles into f K ranges when that pays
        us = min(us, fixed + tiles // at_once * (k_us + per_tile) + k_us / f + per_tile + per_cut)
    return us


def _cheapest_tile_f32(M, N, K, sms=148):
    """(estimate, tile, split); a split only where all its units run at once, with four K blocks each or more."""
    best = None
    for tile in _TILE_COST_F32:
        variant, bm, bn, bk = tile
        tiles, at_once = -(-M // bm) * -(-N // bn), sms // 2 if variant == 4 else sms
        for split in (1, 2, 3, 4, 6, 8):
            if split > 1 and (tiles * split > at_once or K // bk < 4 * split):
                continue
            us = _tile_us_f32(tile, split, M, N, K)
            if best is None or us < best[0]:
                best = (us, tile, split)
    return best


# Tiles of the split fp32 kernel (KERNEL_VARIANT 6): BLOCK_SIZE_N -> microseconds {fixed, with the split's launch; per million
# values of A and B for the split; per 64 values of K; per tile beyond them; per cut into K ranges}. Fitted to 111 device
# timings (graph replay, rotating operands) on 32 shapes of 128..4864 x 512..11008 x 256..10496, 9 % rms; large products,
# which the power cap slows down by up to a third, are estimated as much too low as the 3xTF32 tiles above.
_TILE_COST_F32_SPLIT = {
    128: (7.5, 1.82, 0.498, 2.4, 2.3),
    256: (6.6, 1.74, 0.723, 6.0, 7.8),
}
_SPLIT_BYTES = 2 << 30  # most memory that a product's parts may take: 4 bytes a value


def _tile_us_f32_split(bn, split, M, N, K, sms=148):
    """Estimated time of an fp32 product on the split kernel, in microseconds."""
    fixed, per_value, per_block, per_tile, per_cut = _TILE_COST_F32_SPLIT[bn]
    tiles, blocks, pairs = -(-M // 256) * -(-N // bn), -(-K // 64), sms // 2
    fixed += per_value * 1e-6 * (M * K + K * N)
    if split > 1:
        return fixed + -(-tiles * split // pairs) * (-(-blocks // split) * per_block + per_tile) + per_cut
    us = fixed + -(-tiles // pairs) * (blocks * per_block + per_tile)
    f = min(8, pairs // (tiles % pairs)) if tiles % pairs else 0
    if f >= 2:  # the launcher cuts the remainder tiles into f K ranges when that pays
        us = min(us, fixed + tiles // pairs * (blocks * per_block + per_tile) + -(-blocks // f) * per_block + per_tile + per_cut)
    return us


def _cheapest_tile_f32_split(M, N, K, sms=148):
    """(estimate, BLOCK_SIZE_N, split), or None where the parts would take too much memory."""
    if 4 * (M * K + K * N) > _SPLIT_BYTES:
        return None
    best = None
    for bn in _TILE_COST_F32_SPLIT:
        for split in (1, 2, 3, 4, 6, 8):
            if split > 1 and (-(-M // 256) * -(-N // bn) * split > sms // 2 or K // 64 < 4 * split):
                continue
            us = _tile_us_f32_split(bn, split, M, N, K)
            if best is None or us < best[0]:
                best = (us, bn, split)
    return best


def tuned_config(M: int, N: int, K: int, dtype: EnumKernelDType, isATranspose: int = 0, db=None, batch: int = 1,
                 b_transposed: bool = False, single_pass: bool = False) -> KernelArgMatmul:
    """Best known config of a shape: the kernel database's entry when the shape was tuned; else (16-bit types, and
    single fp32 products) the tile with the smallest estimated time - the plain rule's choice is kept while the estimate
    puts it within 10 % of that: the estimates of the two largest tiles are up to that much too low where a remainder is
    cut up (2048x11008x4096: 512x256x64 estimated 110, 256x256x128 118 us; measured 142 and 135, and 165 and 148 once the
    power cap holds the clock down). A plain cluster split-K choice is kept within 5 %: of 46 shapes (128 to 512 rows, K 2048 to
    14336) where it is 5 to 10 % behind by estimate the cheapest tile was 3 to 20 % ahead, measured, on all but those with 44
    clusters of three (512x4096x11008 39.4 estimated against 36.3, 40.0 and 35.9 measured); within 5 % it was ahead by 4 to 16 %
    on five shapes, behind by 10 % on one. ``batch`` > 1: M, N, K are one batch's, the config fits all batches' tiles walked
    together, and the database, which holds single products, is not asked. ``b_transposed``: B is stored N x K.
    ``single_pass``: a config of the single-pass kernels (KERNEL_VARIANT 2 and 4), which alone can store fp32 results of
    16-bit operands; 16-bit types."""
    from codegendemo_b200.kcg.InfoDb import KernelDb
    if batch == 1:
        db = db if db is not None else KernelDb()
        hit = db.lookup(M, N, K, int(dtype), isATranspose)
        if hit is not None:
            kpm = KernelArgMatmul.fromJson(hit["config"])
            takes = (2, 4) if single_pass else (2, 4, 5)
            if not (b_transposed or single_pass) or kpm.KERNEL_VARIANT in takes or \
                    (kpm.KERNEL_VARIANT == 0 and kpm.usesTensorCores()):
                return _with_b_transposed(kpm) if b_transposed else kpm
            # (a kernel that cannot do what is asked: the rule decides)
    plain = _plain_rule(batch * M, N, K, dtype, isATranspose)
    if M % plain.BLOCK_SIZE_M:
        plain = _plain_rule(M, N, K, dtype, isATranspose)
    plain.M = M
    if int(dtype) != int(EnumKernelDType.float32) and M % 128 == 0 and N % 64 == 0 and K % 64 == 0:
        us, tile, split = _cheapest_tile(M, N, K, batch, single_pass)
        have = (plain.KERNEL_VARIANT or 2, plain.BLOCK_SIZE_M, plain.BLOCK_SIZE_N, plain.BLOCK_SIZE_K)
        if have not in _TILE_COST or single_pass and have[0] == 5 or \
                _tile_us(have, plain.LOCAL_SPLIT_U, M, N, K, batch) > (1.05 if have[0] == 5 else 1.1) * us:
            variant, bm, bn, bk = tile
            stages = dict(NUM_STAGES=4) if bm == 512 else {}
            plain = default_config(M, N, K, dtype, KERNEL_VARIANT=variant, BLOCK_SIZE_M=bm, BLOCK_SIZE_N=bn,
                                   BLOCK_SIZE_K=bk, LOCAL_SPLIT_U=split, isATranspose=isATranspose,
                                   EDGE_TILES=int(M % bm != 0 or N % bn != 0 or K % bk != 0), **stages)
    elif batch == 1 and not isATranspose and M % 128 == 0 and N % 64 == 0 and K % 64 == 0:
        us, tile, split = _cheapest_tile_f32(M, N, K)
        have = (plain.KERNEL_VARIANT or 2, plain.BLOCK_SIZE_M, plain.BLOCK_SIZE_N, plain.BLOCK_SIZE_K)
        in_parts = _cheapest_tile_f32_split(M, N, K)
        if in_parts is not None and in_parts[0] < 0.95 * us:
            # operands split in memory once, not in every tile that reads them: from about 512 rows on (both kernels'
            # times in _TILE_COST_F32_SPLIT's fit: 128x4096x4096 35 us as 3xTF32, 59 split; 512x8704x2048 79 / 70; 1024x7936x768
            # 65 / 47; 4096^3 495 / 350; of 32 shapes none that this line sends there was slower)
            _, bn, split = in_parts
            plain = default_config(M, N, K, dtype, KERNEL_VARIANT=6, BLOCK_SIZE_M=256, BLOCK_SIZE_N=bn, BLOCK_SIZE_K=64,
                                   LOCAL_SPLIT_U=split, EDGE_TILES=int(M % 256 != 0 or N % bn != 0))
        elif have not in _TILE_COST_F32 or _tile_us_f32(have, 1, M, N, K) > 1.1 * us:
            variant, bm, bn, bk = tile
            plain = default_config(M, N, K, dtype, KERNEL_VARIANT=variant, BLOCK_SIZE_M=bm, BLOCK_SIZE_N=bn,
                                   BLOCK_SIZE_K=bk, LOCAL_SPLIT_U=split, NUM_STAGES=_TILE_COST_F32[tile][4],
                                   EDGE_TILES=int(M % bm != 0 or N % bn != 0 or K % bk != 0))
    return _with_b_transposed(plain) if b_transposed else plain


def _with_b_transposed(kpm):
    """The same config for a B stored N x K: an automatic choice of the kernel is made explicit; the cluster split-K
    kernel takes such a B under the rules of EDGE_TILES."""
    if kpm.KERNEL_VARIANT == 0 and kpm.usesTensorCores():
        kpm.KERNEL_VARIANT = 2
    if kpm.KERNEL_VARIANT == 5:
        kpm.EDGE_TILES = 1
    kpm.IS_BTRANS = 1
    return kpm


def _plain_rule(M: int, N: int, K: int, dtype: EnumKernelDType, isATranspose: int = 0) -> KernelArgMatmul:
    """A rule of thumb over tiles that divide the problem (CTA-pair kernels once their larger tiles still fill
    the 74 pairs for several waves, single-CTA tiles otherwise)."""
    pairs = 74
    if int(dtype) == int(EnumKernelDType.float32):
        if M % 256 == 0 and N % 256 == 0 and K % 32 == 0 and (M // 256) * (N // 256) >= pairs:
            return default_config(M, N, K, dtype, KERNEL_VARIANT=4, BLOCK_SIZE_M=256, BLOCK_SIZE_N=256,
                                  BLOCK_SIZE_K=32, NUM_STAGES=3, isATranspose=isATranspose)
        if N % 256 == 0 and K % 16 == 0:
            return default_config(M, N, K, dtype, BLOCK_SIZE_N=256, BLOCK_SIZE_K=16, NUM_STAGES=4,
                                  isATranspose=isATranspose)
        return default_config(M, N, K, dtype, BLOCK_SIZE_N=128 if N % 128 == 0 else 64, isATranspose=isATranspose)
    tiles256 = (M // 256) * (N // 256) if M % 256 == 0 and N % 256 == 0 else 0
    if K <= 512 and K % 64 == 0 and N % 256 == 0:
        # short K: the epilogue weighs as much as the main loop, so take the tile whose two TMEM accumulator
        # buffers overlap them
        return default_config(M, N, K, dtype, BLOCK_SIZE_N=256, BLOCK_SIZE_K=64, isATranspose=isATranspose)
    if M % 512 == 0 and N % 256 == 0 and K % 64 == 0 and (M // 512) * (N // 256) >= 6 * pairs:
        # six waves and more of 512x256 pair tiles: the largest tile (fewest operand bytes per flop through
        # L2), its accumulator released in halves. Measured in short bursts at full clock (how the benchmark
        # runs) it leads; under a sustained power cap the 256x256x128 tile below overtakes it by a few percent.
        return default_config(M, N, K, dtype, KERNEL_VARIANT=4, BLOCK_SIZE_M=512, BLOCK_SIZE_N=256, BLOCK_SIZE_K=64,
                              NUM_STAGES=4, isATranspose=isATranspose)
    if K % 128 == 0 and tiles256 >= pairs:
        # one to twelve waves of 256x256 pair tiles: CTA pairs with 128-wide K blocks (half as many stage
        # hand-offs per byte as 64-wide ones, two accumulator buffers, remainder split run first); best or within 2 % of
        # the best on every such shape measured, from 512 x 11008 x 4096 to 4096 x 8192 x 8192
        return default_config(M, N, K, dtype, KERNEL_VARIANT=4, BLOCK_SIZE_M=256, BLOCK_SIZE_N=256,
                              BLOCK_SIZE_K=128, isATranspose=isATranspose)
    if K % 64 == 0 and tiles256 >= pairs:
        return default_config(M, N, K, dtype, KERNEL_VARIANT=4, BLOCK_SIZE_M=256, BLOCK_SIZE_N=256,
                              BLOCK_SIZE_K=64, isATranspose=isATranspose)
    pick = clusterk_choice(M, N, K)
    if pick is not None:
        # fewer 128-row tiles than SMs: K is split over the CTAs of a cluster (KERNEL_VARIANT 5, reduction in
        # shared memory) so that two to four times as many SMs stream the operands
        bn, bk, split = pick
        return default_config(M, N, K, dtype, KERNEL_VARIANT=5, BLOCK_SIZE_N=bn, BLOCK_SIZE_K=bk,
                              LOCAL_SPLIT_U=split, isATranspose=isATranspose)
    if N % 128 == 0 and K % 128 == 0 and K >= 1024:
        # few tiles: small tiles with long K blocks (best on the 128- and 512-row shapes)
        return default_config(M, N, K, dtype, BLOCK_SIZE_N=128, BLOCK_SIZE_K=128, isATranspose=isATranspose)
    return default_config(M, N, K, dtype, isATranspose=isATranspose)


def clusterk_choice(M: int, N: int, K: int, sms: int = 148):
    """(BLOCK_SIZE_N, BLOCK_SIZE_K, LOCAL_SPLIT_U) of the cluster split-K kernel for a 16-bit problem with fewer
    128-row tiles than SMs, or None when it does not apply. Of the tile widths 128 and 256, each with the largest
    split of 2..4 whose CTAs still fit one wave, the one that occupies more SMs wins; at equal count the wider
    tile (fewer operand bytes through each SM, less to exchange). Measured: 128 x 4096 x 4096 -> 128 wide, split 4;
    128 x 11008 x K -> 256 wide, split 3; 512 x 4096 x K -> 256 wide, split 2, each ahead of the whole-K kernels."""
    if M % 128 != 0 or M > 512 or K < 2048:
        return None
    best = None
    for bn, bk in ((128, 128), (256, 64)):
        if N % bn != 0 or K % bk != 0:
            continue
        tiles = (M // 128) * (N // bn)
        split = min(4, sms // tiles) if tiles > 0 else 0
        if split < 2 or (K // bk) < 4 * split:
            continue
        ctas = tiles * split
        if best is None or ctas >= best[0]:
            best = (ctas, bn, bk, split)
    return None if best is None else best[1:]


def build_kernel(kpm: KernelArgMatmul, deviceId: int = 0):
    """Compile (or fetch from the cubin cache) and wrap one config; returns (UserInputs, CompiledKernel)."""
    kpm.check()
    compiler = KCGCompiler()
    path, name, gx, gy, gz, bx, by, bz = compiler.compileKernel(kpm)[0]
    inConfig = UserInputs(path, name, kpm, compiler.lastInfo)
    inConfig.m_gridDims = [gx, gy, gz]
    inConfig.m_blockDims = [bx, by, bz]
    inConfig.operatorKind = EnumOperator.Matmul
    return inConfig, CompiledKernelFactory.getKernel(inConfig, deviceId)


_warm = None  # csrc/kcg_torchcall.cpp once something was launched, False where it was not built for this torch


def _warm_calls():
    """The module of the warm calls, bound to the library; False without it."""
    global _warm
    if _warm is None:
        import ctypes
        import torch
        try:
            from codegendemo_b200 import _torchcall
            found = _torchcall if _torchcall.TORCH_VERSION == torch.__version__.split("+")[0] else False
        except ImportError:
            found = False
        if found:
            lib = _lib.get_lib()
            found.bind(*(ctypes.cast(f, ctypes.c_void_p).value for f in (lib.kcg_launch_gemm_strided, lib.kcg_attention_fwd)),
                       _lib.check)
            found.bind_trim(ctypes.cast(lib.kcg_internal_trim_if_low, ctypes.c_void_p).value)
        _warm = found
    return _warm


def _remember(kern, t, M, N, K, batch, b_transposed):
    """The next call of this shape on plain contiguous tensors may be a warm one. (A launch has been made with `kern`.)"""
    launcher, warm = getattr(kern, "m_launcher", None), _warm_calls()
    if warm and isinstance(launcher, CudaLauncher) and t.is_cuda:
        warm.remember(M, N, K, batch, int(FromTorchType(t.dtype)), t.device.index or 0, int(bool(b_transposed)),
                      launcher.m_runtime.m_function, launcher.m_infoAddr, launcher)


_KERNELS = {}  # (operator, shape, dtype, device, options) -> kernel; True == 1, so operators must not share keys


def _row_pitch(t, what: str) -> int:
    """Leading dimension (elements between rows) of a 2-D tensor whose rows are contiguous: a plain
    matrix or a column block / row block view of a wider row-major one."""
    shape, stride = t.shape, t.stride()
    if len(shape) != 2 or (shape[1] > 1 and stride[1] != 1):
        raise ValueError(f"{what} must be a 2-D tensor with contiguous rows (a view with a row pitch is fine)")
    return stride[0] if shape[0] > 1 else shape[1]


def matmul(a, b, c=None, alpha=1.0, beta=0.0, bias=None, relu=False, b_transposed=False, **keys):
    """``c = a @ b`` on the current CUDA device through the kernel database's config for the shape
    (or a default config tuned by keyword). ``alpha``, ``beta``, ``bias`` (N values of c's dtype) and
    ``relu`` fuse ``c = act(alpha * a @ b + beta * c + bias)`` into the kernel's store. The operands may
    be views with a row pitch (column or row blocks of wider row-major tensors): their leading dimensions go
    to the strided launch entry, nothing is copied. ``b_transposed=True`` takes ``b`` stored N x K and computes
    ``a @ b.T`` (16-bit dtypes). Compiled and loaded kernels are kept per (shape, dtype, device, keys)."""
    if _warm and c is None and not keys and type(alpha) is float and alpha == 1.0 and type(beta) is float and beta == 0.0:
        c = _warm.matmul(a, b, bias, relu, b_transposed)
        if c is not None:
            return c
    M, K = a.shape
    if b_transposed:
        N, K2 = b.shape
    else:
        K2, N = b.shape
    assert K == K2
    lda = ldb = ldc = 0  # contiguous
    if c is None and a.is_contiguous() and b.is_contiguous():
        if beta != 0.0:
            raise ValueError("beta != 0 needs the c to scale")
        c = a.new_empty((M, N))
    else:
        lda, ldb = _row_pitch(a, "a"), _row_pitch(b, "b")
        if c is None:
            if beta != 0.0:
                raise ValueError("beta != 0 needs the c to scale")
            c = a.new_empty((M, N))
        ldc = _row_pitch(c, "c")
        if lda == K and ldb == (K if b_transposed else N) and ldc == N:
            lda = ldb = ldc = 0
    dev = a.device.index or 0
    key = ("mm", M, N, K, a.dtype, dev, tuple(sorted(keys.items())) if keys else (), bool(b_transposed))
    kern = _KERNELS.get(key)
    if kern is None:
        dt = FromTorchType(a.dtype)
        if keys:
            kpm = default_config(M, N, K, dt, **keys)
            if b_transposed:
                kpm = _single_pass_16bit(kpm, M, N, K, dt)
                kpm.IS_BTRANS = 1
        else:
            kpm = tuned_config(M, N, K, dt, b_transposed=b_transposed)
        _, kern = build_kernel(kpm, dev)
        _KERNELS[key] = kern
        keep = not keys
    else:
        keep = False
    kern.m_launcher.launchKernel(dev, a, b, c, alpha=alpha, beta=beta, bias=bias, relu=relu, lda=lda, ldb=ldb, ldc=ldc)
    if keep:
        _remember(kern, a, M, N, K, 0, b_transposed)
    return c


def _single_pass_16bit(kpm, M, N, K, dt):
    """An N x K stored B runs on the single-pass tcgen05 kernels (variants 2 and 4) only: keep a tuned config of
    those families, else fall back to the default tile."""
    if kpm.KERNEL_VARIANT in (2, 4) or (kpm.KERNEL_VARIANT == 0 and kpm.usesTensorCores()):
        if kpm.KERNEL_VARIANT == 0:
            kpm.KERNEL_VARIANT = 2
        return kpm
    return default_config(M, N, K, dt, KERNEL_VARIANT=2)


def _attention_tile(heads, m, n, kk, dt, scores):
    """Config of one of the attention chain's batched products, per head m x n x kk. ``scores``: q k^T with k as stored;
    the scores leave as fp32: rounded to 16 bits first, their error (up to 2^-9 of a score of several units) would be
    amplified by the softmax's exp."""
    kpm = tuned_config(m, n, kk, dt, batch=heads, b_transposed=scores, single_pass=True)
    if scores:
        kpm.setOutputDtype(EnumKernelDType.float32)
    return kpm


def attention(q, k, v, scale=None, out=None):
    """``softmax(scale * q @ k^T) @ v`` per head, the attention-shaped chain, as three launches on the current
    stream: a batched product with k taken as stored (keys x head_dim, no transposed copy) whose epilogue applies
    ``scale`` and which stores the scores as fp32; a row softmax (fp32 arithmetic) from the scores into
    probabilities of the inputs' dtype; a batched product with v. ``q`` is (heads, Sq, d), ``k`` and ``v`` are
    (heads, Sk, d), all contiguous fp16 / bf16; ``heads`` may be batch * heads flattened. The Sq x Sk score and
    probability matrices are materialised; Sk must be a multiple of 8. Returns (heads, Sq, d)."""
    import ctypes
    import torch
    H, Sq, D = q.shape
    H2, Sk, D2 = k.shape
    assert H == H2 and D == D2 and tuple(v.shape) == (H, Sk, D)
    assert q.is_contiguous() and k.is_contiguous() and v.is_contiguous()
    assert q.dtype in (torch.float16, torch.bfloat16) and k.dtype == q.dtype and v.dtype == q.dtype
    if scale is None:
        scale = 1.0 / math.sqrt(D)
    dt = FromTorchType(q.dtype)
    dev = q.device.index or 0
    key = ("attn", H, Sq, Sk, D, int(dt), dev)
    kerns = _KERNELS.get(key)
    if kerns is None:
        def tile_for(m, n, kk, scores):
            return build_kernel(_attention_tile(H, m, n, kk, dt, scores), dev)[1]
        kerns = (tile_for(Sq, Sk, D, True), tile_for(Sq, D, Sk, False))
        _KERNELS[key] = kerns
    scores = torch.empty((H, Sq, Sk), dtype=torch.float32, device=q.device)
    probs = torch.empty((H, Sq, Sk), dtype=q.dtype, device=q.device)
    if out is None:
        out = torch.empty((H, Sq, D), dtype=q.dtype, device=q.device)
    kerns[0].run(q, k, scores, alpha=float(scale), batch=H)
    _lib.check(_lib.get_lib().kcg_softmax_rows_ex(dev, ctypes.c_uint64(DeviceInfo.get_cuda_stream(dev)),
                                                  ctypes.c_uint64(scores.data_ptr()), int(EnumKernelDType.float32), 0,
                                                  ctypes.c_uint64(probs.data_ptr()), int(dt), 0, H * Sq, Sk, 1.0))
    kerns[1].run(probs, v, out, batch=H)
    return out


def attention_fused(q, k, v, scale=None, out=None):
    """``softmax(scale * q @ k^T) @ v`` per head, fused (``kcg_attention_fwd``, one or two launches): scores and
    probabilities stay on the SM. ``q`` is (heads, Sq, d), ``k`` and ``v`` are (heads, Sk, d), all
    contiguous fp16 / bf16 with d = 64 or 128; any Sq and Sk. Returns (heads, Sq, d). ``attention`` above is the
    three-launch form of the same chain."""
    if _warm and scale is None and out is None:
        out = _warm.attention(q, k, v)
        if out is not None:
            return out
    import torch
    H, Sq, D = q.shape
    H2, Sk, D2 = k.shape
    assert H == H2 and D == D2 and tuple(v.shape) == (H, Sk, D)
    assert q.is_contiguous() and k.is_contiguous() and v.is_contiguous()
    assert q.dtype in (torch.float16, torch.bfloat16) and k.dtype == q.dtype and v.dtype == q.dtype
    if scale is None:
        scale = 1.0 / math.sqrt(D)
    if out is None:
        out = q.new_empty((H, Sq, D))
    assert out.is_contiguous() and tuple(out.shape) == (H, Sq, D) and out.dtype == q.dtype
    dev = q.device.index or 0
    if _lib.pycall is None:
        _lib.get_lib()
    dt = EnumKernelDType.bfloat16 if q.dtype == torch.bfloat16 else EnumKernelDType.float16
    status = _lib.pycall.attention(dev, DeviceInfo.get_cuda_stream(dev), q, k, v, out, dt, H, Sq, Sk, D, scale)
    if status:
        _lib.check(status)
    if _warm is None:
        _warm_calls()
    return out


def attention_status(device: int = 0) -> None:
    """Synchronises the device and raises if a bounded wait of the fused attention kernel ran out."""
    import ctypes
    out = (ctypes.c_uint32 * 4)()
    _lib.check(_lib.get_lib().kcg_attention_status(int(device), out))


def bmm(a, b, c=None, alpha=1.0, beta=0.0, bias=None, relu=False, **keys):
    """``c[i] = a[i] @ b[i]`` (``torch.bmm`` layout: a is batch x M x K, b is batch x K x N, both
    contiguous) as ONE launch of the kernel compiled for a single batch's M, N, K: the persistent grid
    walks the tiles of all batches, so that small per-batch problems fill the GPU together. The
    epilogue keywords are those of ``matmul`` (a bias is shared by the batches)."""
    if _warm and c is None and not keys and type(alpha) is float and alpha == 1.0 and type(beta) is float and beta == 0.0:
        c = _warm.bmm(a, b, bias, relu)
        if c is not None:
            return c
    batch, M, K = a.shape
    batch2, K2, N = b.shape
    assert batch == batch2 and K == K2 and a.is_contiguous() and b.is_contiguous()
    if c is None:
        if beta != 0.0:
            raise ValueError("beta != 0 needs the c to scale")
        c = a.new_empty((batch, M, N))
    dev = a.device.index or 0
    key = ("bmm", M, N, K, a.dtype, dev, tuple(sorted(keys.items())) if keys else (), 0 if keys else batch)
    kern = _KERNELS.get(key)
    if kern is None:
        dt = FromTorchType(a.dtype)
        if keys:
            kpm = default_config(M, N, K, dt, **keys)
        else:
            # the launch walks all batches' tiles as one tall problem: the tile is picked for that much work
            kpm = tuned_config(M, N, K, dt, batch=batch)
        _, kern = build_kernel(kpm, dev)
        _KERNELS[key] = kern
        keep = not keys
    else:
        keep = False
    kern.m_launcher.launchKernel(dev, a, b, c, alpha=alpha, beta=beta, bias=bias, relu=relu, batch=batch)
    if keep:
        _remember(kern, a, M, N, K, batch, False)
    return c
