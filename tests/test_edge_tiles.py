"""Tiles that hang over the edges of the problem (EDGE_TILES), and the rule that picks a 16-bit product's tile."""
import random

import pytest
import torch

from codegendemo_b200 import _lib
from codegendemo_b200.kcg.KCGCompiler import compile_info
from codegendemo_b200.kcg.matmul_op import _TILE_COST, build_kernel, default_config, tuned_config
from codegendemo_b200.kcg.Utils import EnumKernelDType as E, ToTorchType
from oracle import oracle


def _keys(tile, split):
    variant, bm, bn, bk = tile
    keys = dict(KERNEL_VARIANT=variant, BLOCK_SIZE_M=bm, BLOCK_SIZE_N=bn, BLOCK_SIZE_K=bk, LOCAL_SPLIT_U=split,
                EDGE_TILES=1)
    if bm == 512:
        keys["NUM_STAGES"] = 4
    return keys


def _cfg(tile, split, M, N, K, dt=E.bfloat16, btrans=0):
    kpm = default_config(M, N, K, dt, **_keys(tile, split))
    kpm.IS_BTRANS = btrans
    return kpm


def test_every_shape_gets_a_config_the_kernels_can_build():
    """Seeded shapes of multiples of 128 x 64 x 64, single and batched, B stored either way: the rule's config passes
    its own check and the compile entry's rules, and a batched one never hangs over M or K."""
    import ctypes
    rng = random.Random(5)
    lib = _lib.get_lib()
    for i in range(300):
        M, N, K = 128 * rng.randint(1, 64), 64 * rng.randint(1, 128), 64 * rng.randint(1, 128)
        batch, bt = rng.choice([1, 1, 3, 24]), rng.random() < 0.3
        kpm = tuned_config(M, N, K, rng.choice([E.bfloat16, E.float16]), batch=batch, b_transposed=bt)
        kpm.check()
        assert (kpm.M, kpm.N, kpm.K, kpm.IS_BTRANS) == (M, N, K, int(bt))
        assert batch == 1 or (M % kpm.BLOCK_SIZE_M == 0 and K % kpm.BLOCK_SIZE_K == 0)
        opts = _lib.CompileOpts(kernel=kpm.KERNEL_VARIANT, num_stages=kpm.NUM_STAGES, b_trans=kpm.IS_BTRANS,
                                edge_tiles=kpm.EDGE_TILES)
        buf = ctypes.create_string_buffer(1024)
        _lib.check(lib.kcg_kernel_name(_lib.cfg_array(kpm.compileArgs()), ctypes.byref(opts), buf, 1024))


def test_edge_tiles_are_an_option_with_rules_of_their_own():
    with pytest.raises(_lib.KCGError):  # without the option the tile must divide the problem
        compile_info(default_config(128, 192, 64, E.bfloat16, BLOCK_SIZE_N=128).compileArgs(), kernel=2)
    info = compile_info(default_config(384, 192, 96, E.bfloat16, BLOCK_SIZE_N=128).compileArgs(), kernel=2, edge_tiles=1)
    assert info.grid[0] == 3 * 2
    for N, K, kernel in ((200, 64, 2), (192, 68, 2), (192, 64, 1)):  # a block of 64 columns, 16-byte rows, tcgen05 only
        with pytest.raises(_lib.KCGError):
            compile_info(default_config(128, N, K, E.bfloat16, BLOCK_SIZE_N=128).compileArgs(), kernel=kernel, edge_tiles=1)


def test_a_config_pickled_before_the_option_existed():
    """An autotune run that was interrupted leaves pickled configs behind; those of an older version lack the key."""
    import pickle
    kpm = default_config(128, 128, 64, E.bfloat16)
    del kpm.__dict__["EDGE_TILES"]
    old = pickle.loads(pickle.dumps(kpm))
    old.check()
    assert old.jsonfy() == default_config(128, 128, 64, E.bfloat16).jsonfy()


def test_every_fp32_shape_gets_a_config_the_kernels_can_build():
    import ctypes
    rng = random.Random(8)
    lib = _lib.get_lib()
    for i in range(200):
        M, N, K = 128 * rng.randint(1, 64), 64 * rng.randint(1, 172), 64 * rng.randint(1, 172)
        kpm = tuned_config(M, N, K, E.float32)
        kpm.check()
        assert (kpm.M, kpm.N, kpm.K) == (M, N, K)
        opts = _lib.CompileOpts(kernel=kpm.KERNEL_VARIANT, num_stages=kpm.NUM_STAGES, edge_tiles=kpm.EDGE_TILES)
        buf = ctypes.create_string_buffer(1024)
        _lib.check(lib.kcg_kernel_name(_lib.cfg_array(kpm.compileArgs()), ctypes.byref(opts), buf, 1024))


@pytest.mark.gpu
# a tile of every kind the fp32 rule can pick, over the edges of M, N and K, whole and cut into K ranges
@pytest.mark.parametrize("shape", [(128, 64, 64), (384, 320, 192), (640, 832, 1088)], ids=lambda s: "x".join(map(str, s)))
def test_fp32_tiles_over_the_edges(shape):
    from codegendemo_b200.kcg.matmul_op import _TILE_COST_F32
    M, N, K = shape
    gen = torch.Generator().manual_seed(2)
    a, b = [torch.rand(s, generator=gen) * 2 - 1 for s in ((M, K), (K, N))]
    bias = torch.rand(N, generator=gen)
    ref = a.double() @ b.double()
    for tile, cost in _TILE_COST_F32.items():
        for split in (1, 3):
            if split > 1 and K // tile[3] < 4 * split:
                continue
            kpm = default_config(M, N, K, E.float32, KERNEL_VARIANT=tile[0], BLOCK_SIZE_M=tile[1], BLOCK_SIZE_N=tile[2],
                                 BLOCK_SIZE_K=tile[3], NUM_STAGES=cost[4], LOCAL_SPLIT_U=split, EDGE_TILES=1)
            _, kern = build_kernel(kpm, 0)
            wide = torch.full((M + 2, N + 64), float("nan"), device="cuda")
            c = wide[1:1 + M, 32:32 + N]
            for kw, want in ((dict(), ref), (dict(bias=bias.cuda(), relu=True), (ref + bias.double()).clamp(min=0))):
                kern.run(a.cuda(), b.cuda(), c, ldc=N + 64, **kw)
                kern.checkStatus()
                # three TF32 products: 2^-21 of the operands' lengths' product, which |row| * |column| bounds
                bound = 2.0 ** -20 * a.double().norm(dim=1)[:, None] * b.double().norm(dim=0)[None] + 2.0 ** -22
                assert ((c.cpu().double() - want).abs() <= bound).all(), (tile, split)
            wide[1:1 + M, 32:32 + N] = float("nan")
            assert wide.isnan().all(), (tile, split)


TILES = [(t, s) for t in _TILE_COST for s in ((2, 3, 4)[:len(_TILE_COST[t][2])] if t[0] == 5 else (1,))]
# one tile short of everything; one block past a tile in N, half a K block past the last; several tiles and waves
SHAPES = [(128, 64, 64), (384, 320, 192), (640, 832, 1088)]


@pytest.mark.gpu
@pytest.mark.parametrize("tile,split", TILES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_edge_tiles_match_the_oracle_and_stay_inside_c(tile, split):
    """Every tile of the rule on problems it does not divide, C a corner of a larger poisoned matrix of which the
    rest must stay untouched; plain, with B stored N x K, and with bias and ReLU (whose operands end at the edge)."""
    for M, N, K in SHAPES:
        if -(-K // tile[3]) < split:
            continue
        A, B = oracle.make_inputs(M, N, K, torch.bfloat16, "normal", seed=21)
        ref = oracle.host_matmul(A, B)
        bias = torch.rand(N, generator=torch.Generator().manual_seed(2)).to(torch.bfloat16)
        for btrans, fused in ((0, False), (1, False), (0, True)):
            _, kern = build_kernel(_cfg(tile, split, M, N, K, btrans=btrans), 0)
            big = torch.full((M + 512, N + 256), 7.0, dtype=torch.bfloat16, device="cuda:0")
            c = big[:M, :N]
            c.fill_(float("nan"))
            b = (B.t().contiguous() if btrans else B).cuda()
            kw = dict(bias=bias.cuda(), relu=True) if fused else {}
            kern.run(A.cuda(), b, c, ldc=N + 256, **kw)
            kern.checkStatus()
            want = oracle.host_matmul_fused(A, B, bias=bias, relu=True) if fused else ref
            err = oracle.rel_errors(c, want)
            assert not err["nan"] and err["max_rel"] <= oracle.TOL_16BIT, (M, N, K, btrans, fused, err)
            assert bool((big[M:] == 7.0).all()) and bool((big[:, N:] == 7.0).all()), "wrote past C"


@pytest.mark.gpu
# every tile cut into K ranges that are summed out of the operand ring, rows past M among them; N inside the tiles (bulk
# copies of the sums) and past them (plain stores)
@pytest.mark.parametrize("shape", [(384, 512, 8192), (640, 320, 4096)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("tile,split", [((4, 256, 256, 64), 8), ((4, 512, 256, 64), 4), ((2, 256, 192, 64), 4),
                                        ((4, 256, 128, 128), 3)], ids=lambda v: str(v).replace(", ", "x"))
def test_split_edge_tiles_scale_and_add_c(shape, tile, split):
    """c = alpha a b + beta c with C a corner of a larger matrix: C is read inside its rows only, nothing else changes."""
    M, N, K = shape
    A, B = oracle.make_inputs(M, N, K, torch.bfloat16, "normal", seed=22)
    kpm = _cfg(tile, split, M, N, K)
    _, kern = build_kernel(kpm, 0)
    big = torch.randn((M + 512, N + 256), generator=torch.Generator().manual_seed(3)).to(torch.bfloat16)
    want = 0.5 * (A.double() @ B.double()) - 2.0 * big[:M, :N].double()
    dev = big.cuda()
    kern.run(A.cuda(), B.cuda(), dev[:M, :N], ldc=N + 256, alpha=0.5, beta=-2.0)
    kern.checkStatus()
    out = dev.cpu()
    # one rounding to bf16 (half a unit of the result), 32-bit sums of terms whose sizes add up to |A| |B|
    bound = 2.0 ** -8 * want.abs() + 2.0 ** -18 * (A.double().abs() @ B.double().abs())
    assert ((out[:M, :N].double() - want).abs() <= bound).all()
    assert torch.equal(out[M:], big[M:]) and torch.equal(out[:, N:], big[:, N:])


@pytest.mark.gpu
def test_edge_tiles_hold_over_many_waves_and_repeat_bitwise():
    """Several waves of tiles that hang over both edges, every element checked against a device fp32 product: the
    staging buffers of skipped blocks must not be counted as stored (a fifth of the tiles came out wrong)."""
    M, N, K = 3968, 12672, 256
    A, B = (torch.randn(s, generator=torch.Generator("cuda").manual_seed(3), device="cuda") for s in ((M, K), (K, N)))
    A, B = (A / 16).to(torch.bfloat16), B.to(torch.bfloat16)
    ref = A.float() @ B.float()
    for tile in ((2, 128, 192, 64), (2, 256, 256, 64), (4, 256, 256, 128), (4, 512, 256, 64)):
        _, kern = build_kernel(_cfg(tile, 1, M, N, K), 0)
        out = []
        for _ in range(2):
            c = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda:0")
            kern.run(A, B, c)
            kern.checkStatus()
            out.append(c)
        # a bf16 rounding is at most 2^-8 of the value; the fp32 sums differ by far less
        assert bool(((out[0].float() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all())
        assert torch.equal(out[0], out[1])


@pytest.mark.gpu
def test_batched_products_with_ragged_widths():
    from codegendemo_b200.kcg.matmul_op import bmm
    for batch, M, N, K in ((3, 128, 192, 64), (5, 384, 832, 192), (2, 256, 320, 1088)):
        a = torch.randn((batch, M, K), generator=torch.Generator().manual_seed(4)).div_(K ** 0.5).to(torch.bfloat16)
        b = torch.randn((batch, K, N), generator=torch.Generator().manual_seed(5)).to(torch.bfloat16)
        b[0, -1] = float("inf")  # the rows past a batch's K are the next batch's: they must not be touched
        c = bmm(a.cuda(), b.cuda()).cpu()
        for i in range(1, batch):
            err = oracle.rel_errors(c[i], oracle.host_matmul(a[i], b[i]))
            assert not err["nan"] and err["max_rel"] <= oracle.TOL_16BIT, (i, err)
