"""The split fp32 kernel (KERNEL_VARIANT 6): fp16 parts of both operands, written in front of the product, and the 3xTF32
kernel in the same launch where values do not split."""
import ctypes
import os
import random
import subprocess

import pytest
import torch

from codegendemo_b200 import _lib
from codegendemo_b200.kcg.KCGCompiler import compile_info
from codegendemo_b200.kcg.matmul_op import build_kernel, default_config, matmul, tuned_config
from codegendemo_b200.kcg.Utils import EnumKernelDType as E


def _kernel(M, N, K, bn, split=1):
    return build_kernel(default_config(M, N, K, E.float32, KERNEL_VARIANT=6, BLOCK_SIZE_M=256, BLOCK_SIZE_N=bn, BLOCK_SIZE_K=64,
                                       LOCAL_SPLIT_U=split, EDGE_TILES=1), 0)[1]


def _as_tf32(M, N, K, bn):
    """The kernel this one falls back to."""
    return build_kernel(default_config(M, N, K, E.float32, KERNEL_VARIANT=4, BLOCK_SIZE_M=256, BLOCK_SIZE_N=bn, BLOCK_SIZE_K=32,
                                       NUM_STAGES=3 if bn == 256 else 6, EDGE_TILES=1), 0)[1]


def _bound(a, b):
    """What 3xTF32 guarantees of a value: products left out and rounded, and sums of K terms in fp32."""
    return 2.0 ** -20 * (a.double().abs() @ b.double().abs())


def _split(x, axis):
    """hi, lo and 2^-e of the split kernel, in 64 bits: 64 values along `axis` share an exponent."""
    top = x.abs().amax(dim=axis, keepdim=True)
    scale = torch.where(top > 0, torch.exp2(14 - torch.floor(torch.log2(torch.where(top > 0, top, torch.ones_like(top))))), 1.0)
    y = x.double() * scale
    hi = y.half().double()
    return hi, ((y - hi) * 4096).half().double() / 4096, 1 / scale


def test_two_parts_keep_21_bits():
    """The arithmetic of the split: 2^-22 of a value is lost at most down to 2^-28 of the largest beside it, and the product
    that is left out is below 2^-24."""
    gen = torch.Generator().manual_seed(1)
    x = torch.rand((256, 64), generator=gen) * 2 - 1
    x = (x * torch.exp2(-torch.randint(0, 28, x.shape, generator=gen).float()))
    x[:, 0] = 1.0
    hi, lo, inv = _split(x, 1)
    assert ((hi + lo) * inv - x.double()).abs().le(2.0 ** -22 * x.double().abs()).all()
    assert (lo.abs() <= 2.0 ** -11 * hi.abs().clamp(min=2.0 ** -14)).all() and hi.abs().max() < 65504


def test_configs_and_the_rule():
    for bn, stages, threads in ((128, 4, 640), (256, 3, 512)):
        kpm = default_config(384, 320, 192, E.float32, KERNEL_VARIANT=6, BLOCK_SIZE_M=256, BLOCK_SIZE_N=bn, BLOCK_SIZE_K=64,
                             EDGE_TILES=1)
        kpm.check()
        info = compile_info(kpm.compileArgs(), kernel=6, edge_tiles=1)
        assert (info.kernel, info.stages, info.block[0]) == (_lib.KERNEL_F32_SPLIT, stages, threads)
        assert list(info.cluster) == [2, 1, 1] and info.smem_bytes <= 227 * 1024
    for bad in (dict(BLOCK_SIZE_M=512), dict(BLOCK_SIZE_N=192), dict(BLOCK_SIZE_K=32), dict(isATranspose=1)):
        keys = {**dict(KERNEL_VARIANT=6, BLOCK_SIZE_M=256, BLOCK_SIZE_N=256, BLOCK_SIZE_K=64), **bad}
        with pytest.raises(RuntimeError):
            compile_info(default_config(1024, 768, 512, E.float32, **keys).compileArgs(), kernel=6, edge_tiles=1)
    with pytest.raises(RuntimeError):  # 16-bit data
        compile_info(default_config(256, 256, 256, E.float16, KERNEL_VARIANT=6, BLOCK_SIZE_M=256, BLOCK_SIZE_K=64).compileArgs(),
                     kernel=6)

    class NoDb:
        def lookup(self, *shape):
            return None

    def variant(M, N, K):
        return tuned_config(M, N, K, E.float32, db=NoDb()).KERNEL_VARIANT
    assert variant(4096, 4096, 4096) == 6 and variant(1024, 7936, 768) == 6
    assert variant(128, 4096, 4096) != 6       # few rows: B would be written and read once more for one row of tiles
    assert variant(65536, 8192, 8192) != 6     # 2.25 GB of parts


@pytest.mark.parametrize("bn", [128, 256])
def test_both_kernels_of_a_launch_cover_every_tile(bn, tmp_path, monkeypatch):
    """One plan is walked in K blocks of 64, or of 32 by the kernel that a launch falls back to: in every mode of
    KCG_TAIL_SPLIT both walks cover every tile's K once, within the slots of the launch."""
    lib = _lib.get_lib()
    lib.kcg_internal_plan_split.argtypes = [ctypes.POINTER(_lib.KernelInfo), ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int)]
    tests = os.path.dirname(os.path.abspath(__file__))
    kernels = os.path.join(os.path.dirname(tests), "codegendemo_b200", "csrc", "kernels")
    for bk in (64, 32):
        subprocess.run(["g++", "-O1", "-std=c++17", "-I/usr/local/cuda/include", "-I" + kernels, "-DWIC_BM=256", f"-DWIC_BN={bn}",
                        f"-DWIC_BK={bk}", "-o", str(tmp_path / str(bk)), os.path.join(tests, "work_iter_check.cpp")], check=True)
    rng = random.Random(bn)
    layers = set()
    for M, N, K in [(4096, 4096, 4096), (2048, 11008, 11008)] + [
            (256 * rng.randint(1, 20), bn * rng.randint(1, 40), rng.choice([4 * rng.randint(16, 400), 64 * rng.randint(4, 172)]))
            for _ in range(10)]:
        for mode in (None, "1", "2", "3", "4", "5"):
            if mode is None:
                monkeypatch.delenv("KCG_TAIL_SPLIT", raising=False)
            else:
                monkeypatch.setenv("KCG_TAIL_SPLIT", mode)
            kpm = default_config(M, N, K, E.float32, KERNEL_VARIANT=6, BLOCK_SIZE_M=256, BLOCK_SIZE_N=bn, BLOCK_SIZE_K=64, EDGE_TILES=1)
            info = compile_info(kpm.compileArgs(), kernel=6, edge_tiles=1)
            out = (ctypes.c_int * 7)()
            assert lib.kcg_internal_plan_split(ctypes.byref(info), 0, 1, out) == 0
            tiles, first, factor, sk_per, ranges, at_once, units_first = out
            assert (sk_per, ranges) == (0, 0)
            layers.add(factor > 1)
            grid, slots = min(first + (tiles - first) * factor, at_once), (tiles - first) * factor
            for bk in (64, 32):
                r = subprocess.run([str(tmp_path / str(bk))] + [str(v) for v in (M, N, K, first, factor, sk_per, grid, slots, units_first)],
                                   capture_output=True, text=True)
                assert r.returncode == 0 and r.stdout.startswith("OK"), (M, N, K, mode, bk, list(out), r.stdout + r.stderr)
    assert layers == {False, True}


@pytest.mark.gpu
# one chunk of K; tiles and panels of rows over the edges, K no multiple of a chunk; several tiles and chunks past the ring
@pytest.mark.parametrize("shape", [(128, 64, 64), (384, 320, 196), (640, 832, 1092)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("bn,split", [(128, 1), (128, 3), (256, 1), (256, 2)])
def test_tiles_over_the_edges(shape, bn, split):
    M, N, K = shape
    if K < 64 * 2 * split:
        split = 1
    kern = _kernel(M, N, K, bn, split)
    gen = torch.Generator().manual_seed(2)
    wide_a, wide_b = [torch.rand(s, generator=gen).cuda() * 2 - 1 for s in ((M, K + 8), (K, N + 64))]
    a, b = wide_a[:, 4:4 + K], wide_b[:, 64:]
    bias = torch.rand(N, generator=gen).cuda()
    old = torch.rand((M, N), generator=gen).cuda()
    ref = a.double() @ b.double()
    wide = torch.full((M + 2, N + 64), float("nan"), device="cuda")
    c = wide[1:1 + M, 32:32 + N]
    for kw, want in ((dict(), ref), (dict(bias=bias, relu=True), (ref + bias.double()).clamp(min=0)),
                     (dict(alpha=0.5, beta=2.0), 0.5 * ref + 2.0 * old.double())):
        c.copy_(old)
        kern.run(a, b, c, lda=K + 8, ldb=N + 64, ldc=N + 64, **kw)
        kern.checkStatus()
        assert ((c.double() - want).abs() <= _bound(a, b) + 2.0 ** -22 * want.abs().clamp(min=1)).all(), kw
    first = c.clone()
    c.copy_(old)
    kern.run(a, b, c, lda=K + 8, ldb=N + 64, ldc=N + 64, alpha=0.5, beta=2.0)
    assert torch.equal(c, first)
    wide[1:1 + M, 32:32 + N] = float("nan")
    assert wide.isnan().all()


@pytest.mark.gpu
def test_closer_than_three_tf32_products():
    M, N, K = 512, 512, 4096
    gen = torch.Generator(device="cuda").manual_seed(3)
    a, b = [torch.rand(s, generator=gen, device="cuda") * 2 - 1 for s in ((M, K), (K, N))]
    ref = a.double() @ b.double()
    out = [torch.empty((M, N), device="cuda") for _ in range(2)]
    _kernel(M, N, K, 256).run(a, b, out[0])
    _as_tf32(M, N, K, 256).run(a, b, out[1])
    err = [float((c.double() - ref).norm() / ref.norm()) for c in out]
    assert err[0] < 0.5 * err[1], err  # (measured 1.9e-7 and 1.0e-6)


def _planted(kind, a, b):
    if kind == "inf":
        a[3, 5], b[7, 9] = float("inf"), float("-inf")
    elif kind == "nan":
        b[70, 17] = float("nan")
    elif kind == "huge":
        a[1] *= 2.0 ** 70
    elif kind == "tiny":
        b[:, 2] *= 2.0 ** -70
        b[:, 3] *= 2.0 ** -130
    elif kind == "far below":  # a value that counts, 2^-35 of the largest beside it
        a[9, 1], a[9, 2] = 2.0 ** 20, 1.2345678e-5
        b[1], b[2] = 0.0, 2.0 ** 20
    elif kind == "vanishes":  # 2^-115 beside 2^50: its factor makes it a zero
        a[9] = 0.0
        a[9, 1], a[9, 2] = 2.0 ** 50, 1.5 * 2.0 ** -115
        b[1] = 0.0
    elif kind == "column vanishes":  # 2^-112 in a column whose other values are near 2^40
        a[:, 24], a[9] = 0.0, 0.0
        a[9, 2] = 1.0
        b[:, 4] *= 2.0 ** 40
        b[2, 4] = 1.5 * 2.0 ** -112
    return a, b


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["inf", "nan", "huge", "tiny", "far below", "vanishes", "column vanishes"])
@pytest.mark.parametrize("bn", [128, 256])
@pytest.mark.parametrize("fused", [False, True])
def test_values_that_do_not_split(kind, bn, fused):
    """The 3xTF32 kernel's results, bit for bit; and the next call on the stream is not affected."""
    M, N, K = 384, 320, 192
    gen = torch.Generator().manual_seed(5)
    plain = [torch.rand(s, generator=gen) * 2 - 1 for s in ((M, K), (K, N))]
    a, b = [t.cuda() for t in _planted(kind, *[t.clone() for t in plain])]
    kw = dict(bias=torch.rand(N, generator=gen).cuda(), relu=True) if fused else {}
    kern, other = _kernel(M, N, K, bn), _as_tf32(M, N, K, bn)
    c, want = [torch.full((M, N), 7.0, device="cuda") for _ in range(2)]
    other.run(a, b, want, **kw)
    for _ in range(2):
        c.fill_(7.0)
        kern.run(a, b, c, **kw)
        kern.checkStatus()
        assert torch.equal(c.nan_to_num(nan=123.0), want.nan_to_num(nan=123.0))
    a, b = [t.cuda() for t in plain]
    kern.run(a, b, c, **kw)
    other.run(a, b, want, **kw)
    assert not torch.equal(c, want)  # (closer to the exact product than that)
    ref = a.double() @ b.double()
    ref = (ref + kw["bias"].double()).clamp(min=0) if fused else ref
    assert ((c.double() - ref).abs() <= _bound(a, b) + 2.0 ** -22).all()


@pytest.mark.gpu
def test_values_that_split():
    """Rows, columns and stretches of K of very different size, zeros, and exponents up to the limits: the split kernel's own
    result, within what 3xTF32 guarantees."""
    M, N, K = 256, 256, 256
    gen = torch.Generator().manual_seed(6)
    a, b = [torch.rand(s, generator=gen) * 2 - 1 for s in ((M, K), (K, N))]
    a *= torch.exp2(torch.randint(-45, 46, (M, 1), generator=gen).float())
    b *= torch.exp2(torch.randint(-18, 19, (1, N), generator=gen).float())
    a[:, 64:128] *= 2.0 ** -3
    b[128:192] = 0.0
    a[5], b[:, 6] = 0.0, 0.0
    a[7, 9:] = 0.0
    a, b = a.cuda(), b.cuda()
    ref = a.double() @ b.double()
    c, other = [torch.empty((M, N), device="cuda") for _ in range(2)]
    kern = _kernel(M, N, K, 256)
    kern.run(a, b, c)
    kern.checkStatus()
    _as_tf32(M, N, K, 256).run(a, b, other)
    assert not torch.equal(c, other)
    assert ((c.double() - ref).abs() <= _bound(a, b)).all()
    assert (c[5] == 0).all() and (c[:, 6] == 0).all()


@pytest.mark.gpu
def test_small_products_of_a_large_column():
    """A column near 2^40 whose other stretch of K is 2^-50 of that: a product near 2^-116 there, with nothing beside it."""
    M, N, K = 256, 256, 128
    gen = torch.Generator().manual_seed(10)
    a, b = [torch.rand(s, generator=gen) + 1 for s in ((M, K), (K, N))]
    b[64:] *= 2.0 ** -50
    b[:, 5] *= 2.0 ** 40
    a[9], b[64, 5] = 0.0, 0.0
    a[9, 64], a[9, 66], b[66, 5] = 2.0 ** -50, 1.25 * 2.0 ** -78, 1.5 * 2.0 ** -38
    a, b = a.cuda(), b.cuda()
    c = torch.empty((M, N), device="cuda")
    kern = _kernel(M, N, K, 256)
    kern.run(a, b, c)
    kern.checkStatus()
    assert ((c.double() - a.double() @ b.double()).abs() <= _bound(a, b)).all()


@pytest.mark.gpu
def test_a_remainder_cut_into_ranges_and_a_graph():
    """More tiles than run at once, the rest cut into K ranges, with a fused bias; captured, it keeps its own parts."""
    M, N, K = 3840, 2560, 1024
    assert tuned_config(M, N, K, E.float32).KERNEL_VARIANT == 6
    gen = torch.Generator(device="cuda").manual_seed(7)
    a, b = [torch.rand(s, generator=gen, device="cuda") * 2 - 1 for s in ((M, K), (K, N))]
    bias = torch.rand(N, generator=gen, device="cuda")
    want = matmul(a, b, bias=bias)
    ref = a.double() @ b.double() + bias.double()
    assert ((want.double() - ref).abs() <= _bound(a, b) + 2.0 ** -22).all()
    c, stream, graph = torch.empty_like(want), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        matmul(a, b, c, bias=bias)
    with torch.cuda.stream(stream):
        matmul(b[:, :1024].contiguous(), a[:1024].contiguous())  # the stream's own workspace
    c.fill_(float("nan"))
    graph.replay()
    assert torch.equal(c, want)
    a.view(-1)[0] = float("nan")
    graph.replay()
    assert c[0].isnan().all() and not c[1:].isnan().any()
    a.view(-1)[0] = 0.5
    ref = matmul(a, b, bias=bias)
    for _ in range(2):
        graph.replay()
        assert torch.equal(c, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["1", "3"])
def test_stream_k_asked_for(mode, monkeypatch):
    """More tiles than run at once, under the modes that lay K blocks end to end: values that split and values that do not."""
    monkeypatch.setenv("KCG_TAIL_SPLIT", mode)
    M, N, K = 2560, 2304, 1024
    gen = torch.Generator(device="cuda").manual_seed(9)
    a, b = [torch.rand(s, generator=gen, device="cuda") * 2 - 1 for s in ((M, K), (K, N))]
    kern = _kernel(M, N, K, 256)
    for _ in range(2):
        for value in (0.5, float("nan")):
            a[2559, 1000] = value
            c = torch.full((M, N), 7.0, device="cuda")
            kern.run(a, b, c)
            kern.checkStatus()
            ref = a.double() @ b.double()
            assert c[2559].isnan().all() or value == 0.5
            assert ((c.double() - ref).abs() <= _bound(a, b))[:2559].all()


@pytest.mark.gpu
def test_parts_larger_than_any_workspace():
    """4 GiB and more of parts: the product is taken as 3xTF32, with the same bits."""
    M, N, K = 1 << 19, 256, 2048
    a = torch.empty((M, K), device="cuda").uniform_(-1, 1, generator=torch.Generator(device="cuda").manual_seed(8))
    b = a[:K, :N].contiguous()
    c, want = [torch.empty((M, N), device="cuda") for _ in range(2)]
    kern = _kernel(M, N, K, 256)
    kern.run(a, b, c)
    kern.checkStatus()
    _as_tf32(M, N, K, 256).run(a, b, want)
    assert torch.equal(c, want)


def _spread(kind, gen):
    """Operands in which some values lie 2^-34 .. 2^-45 below the largest beside them (none is a power of two)."""
    M, N, K = 1280, 832, 1092
    a, b = [torch.rand(s, generator=gen) + 0.5 for s in ((M, K), (K, N))]
    small = lambda n: (torch.rand(n, generator=gen) + 0.5) * torch.exp2(-torch.randint(35, 46, (n,), generator=gen).float())
    if kind in ("a", "both"):  # of the first and the last panel of rows and chunk of K, many of one chunk
        for row, k in ((0, 3), (129, 64), (1279, 1091), (700, 640)):
            a[row, k] = small(1)[0]
        a[300:340, 100:110] = small(400).view(40, 10)
    if kind in ("b", "both"):
        for k, col in ((1, 2), (64, 100), (1091, 831), (641, 300)):
            b[k, col] = small(1)[0]
        b[684:700, 450:470] = small(320).view(16, 20)
    # a row and a column of small values alone but for one, which faces zeros
    a[300] = torch.where(a[300] > 1e-6, 0.0, a[300])
    b[:, 455] = torch.where(b[:, 455] > 1e-6, 0.0, b[:, 455])
    a[300, 64], b[64], b[640, 455], a[:, 640] = 1.0, 0.0, 1.0, 0.0
    return a.cuda(), b.cuda()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["a", "b", "both"])
@pytest.mark.parametrize("bn,split", [(128, 1), (128, 3), (256, 1), (256, 2)])
def test_far_parts(kind, bn, split):
    """A few chunks with values far below the largest beside them: multiplied once more, not the whole product as 3xTF32; every
    value as close as 3xTF32 guarantees, in every call and beside a fused epilogue, and the next call not affected."""
    gen = torch.Generator().manual_seed(21)
    a, b = _spread(kind, gen)
    (M, K), N = a.shape, b.shape[1]
    kern, other = _kernel(M, N, K, bn, split), _as_tf32(M, N, K, bn)
    c, tf32 = [torch.empty((M, N), device="cuda") for _ in range(2)]
    other.run(a, b, tf32)
    ref = a.double() @ b.double()
    bias = torch.rand(N, generator=gen).cuda()
    first = None
    for _ in range(3):
        c.fill_(float("nan"))
        kern.run(a, b, c)
        kern.checkStatus()
        assert ((c.double() - ref).abs() <= _bound(a, b)).all()
        assert first is None or torch.equal(c, first)  # whichever slots the chunks got
        first = c.clone()
    err = [float((t.double() - ref).norm() / ref.norm()) for t in (first, tf32)]
    assert err[0] < 0.6 * err[1], err  # (its own result, not 3xTF32's)
    assert (first[300].abs().max() > 0) == (kind != "b") and (first[:, 455].abs().max() > 0) == (kind != "a")
    kern.run(a, b, c, bias=bias, relu=True)
    assert torch.equal(c, (first + bias).clamp(min=0))
    plain = [t.clamp(min=0.25) for t in (a, b)]
    kern.run(*plain, c)
    kern.checkStatus()
    ref = plain[0].double() @ plain[1].double()
    assert ((c.double() - ref).abs() <= _bound(*plain)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("operand", ["a", "b"])
def test_more_far_values_than_slots(operand, monkeypatch):
    """Far values in every chunk, or below far values: the whole product as 3xTF32, bit for bit, and the next call as ever."""
    monkeypatch.setenv("KCG_TAIL_SPLIT", "0")  # (each kernel's own cuts into K ranges would sum in another order)
    M, N, K = 1280, 832, 1024
    gen = torch.Generator().manual_seed(22)
    plain = [(torch.rand(s, generator=gen) + 0.5).cuda() for s in ((M, K), (K, N))]
    kern, other = _kernel(M, N, K, 256), _as_tf32(M, N, K, 256)
    c, before, want = [torch.empty((M, N), device="cuda") for _ in range(3)]
    kern.run(*plain, before)
    for every in (True, False):
        a, b = [t.clone() for t in plain]
        x = a if operand == "a" else b
        if every:
            x[::64, ::64] = 1.2345678 * 2.0 ** -40
        elif operand == "a":
            x[9, 70:72] = torch.tensor([1.2345678 * 2.0 ** -34, 1.2345678 * 2.0 ** -70]).cuda()
        else:
            x[70:72, 9] = torch.tensor([1.2345678 * 2.0 ** -34, 1.2345678 * 2.0 ** -70]).cuda()
        other.run(a, b, want)
        kern.run(a, b, c)
        kern.checkStatus()
        assert torch.equal(c, want)
        kern.run(*plain, c)
        assert torch.equal(c, before)


@pytest.mark.gpu
def test_far_parts_in_a_graph():
    """Captured, with a remainder cut into ranges: chunks with far parts in one replay, none in the next, others after that."""
    M, N, K = 2560, 2304, 1024
    gen = torch.Generator(device="cuda").manual_seed(23)
    a, b = [torch.rand(s, generator=gen, device="cuda") + 0.5 for s in ((M, K), (K, N))]
    kern = _kernel(M, N, K, 256)
    c, want = [torch.empty((M, N), device="cuda") for _ in range(2)]
    kern.run(a, b, c)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        kern.run(a, b, c)
    for row, col, value in ((9, 3, 1.2345678e-12), (9, 3, 0.5), (2559, 1023, 1.2345678e-13), (2559, 1023, float("nan")), (2559, 1023, 0.5)):
        a[row, col] = b[col, row % N] = value
        graph.replay()
        kern.run(a, b, want)
        assert torch.equal(c.nan_to_num(nan=123.0), want.nan_to_num(nan=123.0))
        if value == value:
            assert ((c.double() - a.double() @ b.double()).abs() <= _bound(a, b)).all()
