"""Fused epilogues of the 3xTF32 kernels: whole tiles through one workspace slot per CTA (pair), remainder tiles cut into K
ranges behind them, as without an epilogue."""
import ctypes
import os
import subprocess

import pytest
import torch

from codegendemo_b200 import _lib
from codegendemo_b200.kcg.KCGCompiler import compile_info
from codegendemo_b200.kcg.matmul_op import bmm, build_kernel, default_config
from codegendemo_b200.kcg.Utils import EnumKernelDType as E

# M, N, K, variant, tile, {whole tiles, K ranges of the others}
CASES = [
    (128, 512, 4096, 2, (128, 64, 32), (0, 8)),      # remainder alone
    (256, 768, 1152, 2, (128, 64, 32), (0, 6)),      # a short K
    (128, 1792, 4096, 2, (128, 256, 16), (0, 8)),    # seven tiles of 256 columns
    (1280, 1024, 4096, 2, (128, 64, 32), (148, 8)),  # a wave of whole tiles, then twelve tiles cut up
    (2560, 2048, 2048, 4, (256, 256, 32), (74, 8)),  # the same on CTA pairs
    (5120, 2176, 256, 4, (256, 128, 32), (340, 1)),  # more whole tiles than slots, none cut up
    (1152, 1088, 4096, 2, (128, 64, 32), (148, 8)),  # 17 columns of tiles: the cut ones straddle rows
]


def _config(M, N, K, variant, tile):
    bm, bn, bk = tile
    return default_config(M, N, K, E.float32, KERNEL_VARIANT=variant, BLOCK_SIZE_M=bm, BLOCK_SIZE_N=bn, BLOCK_SIZE_K=bk,
                          EDGE_TILES=int(M % bm != 0 or N % bn != 0), NUM_STAGES=3 if bn == 256 else 4)


@pytest.mark.parametrize("case", CASES)
def test_the_plan_does_not_depend_on_an_epilogue(case):
    M, N, K, variant, tile, (first, factor) = case
    kpm = _config(M, N, K, variant, tile)
    info = compile_info(kpm.compileArgs(), num_stages=kpm.NUM_STAGES, kernel=kpm.KERNEL_VARIANT, edge_tiles=kpm.EDGE_TILES)
    lib = _lib.get_lib()
    lib.kcg_internal_plan_split.argtypes = [ctypes.POINTER(_lib.KernelInfo), ctypes.c_int, ctypes.c_int,
                                            ctypes.POINTER(ctypes.c_int)]
    plans = []
    for fused in (0, 1):
        out = (ctypes.c_int * 7)()
        assert lib.kcg_internal_plan_split(ctypes.byref(info), fused, 1, out) == 0
        plans.append(list(out))
    assert plans[0] == plans[1]
    assert plans[0][1:3] == [first, factor], plans[0]


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["bias_relu", "beta"])
@pytest.mark.parametrize("case", CASES)
def test_fused_products(case, form):
    M, N, K, variant, tile, _ = case
    _, kern = build_kernel(_config(M, N, K, variant, tile), 0)
    gen = torch.Generator(device="cuda").manual_seed(11)
    a, b, c0 = (torch.randn(s, generator=gen, device="cuda") for s in ((M, K), (K, N), (M, N)))
    bias = torch.randn(N, generator=gen, device="cuda")
    kw = dict(bias=bias, relu=True) if form == "bias_relu" else dict(alpha=0.5, beta=-2.0)
    product = a.double() @ b.double()
    want = torch.relu(product + bias.double()) if form == "bias_relu" else 0.5 * product - 2.0 * c0.double()
    # 3xTF32: products left out and rounded, sums of K terms and the epilogue's additions in fp32
    bound = 2.0 ** -20 * (a.double().abs() @ b.double().abs()) + 2.0 ** -22 * (bias.abs().max() + 2 * c0.double().abs())
    first = None
    for _ in range(3):  # slots, counters and partials of one launch are the next one's
        c = c0.clone() if form == "beta" else torch.full((M, N), float("nan"), device="cuda")
        kern.m_launcher.launchKernel(0, a, b, c, **kw)
        kern.checkStatus()
        assert (c.double() - want).abs().le(bound).all()
        assert first is None or torch.equal(c, first)  # summed in K order, whoever comes last
        first = c


@pytest.mark.gpu
def test_fused_batches():
    gen = torch.Generator(device="cuda").manual_seed(12)
    a, b = torch.randn(3, 128, 2048, generator=gen, device="cuda"), torch.randn(3, 2048, 384, generator=gen, device="cuda")
    bias = torch.randn(384, generator=gen, device="cuda")
    c = bmm(a, b, bias=bias, relu=True)
    want = torch.relu(a.double() @ b.double() + bias.double())
    assert (c.double() - want).abs().le(2.0 ** -20 * (a.double().abs() @ b.double().abs()) + 2.0 ** -22 * bias.abs().max()).all()


@pytest.mark.parametrize("mode", [None, "0", "1", "2", "3", "4", "5"])
def test_slots_lie_inside_the_workspace(mode, tmp_path, monkeypatch):
    """Every tile of a fused launch passes through a slot that the launch has memory for: fewer whole tiles than CTAs, more,
    none, and K blocks laid end to end."""
    if mode is None:
        monkeypatch.delenv("KCG_TAIL_SPLIT", raising=False)
    else:
        monkeypatch.setenv("KCG_TAIL_SPLIT", mode)
    lib = _lib.get_lib()
    for f in (lib.kcg_internal_plan_split, lib.kcg_internal_launch_slots):
        f.argtypes = [ctypes.POINTER(_lib.KernelInfo), ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int)]
    tests = os.path.dirname(os.path.abspath(__file__))
    kernels = os.path.join(os.path.dirname(tests), "codegendemo_b200", "csrc", "kernels")
    programs, wholes = {}, []
    more = [(4096, 4096, 2048, 4, (256, 256, 32), None), (3456, 768, 1408, 2, (128, 128, 32), None),
            (2048, 4096, 4096, 4, (256, 128, 32), None), (256, 256, 512, 4, (256, 128, 32), None)]
    for M, N, K, variant, tile, _ in CASES + more:
        kpm = _config(M, N, K, variant, tile)
        info = compile_info(kpm.compileArgs(), num_stages=kpm.NUM_STAGES, kernel=kpm.KERNEL_VARIANT, edge_tiles=kpm.EDGE_TILES)
        plan, slots = (ctypes.c_int * 7)(), (ctypes.c_int * 3)()
        assert lib.kcg_internal_plan_split(ctypes.byref(info), 1, 1, plan) == 0
        assert lib.kcg_internal_launch_slots(ctypes.byref(info), 1, 1, slots) == 0
        if tile not in programs:
            programs[tile] = str(tmp_path / "x".join(map(str, tile)))
            subprocess.run(["g++", "-O1", "-std=c++17", "-I/usr/local/cuda/include", "-I" + kernels, "-o", programs[tile],
                            os.path.join(tests, "slot_check.cpp")] + [f"-DSC_B{d}={v}" for d, v in zip("MNK", tile)], check=True)
        r = subprocess.run([programs[tile]] + [str(v) for v in (M, N, K, plan[1], plan[2], plan[3], *slots)], capture_output=True, text=True)
        assert r.returncode == 0, (M, N, K, tile, list(plan), list(slots), r.stdout + r.stderr)
        wholes.append(int(r.stdout.split()[1]))
        slots_plain = (ctypes.c_int * 3)()
        assert lib.kcg_internal_launch_slots(ctypes.byref(info), 0, 1, slots_plain) == 0
        assert slots_plain[2] == 0 and list(slots_plain[:2]) == list(slots[:2])
    assert 0 in wholes or mode == "0"
    assert max(wholes) > 148
