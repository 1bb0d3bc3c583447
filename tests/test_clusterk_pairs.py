"""Cluster split-K on CTA pairs (KERNEL_VARIANT 5 with BLOCK_SIZE_M = 256), and the extension module that launches."""
import pytest
import torch

from codegendemo_b200 import _lib
from codegendemo_b200.kcg.KCGCompiler import compile_info
from codegendemo_b200.kcg.matmul_op import build_kernel, default_config
from codegendemo_b200.kcg.Utils import EnumKernelDType as E
from oracle import oracle


def _cfg(M, N, K, bn, bk, **keys):
    return default_config(M, N, K, E.bfloat16, KERNEL_VARIANT=5, BLOCK_SIZE_M=256, BLOCK_SIZE_N=bn, BLOCK_SIZE_K=bk,
                          LOCAL_SPLIT_U=2, EDGE_TILES=1, **keys)


def test_config():
    info = compile_info(_cfg(512, 4096, 4096, 256, 64).compileArgs(), kernel=5, edge_tiles=1)
    assert list(info.cluster) == [4, 1, 1] and info.grid[0] == 2 * 16 * 4 and info.block[0] == 192 and info.splitk == 2
    assert info.smem_bytes == info.stages * (128 + 128) * 64 * 2 + 2048 <= 227 * 1024
    for bad in (dict(LOCAL_SPLIT_U=3), dict(BLOCK_SIZE_N=64), dict(BLOCK_SIZE_M=512)):
        kpm = _cfg(512, 4096, 4096, 256, 64)
        for k, v in bad.items():
            setattr(kpm, k, v)
        with pytest.raises(_lib.KCGError):
            compile_info(kpm.compileArgs(), kernel=5, edge_tiles=1)


@pytest.mark.gpu
@pytest.mark.parametrize("bn,bk", [(128, 64), (128, 128), (256, 64), (256, 128)])
# one K block a range; an odd number of blocks (ranges of unequal length), the last one half full; past the ring
@pytest.mark.parametrize("K", [256, 1248, 4096])
def test_matches_the_oracle(bn, bk, K):
    M, N = 384, 320
    a, b = oracle.make_inputs(M, N, K, torch.bfloat16, "normal", seed=9)
    ref = oracle.host_matmul(a, b)
    for a_trans in (0, 1):
        _, kern = build_kernel(_cfg(M, N, K, bn, bk, isATranspose=a_trans), 0)
        c = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
        kern.run((a.t().contiguous() if a_trans else a).cuda(), b.cuda(), c)
        kern.checkStatus()
        err = oracle.rel_errors(c, ref)
        assert err["max_rel"] <= oracle.tolerance_for(torch.bfloat16) and err["allclose_ref"], (a_trans, err)


@pytest.mark.gpu
def test_batched():
    batch, M, N, K = 3, 512, 192, 640
    gen = torch.Generator().manual_seed(3)
    a, b = [(torch.randn(s, generator=gen) / K ** 0.25).to(torch.bfloat16) for s in ((batch, M, K), (batch, K, N))]
    for bn, bk in ((128, 128), (256, 64)):
        _, kern = build_kernel(_cfg(M, N, K, bn, bk), 0)
        c = torch.full((batch, M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
        kern.run(a.cuda(), b.cuda(), c, batch=batch)
        kern.checkStatus()
        for i in range(batch):
            err = oracle.rel_errors(c[i], oracle.host_matmul(a[i], b[i]))
            assert err["max_rel"] <= oracle.tolerance_for(torch.bfloat16), (bn, i, err)


def test_launch_module_checks_its_arguments():
    _lib.get_lib()
    call = _lib.pycall.gemm
    rest = (0, 0, 0, 1, 1.0, 0.0, None, False)
    for bad in (None, 1.5, "x"):
        with pytest.raises(TypeError):
            call(0, 0, 0, 0, bad, 1, 1, *rest)
    with pytest.raises(TypeError):
        call(0, 0, 0, 0, 1, 1)
    with pytest.raises((OverflowError, TypeError)):
        call(0, 0, 0, 0, -1, 1, 1, *rest)
    assert call(0, 0, 0, 0, 16, 16, 16, *rest) == _lib.E_BAD_ARG  # no kernel: the library's own check
    assert _lib.pycall.attention(0, 0, 0, 16, 16, 16, 62, 1, 1, 1, 64, 0.1) == _lib.E_BAD_ARG
