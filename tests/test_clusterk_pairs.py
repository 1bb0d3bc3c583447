"""Cluster split-K on CTA pairs (KERNEL_VARIANT 5 with BLOCK_SIZE_M = 256), and the extension module that launches."""
import pytest
import torch

from codegendemo_b200 import _lib
from codegendemo_b200.kcg.KCGCompiler import compile_info
from codegendemo_b200.kcg.matmul_op import _CLUSTERS, build_kernel, default_config, tuned_config
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
# the shortest (one block of 128 a range); past the ring with equal ranges, the last block half (64) or three quarters (128)
# full; an odd number of blocks past the ring, hence unequal ranges, of 64 (10 + 9) and of both (17 + 16, 9 + 8), the last
# one half full (a quarter of 128 at 1184)
@pytest.mark.parametrize("K", [256, 1248, 1184, 2112, 4096])
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


class _NoDb:
    def lookup(self, *shape):
        return None


def _rule(M, N, K):
    kpm = tuned_config(M, N, K, E.bfloat16, db=_NoDb())
    return (kpm.KERNEL_VARIANT, kpm.BLOCK_SIZE_M, kpm.BLOCK_SIZE_N, kpm.LOCAL_SPLIT_U)


def test_rule_counts_the_clusters_that_run_at_once():
    """Of 44 clusters of three some start late: two ranges of narrower tiles are ahead (256x4224x11008 31.9 / 28.8 us). 42
    run at once: there the three ranges are (384x3584x11008 30.1 / 37.6). No choice is left with a second wave of clusters."""
    for K in (9216, 11008, 14336):
        assert _rule(256, 4224, K) == (5, 128, 128, 2)
    assert _rule(384, 3584, 11008) == (5, 128, 256, 3)
    for M in (128, 256, 384, 512, 640):
        for N in range(512, 8193, 64):
            for K in (2048, 4096, 8192):
                variant, bm, bn, split = _rule(M, N, K)
                if variant == 5:
                    assert -(-M // bm) * -(-N // bn) <= _CLUSTERS[split * bm // 128], (M, N, K)


def test_rule_takes_pairs_from_four_blocks_a_range_on():
    """K = 768: 64 columns a CTA are ahead of CTA pairs (512x2048 5.9 / 6.5 us); at 1024 and more pairs are chosen."""
    for M, N in ((256, 3072), (512, 2048), (896, 896), (1280, 768), (768, 1344), (256, 8192)):
        for K in (512, 640, 704, 768, 896, 960):
            variant, bm, _, _ = _rule(M, N, K)
            assert not (variant == 5 and bm == 256), (M, N, K)
    for K in (1024, 1536, 2048):
        assert _rule(512, 2048, K) == (5, 256, 128, 2)


@pytest.mark.gpu
@pytest.mark.parametrize("bn,bk,stages", [(128, 64, 3), (128, 128, 2), (256, 64, 4)])
def test_pairs_that_share_an_sm(bn, bk, stages):
    """Short rings leave room for several CTAs on an SM, and more clusters than fit come and go: a pair's tensor memory is
    taken by the next CTA as soon as it is given back, so neither half may still read its accumulator by then. Launches that
    follow one another without a wait, two kernels in turn on two streams, give the bits of launches one at a time."""
    M = N = 2048
    K = 320
    a, b = [x.cuda() for x in oracle.make_inputs(M, N, K, torch.bfloat16, "normal", seed=3)]
    _, kern = build_kernel(_cfg(M, N, K, bn, bk, NUM_STAGES=stages), 0)
    _, other = build_kernel(default_config(M, N, K, E.bfloat16, KERNEL_VARIANT=2, BLOCK_SIZE_N=64, BLOCK_SIZE_K=64,
                                           NUM_STAGES=2), 0)
    alone = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    kern.run(a, b, alone)
    kern.checkStatus()
    err = oracle.rel_errors(alone, oracle.host_matmul(a.cpu(), b.cpu()))
    assert err["max_rel"] <= oracle.tolerance_for(torch.bfloat16)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = [torch.full((2, M, N), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(8)]
    torch.cuda.synchronize()
    for c in outs:
        for s in streams:
            with torch.cuda.stream(s):
                kern.run(a, b, c[0] if s is streams[0] else c[1])
                other.run(a, b, torch.empty((M, N), dtype=torch.bfloat16, device="cuda"))
    torch.cuda.synchronize()
    kern.checkStatus()
    for c in outs:
        assert torch.equal(c[0], alone) and torch.equal(c[1], alone)
