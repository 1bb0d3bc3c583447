"""Which kernel the Python operators pick and keep for a call."""
import pytest
import torch

from codegendemo_b200.kcg import matmul_op


class _Stub:
    """Stands for a compiled kernel: remembers its config, launches nothing."""

    def __init__(self, kpm):
        self.kpm, self.launches = kpm, []
        self.m_launcher = self

    def launchKernel(self, dev, a, b, c, **kw):
        self.launches.append(kw)


@pytest.fixture
def stubs(monkeypatch):
    made = []

    def build(kpm, dev=0):
        kpm.check()
        made.append(_Stub(kpm))
        return None, made[-1]
    monkeypatch.setattr(matmul_op, "build_kernel", build)
    monkeypatch.setattr(matmul_op, "_KERNELS", {})
    return made


@pytest.mark.parametrize("bmm_first", [False, True])
def test_a_batch_of_one_and_a_transposed_b_do_not_share_a_kernel(stubs, bmm_first):
    x = torch.zeros((256, 256), dtype=torch.bfloat16)
    calls = [lambda: matmul_op.matmul(x, x, b_transposed=True), lambda: matmul_op.bmm(x[None], x[None])]
    for call in calls[::-1] if bmm_first else calls:
        call()
    assert [len(k.launches) for k in stubs] == [1, 1]
    assert sorted(k.kpm.IS_BTRANS for k in stubs) == [0, 1]


def test_a_stored_config_that_cannot_read_a_transposed_b_gives_way():
    """The kernel database may hold an FFMA config for a 16-bit shape; b_transposed then takes the rule's tile."""
    from codegendemo_b200.kcg.KCGCompiler import compile_info
    from codegendemo_b200.kcg.Utils import EnumKernelDType as E

    class Db:
        def lookup(self, *key):
            simt = dict(KERNEL_VARIANT=1, BLOCK_SIZE_M=128, BLOCK_SIZE_N=128, BLOCK_SIZE_K=16, THREAD_SIZE_M=8,
                        THREAD_SIZE_N=8, WARP_SCATTER_WIDTH_A=4, WARP_SCATTER_WIDTH_B=4, THREAD_SCATTER_WIDTH_A=4,
                        THREAD_SCATTER_WIDTH_B=4)
            return {"config": matmul_op.default_config(256, 256, 256, E.bfloat16, **simt).jsonfy()}
    assert matmul_op.tuned_config(256, 256, 256, E.bfloat16, db=Db()).KERNEL_VARIANT == 1
    kpm = matmul_op.tuned_config(256, 256, 256, E.bfloat16, db=Db(), b_transposed=True)
    kpm.check()
    assert kpm.KERNEL_VARIANT in (2, 4, 5) and kpm.IS_BTRANS == 1
    compile_info(kpm.compileArgs(), num_stages=kpm.NUM_STAGES, kernel=kpm.KERNEL_VARIANT, b_trans=1,
                 edge_tiles=kpm.EDGE_TILES)


# heads, queries, keys, head dimension of the three-launch attention; the first two are where the rule over all kernels
# prefers the cluster split-K kernel for a product
ATTENTION = [(8, 512, 2048, 128), (32, 128, 8192, 128), (16, 2048, 2048, 128), (4, 128, 1024, 64), (1, 384, 320, 64),
             (2, 256, 192, 64)]


def test_attention_takes_the_best_single_pass_tile():
    from codegendemo_b200.kcg.Utils import EnumKernelDType as E
    for heads, sq, sk, d in ATTENTION:
        for m, n, k, scores in ((sq, sk, d, True), (sq, d, sk, False)):
            kpm = matmul_op._attention_tile(heads, m, n, k, E.bfloat16, scores)
            kpm.check()
            tile = (kpm.KERNEL_VARIANT or 2, kpm.BLOCK_SIZE_M, kpm.BLOCK_SIZE_N, kpm.BLOCK_SIZE_K)
            best = matmul_op._cheapest_tile(m, n, k, heads, single_pass=True)[0]
            assert tile[0] in (2, 4) and kpm.IS_BTRANS == int(scores)
            assert matmul_op._tile_us(tile, 1, m, n, k, heads) <= 1.1 * best, (heads, m, n, k)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", ATTENTION, ids=lambda s: "x".join(map(str, s)))
def test_attention_in_three_launches(shape):
    heads, sq, sk, d = shape
    gen = torch.Generator().manual_seed(2)
    q, k, v = [torch.randn((heads, n, d), generator=gen).to(torch.bfloat16) for n in (sq, sk, sk)]
    out = matmul_op.attention(q.cuda(), k.cuda(), v.cuda()).cpu().double()
    p = torch.softmax(q.double() @ k.double().transpose(1, 2) * d ** -0.5, dim=-1)
    # probabilities and the result are each rounded once to bf16: half a unit each; 32-bit sums far below that
    bound = 2.0 ** -8 * (p @ v.double()).abs() + 2.0 ** -8 * (p @ v.double().abs()) + 1e-5
    assert ((out - p @ v.double()).abs() <= bound).all()


@pytest.mark.gpu
@pytest.mark.parametrize("bmm_first", [False, True])
def test_a_batch_of_one_and_a_transposed_b_on_one_shape(bmm_first, monkeypatch):
    monkeypatch.setattr(matmul_op, "_KERNELS", {})
    gen = torch.Generator().manual_seed(1)
    a, b = [(torch.randn((256, 256), generator=gen) / 16).to(torch.bfloat16).cuda() for _ in range(2)]
    calls = [(lambda: matmul_op.matmul(a, b, b_transposed=True), b.t()), (lambda: matmul_op.bmm(a[None], b[None])[0], b)]
    for call, right in calls[::-1] if bmm_first else calls:
        # one rounding to bf16 (half a unit), and 32-bit sums far below it
        ref = a.double() @ right.double()
        assert ((call().double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5).all()
