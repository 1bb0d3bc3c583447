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
