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
