"""3xTF32 kernels whose A operand goes through tensor memory (tiles of up to 192 columns): the same products in the same
order as the form that keeps A in shared memory, so the results are compared bit for bit with that form's."""
import pytest
import torch

from codegendemo_b200.kcg.matmul_op import build_kernel, default_config
from codegendemo_b200.kcg.Utils import EnumKernelDType as E

# (KERNEL_VARIANT, BLOCK_SIZE_M, N, K, stages): one and two CTAs, two, three and four K blocks in tensor memory, both
# swizzles of a 16- and a 32-wide K block; fewer stages than would fit
TILES = [(2, 128, 64, 32, 6), (2, 128, 128, 32, 3), (2, 128, 192, 32, 2), (2, 128, 128, 16, 4), (4, 256, 128, 32, 6),
         (4, 256, 128, 16, 2), (4, 256, 192, 32, 5), (4, 256, 192, 16, 8)]
SHARED_A = (2, 256, 64, 32, 2)  # two accumulators a CTA: A stays in shared memory


def _run(tile, a, b, N, a_trans):
    K, M = a.shape if a_trans else a.shape[::-1]
    kpm = default_config(M, N, K, E.float32, KERNEL_VARIANT=tile[0], BLOCK_SIZE_M=tile[1], BLOCK_SIZE_N=tile[2],
                         BLOCK_SIZE_K=tile[3], NUM_STAGES=tile[4], isATranspose=int(a_trans), EDGE_TILES=1)
    _, kern = build_kernel(kpm, 0)
    c = torch.full((M, N), float("nan"), device="cuda")
    kern.run(a, b, c)
    kern.checkStatus()
    return c


@pytest.mark.gpu
@pytest.mark.parametrize("a_trans", [False, True], ids=["MxK", "KxM"])
# one block of K, fewer than the tensor memory holds, past every ring; the last block of K and the last tiles hang over
@pytest.mark.parametrize("shape", [(128, 64, 32), (256, 192, 80), (384, 320, 1104)], ids=lambda s: "x".join(map(str, s)))
def test_same_bits_as_with_a_in_shared_memory(shape, a_trans, monkeypatch):
    M, N, K = shape
    monkeypatch.setenv("KCG_TAIL_SPLIT", "0")  # K ranges, which depend on the tile, would be summed in another order
    gen = torch.Generator().manual_seed(4)
    a = (torch.rand((M, K), generator=gen) * 2 - 1).cuda()
    b = (torch.rand((K, N), generator=gen) * 2 - 1).cuda()
    if a_trans:
        a = a.t().contiguous()
    want = _run(SHARED_A, a, b, N, a_trans)
    ref = (a.double().t() if a_trans else a.double()) @ b.double()
    # 3xTF32 drops 2^-22 of a product and sums in fp32: 2^-20 of the norms' product bounds both at these K
    assert ((want.double() - ref).abs() <= 2.0 ** -20 * (ref.abs() + K ** 0.5)).all()
    for tile in TILES:
        assert torch.equal(_run(tile, a, b, N, a_trans), want), tile


@pytest.mark.gpu
def test_extreme_values():
    """The lo part of an infinite or NaN value is NaN, and so is every result it enters; values near the ends of the
    exponent range split exactly, and other rows and columns do not notice."""
    M, N, K = 256, 192, 96
    gen = torch.Generator().manual_seed(6)
    a = (torch.rand((M, K), generator=gen) * 2 - 1)
    b = (torch.rand((K, N), generator=gen) * 2 - 1)
    a[3, 5], a[7, 9], a[11, 0] = float("inf"), float("-inf"), float("nan")
    b[2, 17] = float("inf")
    a[20], a[21] = 0.0, 0.0
    a[20, 1], a[21, 1] = 3.3e38, 1.5e-30
    b[1] *= 0.01
    bad = torch.zeros((M, N), dtype=torch.bool)
    bad[[3, 7, 11]] = True
    bad[:, 17] = True
    ref = a.double() @ b.double()
    for tile in [SHARED_A] + TILES:
        c = _run(tile, a.cuda(), b.cuda(), N, False).cpu()
        assert torch.equal(c.isnan(), bad), tile
        ok = ~bad
        err = (c.double() - ref).abs()
        # (rows 20 and 21: one product each, exact but for the dropped lo*lo and three roundings)
        bound = 2.0 ** -20 * (a.double().abs() @ b.double().abs()) + 1e-37
        assert (err[ok] <= bound[ok]).all(), tile
