"""The 256-row fused attention kernel where its maxima, its last steps and its second query tile can go wrong."""
import pytest
import torch


def _reference(q, k, v, scale):
    p = torch.softmax(q.double() @ k.double().transpose(1, 2) * scale, dim=-1)
    return p @ v.double()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
# one step; keys that end in each of a step's four pieces; an odd number of steps; a second tile of one row or none
@pytest.mark.parametrize("shape", [(3, 256, 128, 128), (2, 129, 1, 64), (2, 128, 33, 128), (2, 257, 193, 64),
                                   (1, 300, 353, 128), (2, 255, 384, 128)], ids=lambda s: "x".join(map(str, s)))
def test_rows_match_the_composition_in_64_bits(shape, dtype):
    from codegendemo_b200.kcg.matmul_op import attention_fused, attention_status
    heads, sq, sk, d = shape
    gen = torch.Generator().manual_seed(3)
    q, k, v = [torch.randn((heads, n, d), generator=gen).to(dtype) for n in (sq, sk, sk)]
    out = torch.full((heads, sq, d), float("nan"), dtype=dtype, device="cuda")
    attention_fused(q.cuda(), k.cuda(), v.cuda(), out=out)
    attention_status(0)
    # probabilities and the result are each rounded once to 16 bits (half a unit of the largest value, twice)
    half_unit = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12
    assert (out.cpu().double() - _reference(q, k, v, d ** -0.5)).abs().max().item() <= 2.1 * half_unit * v.abs().max().item()


@pytest.mark.gpu
@pytest.mark.parametrize("step", [0.02, 0.5, 7.9, 8.1, 40.0])
def test_maximum_that_climbs_with_every_step(step):
    """Scores that grow by `step` (in the exp2 domain) from one 128-key step to the next, in some rows only: the
    maximum moves by a little or a lot, and O and the sums follow."""
    from codegendemo_b200.kcg.matmul_op import attention_fused, attention_status
    heads, sq, sk, d = 2, 256, 1280, 64
    gen = torch.Generator().manual_seed(4)
    q, k, v = [0.1 * torch.randn((heads, n, d), generator=gen) for n in (sq, sk, sk)]
    q[:, :, 0] = 1.0
    q[:, 1::3, 0] = -1.0
    q[:, 2::3, 0] = 0.0
    k[:, :, 0] = (torch.arange(sk) // 128 * step * 0.6931471805599453)[None]
    q, k, v = q.half(), k.half(), v.half()
    out = attention_fused(q.cuda(), k.cuda(), v.cuda(), scale=1.0)
    attention_status(0)
    assert (out.cpu().double() - _reference(q, k, v, 1.0)).abs().max().item() <= 2.1 * 2.0 ** -12 * v.abs().max().item()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("sk", [512, 4096], ids=["whole", "key_split"])
def test_the_largest_probability_is_not_rounded(sk, dtype):
    """Two keys carry all the weight, and the larger one comes later by 0.3 to 7.8 in the exp2 domain: taken against the
    running maximum its probability is 1 in 16 bits as well, so only the smaller one and the result are rounded."""
    from codegendemo_b200.kcg.matmul_op import attention_fused
    heads, sq, d = 16, 128, 128
    gen = torch.Generator().manual_seed(6)
    v = torch.randn((heads, sk, d), generator=gen).to(dtype)
    q, k = torch.zeros((heads, sq, d), dtype=dtype), torch.zeros((heads, sk, d), dtype=dtype)
    q[:, :, 0] = 1.0
    k[:, :, 0] = -200.0
    k[:, 5, 0] = 0.0
    k[:, 300, 0] = (0.3 + 0.5 * torch.arange(heads)) * 0.6931471805599453
    out = attention_fused(q.cuda(), k.cuda(), v.cuda(), scale=1.0).cpu().double()
    p = torch.softmax(q.double() @ k.double().transpose(1, 2), dim=-1)
    ref = p @ v.double()
    half_unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    # half a unit of the result and of the smaller probability; the 32-bit part (exponentials, sums, the joining of
    # the CTAs' parts) within 2^-18 of the largest value
    bound = half_unit * (ref.abs() + p[:, :, 5:6] * v[:, 5:6].double().abs()) + 2.0 ** -18 * v.abs().max().item()
    assert ((out - ref).abs() <= bound).all()


@pytest.mark.gpu
# one CTA per 256 rows, and 2 to 8 that share its keys; the few-row form; excluded: whole first or last ranges of a CTA
@pytest.mark.parametrize("shape", [(2, 128, 512), (2, 300, 4096), (2, 1, 4096), (2, 20, 4096), (2, 40, 2048)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("first", [True, False])
def test_keys_of_minus_infinity_weigh_nothing(shape, first):
    from codegendemo_b200.kcg.matmul_op import attention_fused
    heads, sq, sk = shape
    gen = torch.Generator().manual_seed(8)
    q, k, v = [torch.randn((heads, n, 64), generator=gen) for n in (sq, sk, sk)]
    q[:, :, 0] = 1.0
    k[:, :sk // 2 + 60, 0] = -float("inf")
    if not first:
        k = k.flip(1)
    q, k, v = q.half(), k.half(), v.half()
    out = attention_fused(q.cuda(), k.cuda(), v.cuda()).cpu().double()
    # probabilities and the result are each rounded once to 16 bits (half a unit of the largest value, twice)
    assert (out - _reference(q, k, v, 64 ** -0.5)).abs().max().item() <= 2.1 * 2.0 ** -12 * v.abs().max().item()


@pytest.mark.gpu
def test_nan_and_infinite_scores_stay_in_their_rows():
    from codegendemo_b200.kcg.matmul_op import attention_fused
    gen = torch.Generator().manual_seed(5)
    q, k, v = [torch.randn((2, n, 64), generator=gen).bfloat16() for n in (256, 512, 512)]
    clean = attention_fused(q.cuda(), k.cuda(), v.cuda()).cpu()
    q[0, 5, 3] = float("nan")
    q[1, 200, 3] = float("inf")
    out = attention_fused(q.cuda(), k.cuda(), v.cuda()).cpu()
    assert out[0, 5].isnan().all() and out[1, 200].isnan().all()
    clean[0, 5] = out[0, 5]
    clean[1, 200] = out[1, 200]
    assert torch.equal(out.nan_to_num(7.0), clean.nan_to_num(7.0))


@pytest.mark.gpu
# groups of 256 rows that do not fill a wave share their keys among 2 to 8 CTAs; 150 and 220 groups: whole groups and a
# remainder behind them; a last CTA whose only step has one key; a group of one row; too few keys to share
@pytest.mark.parametrize("shape", [(2, 300, 4097, 128), (1, 65, 8000, 64), (20, 257, 1100, 128), (150, 100, 1025, 64),
                                   (55, 1000, 2049, 128), (40, 256, 1024, 128), (3, 256, 1023, 64)],
                         ids=lambda s: "x".join(map(str, s)))
def test_groups_that_share_their_keys(shape):
    from codegendemo_b200.kcg.matmul_op import attention_fused, attention_status
    heads, sq, sk, d = shape
    gen = torch.Generator(device="cuda").manual_seed(9)
    q, k, v = [torch.randn((heads, n, d), generator=gen, device="cuda").bfloat16() for n in (sq, sk, sk)]
    k[:, sk // 2:] *= 3.0  # the later keys' maxima are the larger ones
    out = torch.full((heads, sq, d), float("nan"), dtype=torch.bfloat16, device="cuda")
    attention_fused(q, k, v, out=out)
    # ordered behind both launches: a copy, and the same call over the same buffer
    copy = out.clone()
    attention_fused(q, k, v, out=out)
    attention_status(0)
    assert torch.equal(copy, out)
    bound = 2.1 * 2.0 ** -9 * v.abs().max().item()  # two roundings to 16 bits, of the probabilities and the result
    for h in range(0, heads, max(1, heads // 8)):
        ref = _reference(q[h:h + 1], k[h:h + 1], v[h:h + 1], d ** -0.5)
        assert (out[h:h + 1].double() - ref).abs().max().item() <= bound
    last = heads - 1
    ref = _reference(q[last:], k[last:], v[last:], d ** -0.5)
    assert (out[last:].double() - ref).abs().max().item() <= bound
