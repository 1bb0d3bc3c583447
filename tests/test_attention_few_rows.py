"""The fused attention entry at few query rows, where a head's keys are shared by the CTAs of a cluster."""
import ctypes
import os
import subprocess
import sys

import pytest
import torch

from codegendemo_b200 import _lib

# (heads, sq, sk, d) of the few-row form: one row and one key; the last row group full, one short, one past it (16, 32,
# 64 rows per kernel form); a last stage of one key; fewer stages than warps or CTAs; a cluster of 16, an odd one, one CTA
# per head; a warp whose keys are all past the end; 33 to 64 rows at every line of the rule that admits them
FEW = [(1, 1, 1, 128), (3, 1, 63, 64), (2, 16, 64, 128), (2, 17, 65, 128), (5, 15, 129, 64), (2, 32, 1000, 128),
       (8, 5, 16384, 128), (8, 3, 8209, 64), (40, 2, 3001, 128), (100, 7, 300, 64), (300, 1, 513, 128),
       (2, 33, 4097, 64), (64, 63, 700, 64), (130, 50, 512, 64), (4, 64, 2049, 128), (5, 47, 513, 128), (8, 63, 3071, 128),
       (9, 34, 2047, 128), (33, 64, 1537, 128), (88, 49, 1536, 128)]
# their neighbours on the other side of each line, which the 256-row kernel takes
MANY = [(4, 65, 2049, 128), (2, 33, 511, 64), (5, 47, 511, 128), (8, 63, 3072, 128), (9, 34, 2048, 128),
        (33, 64, 1535, 128), (89, 49, 1536, 128)]
SHAPES = FEW + MANY


def test_the_shapes_lie_on_their_side_of_the_rule():
    few = _lib.get_lib().kcg_internal_attention_few_rows
    few.argtypes = [ctypes.c_int] * 4
    assert [few(*s) for s in SHAPES] == [1] * len(FEW) + [0] * len(MANY)


def test_no_larger_cluster_than_fits():
    """On a whole GPU up to 16 CTAs share a head's keys; where larger clusters do not fit, the largest that does."""
    splits = _lib.get_lib().kcg_internal_attention_splits
    splits.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_uint]
    assert [splits(h, 16384, 0x1ffff) for h in (1, 8, 12, 20, 32, 100, 140, 300)] == [16, 16, 16, 10, 8, 2, 2, 1]
    assert [splits(h, 16384, 0x1ff) for h in (1, 8, 12, 20, 32, 100, 140, 300)] == [8, 8, 8, 8, 8, 2, 2, 1]
    assert [splits(8, 16384, mask) for mask in (0b1011111, 0b111, 0b1, 0)] == [6, 2, 1, 1]


_EDGES = """
import ctypes, torch
from codegendemo_b200.kcg.matmul_op import attention_fused
q, k, v = [torch.zeros((h, n, 64), dtype=torch.float16, device="cuda") for h, n in ((150, 256), (150, 1024), (150, 1024))]
few = q[:, :1].contiguous()
for x in (few, q):
    attention_fused(x, k, v)
graph = torch.cuda.CUDAGraph(keep_graph=True)
with torch.cuda.graph(graph):
    for x in (few, few, q):  # (the last: whole groups, and a remainder of two that share their keys, behind them)
        attention_fused(x, k, v)
edges = ctypes.CDLL("libcuda.so.1").cuGraphGetEdges_v2
n = ctypes.c_size_t(8)
ends, data = [(ctypes.c_void_p * 8)() for _ in range(2)], (ctypes.c_ubyte * 64)()  # 8 bytes an edge, its type the third
assert edges(ctypes.c_void_p(graph.raw_cuda_graph()), *ends, data, ctypes.byref(n)) == 0 and n.value == 3, n
print(sum(data[8 * i + 2] == 1 for i in range(3)))  # CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC
"""


@pytest.mark.gpu
@pytest.mark.parametrize("pdl,programmatic", [("1", 2), ("0", 0)])
def test_programmatic_launch_can_be_turned_off(pdl, programmatic):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _EDGES], cwd=root, env=dict(os.environ, KCG_PDL=pdl), text=True,
                       capture_output=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert int(r.stdout.split()[-1]) == programmatic


def _inputs(heads, sq, sk, d, dtype, seed=7):
    gen = torch.Generator().manual_seed(seed)
    return [torch.randn((heads, n, d), generator=gen).to(dtype) for n in (sq, sk, sk)]


def _reference(q, k, v, scale):
    p = torch.softmax(q.double() @ k.double().transpose(1, 2) * scale, dim=-1)
    return p @ v.double()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_few_rows_match_the_composition_in_64_bits(shape, dtype):
    from codegendemo_b200.kcg.matmul_op import attention_fused, attention_status
    heads, sq, sk, d = shape
    q, k, v = _inputs(heads, sq, sk, d, dtype)
    out = torch.full((heads, sq, d), float("nan"), dtype=dtype, device="cuda")
    attention_fused(q.cuda(), k.cuda(), v.cuda(), out=out)
    attention_status(0)
    ref = _reference(q, k, v, d ** -0.5)
    # probabilities and the result are each rounded once to 16 bits: half a unit of the largest value, twice; the
    # 32-bit sums and exponentials stay two orders below that
    half_unit = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12
    bound = 2.1 * half_unit * v.abs().max().item()
    assert (out.cpu().double() - ref).abs().max().item() <= bound
    again = torch.empty_like(out)
    attention_fused(q.cuda(), k.cuda(), v.cuda(), out=again)
    assert torch.equal(out, again)


@pytest.mark.gpu
@pytest.mark.parametrize("sq", [1, 20, 64])
def test_few_rows_and_extreme_scores(sq):
    """Scores of +-2000 (all weight on one key of a late stage), and a NaN key: the rows that see it are NaN."""
    from codegendemo_b200.kcg.matmul_op import attention_fused
    q, k, v = _inputs(2, sq, 1500, 64, torch.bfloat16)
    q[:] = 0
    q[:, :, 0] = 2000.0
    k[:] = 0
    k[:, :, 0] = -1.0
    k[:, 1441, 0] = 1.0
    out = attention_fused(q.cuda(), k.cuda(), v.cuda(), scale=1.0).cpu()
    assert torch.equal(out, v[:, 1441:1442].expand(2, sq, 64))
    k[1, 700, 0] = float("nan")
    out = attention_fused(q.cuda(), k.cuda(), v.cuda(), scale=1.0).cpu()
    assert torch.equal(out[0], v[0, 1441:1442].expand(sq, 64)) and out[1].isnan().all()
