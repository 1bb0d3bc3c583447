"""The warm calls of the operators (csrc/kcg_torchcall.cpp): what they take, and that they do what the operator's own way does."""

import ctypes
import gc
import threading
import weakref

import pytest
import torch

from codegendemo_b200 import _lib
from codegendemo_b200 import build as kbuild
from codegendemo_b200.kcg import matmul_op


@pytest.fixture(scope="module")
def warm():
    if kbuild.build_torchcall() is None or not matmul_op._warm_calls():
        pytest.skip("no module of warm calls for this torch")
    return matmul_op._warm_calls()


class _Sub(torch.Tensor):
    pass


def test_everything_but_plain_cuda_tensors_goes_the_operators_way(warm):
    x = torch.zeros((256, 256), dtype=torch.bfloat16)
    for a in (x, x.as_subclass(_Sub), x.to("meta"), x.t(), x.to_sparse(), x[0], 3, None, "a"):
        for b in (x, a):
            assert warm.matmul(a, b, None, False, False) is None
            assert warm.bmm(a, b, None, False) is None
            assert warm.attention(a, b, b) is None
    assert warm.matmul(x) is None and warm.bmm() is None and warm.attention(x, x, x, x) is None


def test_without_the_module_the_operators_go_their_way(warm, monkeypatch):
    class _Kernel:
        def launchKernel(self, dev, a, b, c, **kw):
            c.fill_(7)
    kern = _Kernel()
    kern.m_launcher = kern
    for value in (None, False, warm):
        monkeypatch.setattr(matmul_op, "_warm", value)
        monkeypatch.setattr(matmul_op, "_KERNELS", {})
        monkeypatch.setattr(matmul_op, "build_kernel", lambda kpm, dev=0: (None, kern))
        x = torch.zeros((256, 256), dtype=torch.bfloat16)
        assert (matmul_op.matmul(x, x) == 7).all() and (matmul_op.bmm(x[None], x[None]) == 7).all()


def _calls():
    gen = torch.Generator(device="cuda").manual_seed(1)
    r = lambda *s, dt=torch.bfloat16: torch.randn(s, generator=gen, device="cuda").to(dt) / 16
    for dt in (torch.bfloat16, torch.float16, torch.float32):
        a, b, bias = r(256, 192, dt=dt), r(192, 384, dt=dt), r(384, dt=dt)
        yield matmul_op.matmul, (a, b), {}
        yield matmul_op.matmul, (torch.nn.Parameter(a), b), dict(bias=bias, relu=True)
        if dt != torch.float32:
            yield matmul_op.matmul, (a, r(384, 192, dt=dt)), dict(b_transposed=True, relu=True)
            yield matmul_op.bmm, (r(3, 128, 64, dt=dt), r(3, 64, 192, dt=dt)), dict(bias=r(192, dt=dt))
            yield matmul_op.attention_fused, (r(2, 70, 64, dt=dt), r(2, 200, 64, dt=dt), r(2, 200, 64, dt=dt)), {}


@pytest.mark.gpu
def test_the_same_results(warm, monkeypatch):
    """Also on another stream, under a mode that watches torch's calls, and for operands the warm call does not take."""
    class Watch(torch.utils._python_dispatch.TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))
    taken = []

    class Spy:
        def __getattr__(self, name):
            def call(*args):
                out = getattr(warm, name)(*args)
                taken.append(out is not None)
                return out
            return call if name in ("matmul", "bmm", "attention") else getattr(warm, name)
    stream = torch.cuda.Stream()
    for op, args, kw in _calls():
        op(*args, **kw)
        monkeypatch.setattr(matmul_op, "_warm", False)
        want = op(*args, **kw)
        monkeypatch.setattr(matmul_op, "_warm", Spy())
        taken.clear()
        first, second = op(*args, **kw), op(*args, **kw)
        assert taken == [True, True], (op.__name__, kw.keys())
        assert first.data_ptr() != second.data_ptr() and first.dtype == want.dtype and not first.requires_grad
        with torch.cuda.stream(stream):
            stream.wait_stream(torch.cuda.default_stream())
            third = op(*args, **kw)
        stream.synchronize()
        seen = []
        taken.clear()
        with Watch():
            fourth = op(*args, **kw)
        assert taken == [False] and seen
        for got in (first, second, third, fourth):
            assert torch.equal(got, want), (op.__name__, kw.keys())
        if op is matmul_op.matmul and not kw:
            a = torch.cat([args[0], args[0]], dim=1)[:, args[0].shape[1]:]  # rows with a pitch
            taken.clear()
            assert torch.equal(op(a, args[1]), want) and taken == [False]


@pytest.mark.gpu
def test_errors_of_a_warm_call(warm):
    """An operand that no kernel can read is refused with the library's error, and the next call is not affected."""
    a, b = torch.ones((256, 192), device="cuda", dtype=torch.bfloat16), torch.ones((192, 256), device="cuda", dtype=torch.bfloat16)
    want = matmul_op.matmul(a, b)
    odd = torch.ones(256 * 192 + 1, device="cuda", dtype=torch.bfloat16)[1:].view(256, 192)  # not on 16 bytes
    for _ in range(2):
        with pytest.raises(_lib.KCGError):
            matmul_op.matmul(odd, b)
    with pytest.raises(_lib.KCGError):
        matmul_op.matmul(a, b, bias=torch.ones(257, device="cuda", dtype=torch.bfloat16)[1:])
    with pytest.raises(AssertionError):
        matmul_op.matmul(a, b[:128])
    assert torch.equal(matmul_op.matmul(a, b), want)


def test_a_module_that_does_not_compile(tmp_path, monkeypatch):
    """The build goes on without the warm calls, and leaves no module of an older source to be imported in their place."""
    from codegendemo_b200 import build
    stale = tmp_path / "_torchcall.so"
    stale.write_bytes(b"")
    monkeypatch.setattr(build, "torchcall_path", lambda: str(stale))
    monkeypatch.setenv("CXX", "false")
    assert build.build_torchcall(force=True) is None
    assert not stale.exists()


class _Owner:
    pass


@pytest.mark.gpu
def test_a_launch_holds_what_owns_its_kernel(warm):
    """While a warm call is inside the launch (a stand-in that waits), another thread puts another kernel in its place."""
    gemm_t = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_uint64, ctypes.c_void_p, ctypes.c_int, *[ctypes.c_uint64] * 4,
                              *[ctypes.c_int64] * 3, ctypes.c_int, ctypes.c_void_p)
    inside, go_on, functions = threading.Event(), threading.Event(), []

    def gemm(function, *rest):
        functions.append(function)
        inside.set()
        go_on.wait(20.0)
        return 0
    gemm_c, lib = gemm_t(gemm), _lib.get_lib()
    address = lambda f: ctypes.cast(f, ctypes.c_void_p).value
    a, b = torch.zeros((8, 24), device="cuda"), torch.zeros((24, 40), device="cuda")
    key = (8, 40, 24, 0, 4, a.device.index, 0)
    first, second = _Owner(), _Owner()
    alive = weakref.ref(first)
    warm.remember(*key, 111, 0, first)
    warm.bind(address(gemm_c), address(lib.kcg_attention_fwd), _lib.check)
    try:
        got = []
        caller = threading.Thread(target=lambda: got.append(warm.matmul(a, b, None, False, False)))
        caller.start()
        assert inside.wait(20.0)
        del first
        warm.remember(*key, 222, 0, second)
        gc.collect()
        held = alive() is not None
        go_on.set()
        caller.join(20.0)
        assert held and not caller.is_alive() and got[0].shape == (8, 40)
        gc.collect()
        assert alive() is None
        warm.matmul(a, b, None, False, False)
        assert functions == [111, 222]
    finally:
        go_on.set()
        warm.bind(address(lib.kcg_launch_gemm_strided), address(lib.kcg_attention_fwd), _lib.check)


@pytest.mark.gpu
def test_the_allocator_asks_before_it_takes_memory(warm):
    """What would give the library's workspaces back (a stand-in) is called when torch goes to the device for memory."""
    asked = []
    trim = ctypes.CFUNCTYPE(ctypes.c_bool, ctypes.c_int)(lambda device: bool(asked.append(device)))
    own = ctypes.cast(_lib.get_lib().kcg_internal_trim_if_low, ctypes.c_void_p).value
    torch.cuda.empty_cache()
    warm.bind_trim(ctypes.cast(trim, ctypes.c_void_p).value)
    try:
        t = torch.empty(64 << 20, dtype=torch.uint8, device="cuda")
    finally:
        warm.bind_trim(own)
    assert asked == [t.device.index]


@pytest.mark.gpu
def test_a_product_after_its_workspace_is_gone():
    """Parts, partials and captured graphs after kcg_trim: the same bits."""
    gen = torch.Generator(device="cuda").manual_seed(4)
    a, b = [torch.rand(s, generator=gen, device="cuda") * 2 - 1 for s in ((2048, 2048), (2048, 4096))]
    want = matmul_op.matmul(a, b)
    c = torch.empty_like(want)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        matmul_op.matmul(a, b, c)
    assert _lib.get_lib().kcg_trim(0) == 0
    junk = [torch.full((1 << 22,), 7.0, device="cuda") for _ in range(16)]  # what is free now belongs to others
    graph.replay()
    assert torch.equal(c, want) and torch.equal(matmul_op.matmul(a, b), want)
    assert all(bool((j == 7.0).all()) for j in junk)
