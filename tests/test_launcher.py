"""The launcher without a GPU (the loader and the library's entries are stand-ins): a kernel's first launch from several
threads, and the arguments that a launch takes."""
import ctypes
import os
import subprocess
import sys
import threading
import types

import numpy as np
import pytest
import torch

from codegendemo_b200 import _lib
from codegendemo_b200.kcg import CudaLauncher as cl
from codegendemo_b200.kcg.KCGCompiler import KCGCompiler
from codegendemo_b200.kcg.matmul_op import default_config
from codegendemo_b200.kcg.Utils import EnumKernelDType as E


def _launcher():
    compiler = KCGCompiler()
    path, name, gx, gy, gz, bx, by, bz = compiler.compileKernel(default_config(256, 256, 256, E.bfloat16))[0]
    return cl.CudaLauncher(path, name, compiler.lastInfo["smem_bytes"], {}, [gx, gy, gz], [bx, by, bz], 0, compiler.lastInfo)


def test_first_launches_of_two_threads_share_one_kernel_info(monkeypatch):
    """A second thread stands inside the loading while the first one launches: the structure whose address the first launch
    was given has to stay the launcher's own, or it is freed under that launch."""
    launcher = _launcher()
    late_inside, launching, late_done = threading.Event(), threading.Event(), threading.Event()
    loads, seen = [], []
    from_dict = _lib.KernelInfo.from_dict

    def slow_from_dict(info):
        if threading.current_thread().name == "late":
            late_inside.set()
            launching.wait(1.0)  # (never set where loading is one thread's at a time)
        return from_dict(info)

    def load(self, libFile):
        loads.append(libFile)
        return types.SimpleNamespace(m_function=1)

    def gemm(function, infoAddr, *rest):
        if threading.current_thread().name == "late":
            return 0
        launching.set()
        late_done.wait(5.0)
        seen.append(infoAddr == ctypes.addressof(launcher.m_cInfo) == launcher.m_infoAddr)
        return 0

    monkeypatch.setattr(_lib.KernelInfo, "from_dict", slow_from_dict)
    monkeypatch.setattr(cl.CudaLoaderST, "loadBinary", load)
    monkeypatch.setattr(_lib, "pycall", types.SimpleNamespace(gemm=gemm))

    def late():
        launcher.launchKernel(0, 16, 16, 16, stream=0)
        late_done.set()

    threads = [threading.Thread(target=late, name="late")]
    threads[0].start()
    assert late_inside.wait(5.0)
    threads.append(threading.Thread(target=lambda: launcher.launchKernel(0, 16, 16, 16, stream=0), name="first"))
    threads[1].start()
    for t in threads:
        t.join(20.0)
        assert not t.is_alive()
    assert seen == [True] and len(loads) == 1


class _At:
    """A pointer argument whose data_ptr() returns `value` (or raises it)."""

    def __init__(self, value):
        self.value = value

    def data_ptr(self):
        if isinstance(self.value, Exception):
            raise self.value
        return self.value


def test_launch_takes_what_int_and_float_take(monkeypatch):
    """Stream, sizes and addresses may be anything int() takes (numpy integers among it), the factors anything float() takes;
    an error inside data_ptr() is the caller's own. The entry that is called is a stand-in that records its arguments."""
    lib = _lib.get_lib()
    got = []
    gemm_t = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_uint64, ctypes.c_void_p, ctypes.c_int, *[ctypes.c_uint64] * 4,
                              *[ctypes.c_int64] * 3, ctypes.c_int, ctypes.POINTER(_lib.Epilogue))
    attn_t = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_int, *[ctypes.c_uint64] * 5, *[ctypes.c_int] * 5, ctypes.c_float)

    def gemm(function, info, device, stream, a, b, c, lda, ldb, ldc, batch, epi):
        e = epi.contents if epi else None
        got.append((function, device, stream, a, b, c, lda, ldb, ldc, batch) + ((e.alpha, e.beta, e.bias, e.relu) if e else ()))
        return 0

    def attention(*args):
        got.append(args)
        return 0

    gemm_c, attention_c = gemm_t(gemm), attn_t(attention)
    real = [ctypes.cast(f, ctypes.c_void_p).value for f in (lib.kcg_launch_gemm_strided, lib.kcg_attention_fwd)]
    call = _lib.pycall
    call.bind(*[ctypes.cast(f, ctypes.c_void_p).value for f in (gemm_c, attention_c)])
    try:
        i = np.int64
        assert call.gemm(np.uint64(3), 4, i(0), np.uint64(7), _At(np.uint64(2 ** 63 + 16)), 32, _At(48), i(8), i(0), "16",
                         np.int32(2), np.float32(0.5), np.float64(2.0), _At(i(64)), np.bool_(True)) == 0
        assert got.pop() == (3, 0, 7, 2 ** 63 + 16, 32, 48, 8, 0, 16, 2, 0.5, 2.0, 64, 1)
        assert call.gemm(3, 4, 0.0, 7.0, 16, 32, 48, 0, 0, 0, 1, torch.tensor(1.0), "0", None, None) == 0
        assert got.pop()[:10] == (3, 0, 7, 16, 32, 48, 0, 0, 0, 1)
        assert call.attention(i(0), np.uint64(7), _At(np.uint64(16)), 32, 48, _At(64), E.float16, i(8), 1, i(256), 64,
                              torch.tensor(0.5)) == 0
        assert got.pop() == (0, 7, 16, 32, 48, 64, 2, 8, 1, 256, 64, 0.5)
        for bad, error in ((_At(AttributeError("mine")), AttributeError), (_At(None), TypeError), (object(), TypeError),
                           (None, TypeError), (_At(ValueError()), ValueError)):
            with pytest.raises(error):
                call.gemm(3, 4, 0, 0, bad, 32, 48, 0, 0, 0, 1, 1.0, 0.0, None, False)
        assert not got
    finally:
        call.bind(*real)


def test_library_loads_without_the_launch_module():
    """Compiling and the host-side entries need the C library alone; a launch without the module says how to build it. The
    module is this interpreter's own."""
    code = """
import sys
sys.modules["codegendemo_b200._pycall"] = None  # importing it fails
from codegendemo_b200 import _lib, build
from codegendemo_b200.kcg.KCGCompiler import compile_info
from codegendemo_b200.kcg.matmul_op import default_config
from codegendemo_b200.kcg.Utils import EnumKernelDType as E
assert _lib.get_lib().kcg_version()
assert compile_info(default_config(256, 256, 256, E.bfloat16).compileArgs()).grid[0] == 2
try:
    _lib.pycall.gemm
except RuntimeError as e:
    assert "codegendemo_b200.build" in str(e)
else:
    raise AssertionError("no error")
import importlib.machinery, os
assert build.pycall_path().endswith(importlib.machinery.EXTENSION_SUFFIXES[0]) and os.path.exists(build.pycall_path())
assert not os.path.exists(os.path.join(os.path.dirname(build.pycall_path()), "_pycall.so"))
"""
    subprocess.run([sys.executable, "-c", code], check=True, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
