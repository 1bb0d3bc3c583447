"""The launcher where several threads meet: a kernel's first launch, without a GPU (the loader and the launch are stand-ins)."""
import ctypes
import threading
import types

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
