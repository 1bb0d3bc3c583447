"""Launch boundary: ``launchKernel(device, a, b, c)`` on torch's current stream.

Mirror of ``HIPLauncher`` (Runtime/python/kcg/HIPLauncher.py:264-314). The reference generates,
compiles (gcc) and imports one C launcher per kernel signature; here every kernel takes the same
parameter block, so one C entry (``kcg_launch_gemm``) serves all of them and builds the TMA tensor
maps itself. Pointer arguments may be ints or anything with ``data_ptr()`` (HIPLauncher.py:148-187).
"""
import ctypes
import threading

from codegendemo_b200 import _lib
from codegendemo_b200.kcg.Loader import CudaLoaderST, KernelLibFile
from codegendemo_b200.kcg.Utils import DeviceInfo


_LOADING = threading.Lock()


def _pointer_of(obj) -> int:
    if obj is None:
        raise TypeError("KCG launcher: pointer argument is None")
    if isinstance(obj, int):
        return obj
    ptr = getattr(obj, "data_ptr", None)
    if ptr is None:
        raise TypeError("Pointer argument must be either uint64 or have data_ptr method")
    return int(ptr())


class CudaLauncher:
    def __init__(self, kernelBinaryPath, kernelFuncName, shmSize, signature: dict, gridDims: list,
                 blockDims: list, device=0, kernelInfo: dict = None):
        self.m_libFile = KernelLibFile(kernelBinaryPath, kernelFuncName, shmSize, device)
        self.m_signature = signature
        self.m_gridDims = list(gridDims)
        self.m_blockDims = list(blockDims)
        self.m_shmSize = shmSize
        self.m_device = device
        self.m_kernelInfoDict = kernelInfo
        # loaded lazily in the process that owns the GPU (launchers are pickled across processes)
        self.m_runtime = None
        self.m_cInfo = None
        self.m_infoAddr = 0

    def __getstate__(self):
        st = dict(self.__dict__)
        st["m_runtime"] = None
        st["m_cInfo"] = None
        st["m_infoAddr"] = 0
        return st

    def _getWrapper(self):
        if self.m_runtime is None:
            # One thread loads. A launch reads m_cInfo by its address, with the GIL released and no reference of its own,
            # so the structure is never replaced, and m_runtime, which says that it is there, is set last.
            with _LOADING:
                if self.m_runtime is None:
                    if self.m_kernelInfoDict is None:
                        raise RuntimeError("KCG launcher: kernelInfo missing (compile with KCGCompiler first)")
                    info = dict(self.m_kernelInfoDict)
                    info["grid"], info["block"], info["smem_bytes"] = self.m_gridDims, self.m_blockDims, self.m_shmSize
                    cInfo = _lib.KernelInfo.from_dict(info)
                    runtime = CudaLoaderST().loadBinary(self.m_libFile)
                    self.m_cInfo, self.m_infoAddr = cInfo, ctypes.addressof(cInfo)
                    self.m_runtime = runtime
        return self.m_runtime

    def launchKernel(self, device, *args, stream=None, alpha=1.0, beta=0.0, bias=None, relu=False, peers=None,
                     batch=1, lda=0, ldb=0, ldc=0):
        """(a, b, c) -> c = a.b on `stream` (torch's current stream by default). The keyword
        arguments fuse c = act(alpha * a.b + beta * c + bias) into the kernel's store; `peers` (up to 7
        device addresses or tensors shaped like c) also receive every finished tile: the fused
        all-gather of an M-sharded product. The reference's launcher has no such arguments and the plain
        call behaves as the reference's."""
        rt = self.m_runtime
        if rt is None:
            rt = self._getWrapper()
        if len(args) != 3:
            raise TypeError("matmul kernel takes (a, b, c)")
        if stream is None:
            stream = DeviceInfo.get_cuda_stream(device)
        a, b, c = args
        if not peers:
            # lda, ldb, ldc: elements between rows of operands that are sub-matrices of wider row-major arrays, 0 =
            # contiguous; with batch > 1, (a, b, c) hold `batch` problems of the kernel's M, N, K (torch.bmm layout)
            status = _lib.pycall.gemm(rt.m_function, self.m_infoAddr, device, stream, a, b, c, lda, ldb, ldc, batch, alpha,
                                      beta, bias, relu)
        else:
            epi = None
            if alpha != 1.0 or beta != 0.0 or bias is not None or relu:
                epi = ctypes.byref(_lib.Epilogue(float(alpha), float(beta), _pointer_of(bias) if bias is not None else 0,
                                                 int(bool(relu))))
            if lda or ldb or ldc:
                raise ValueError("a strided launch has no fused all-gather")
            if batch != 1:
                raise ValueError("a batched launch has no fused all-gather")
            if epi is None:
                epi = ctypes.byref(_lib.Epilogue(1.0, 0.0, 0, 0))
            arr = (ctypes.c_uint64 * len(peers))(*[_pointer_of(x) for x in peers])
            status = _lib.get_lib().kcg_launch_gemm_allgather(
                rt.m_function, ctypes.byref(self.m_cInfo), int(device), int(stream), _pointer_of(a), _pointer_of(b),
                _pointer_of(c), epi, arr, len(peers))
        if status:
            _lib.check(status)

    def runHost(self, device, hostA, hostB, hostC, stream=None):
        """Whole operator on host buffers (H2D, kernel, D2H, synchronise)."""
        rt = self._getWrapper()
        if stream is None:
            stream = DeviceInfo.get_cuda_stream(device)
        _lib.check(_lib.get_lib().kcg_matmul_host(ctypes.c_uint64(rt.m_function), ctypes.byref(self.m_cInfo),
                                                  int(device), ctypes.c_uint64(int(stream)),
                                                  ctypes.c_void_p(_pointer_of(hostA)),
                                                  ctypes.c_void_p(_pointer_of(hostB)),
                                                  ctypes.c_void_p(_pointer_of(hostC))))

    def checkStatus(self, device, stream=None):
        if stream is None:
            stream = DeviceInfo.get_cuda_stream(device)
        _lib.check(_lib.get_lib().kcg_check_status(int(device), ctypes.c_uint64(int(stream))))
