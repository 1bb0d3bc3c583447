"""Builds ``libkcg_b200.so`` in-tree and (optionally) a family of cubins ahead of time.

    python -m codegendemo_b200.build            # library + default cubins
    python -m codegendemo_b200.build --lib-only

The library is built with nvcc for sm_100a: its host code binds the CUDA driver lazily (so it loads without a GPU),
and pieces of device code are linked into it (the allocation-free split-K entry, the row softmax, the fused attention).
Beside it stands ``_pycall``, a small extension module for the building interpreter that launches on behalf of Python
callers, and ``_torchcall``, which makes an operator's warm call in one step (optional: without it the operators go their way
through Python). The GEMM kernels themselves are compiled per config by the library's own compile entry with
``nvcc -cubin -gencode arch=compute_100a,code=sm_100a``.
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_HOME = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def _newer(target: str, sources) -> bool:
    if not os.path.exists(target):
        return False
    t = os.path.getmtime(target)
    return all(os.path.getmtime(s) <= t for s in sources)


def pycall_path() -> str:
    """The extension module of this interpreter: its name carries the ABI tag, so another one's is never loaded."""
    import sysconfig
    return os.path.join(HERE, "_pycall" + sysconfig.get_config_var("EXT_SUFFIX"))


def build_pycall(force: bool = False) -> str:
    """The Python extension module that makes the common launches (csrc/kcg_pycall.c)."""
    import shlex
    import shutil
    import sysconfig
    out = pycall_path()
    untagged = os.path.join(HERE, "_pycall.so")  # an earlier build's, for whichever interpreter
    if os.path.exists(untagged):
        os.remove(untagged)
    src = os.path.join(HERE, "csrc", "kcg_pycall.c")
    if force or not _newer(out, [src, os.path.join(os.path.dirname(HERE), "include", "kcg_b200.h")]):
        compilers = [shlex.split(c) for c in (os.environ.get("CC"), sysconfig.get_config_var("CC"), "cc", "gcc") if c]
        cc = next((c for c in compilers if shutil.which(c[0])), ["cc"])
        subprocess.check_call(cc + ["-O2", "-shared", "-fPIC", "-I" + sysconfig.get_paths()["include"], "-o", out, src])
    return out


def torchcall_path() -> str:
    import sysconfig
    return os.path.join(HERE, "_torchcall" + sysconfig.get_config_var("EXT_SUFFIX"))


def build_torchcall(force: bool = False):
    """The extension module of the warm calls (csrc/kcg_torchcall.cpp), against this interpreter's torch; None where there is
    no torch or no C++ compiler to build it with, or where it does not compile (no Python headers, another torch's internals)."""
    import shlex
    import shutil
    import sysconfig
    cxx = next((c for c in (os.environ.get("CXX"), sysconfig.get_config_var("CXX"), "c++", "g++")
                if c and shutil.which(shlex.split(c)[0])), None)
    try:
        import torch
    except ImportError:
        torch = None
    if cxx is None or torch is None or torch.version.cuda is None:
        return None
    out, src = torchcall_path(), os.path.join(HERE, "csrc", "kcg_torchcall.cpp")
    root = os.path.dirname(torch.__file__)
    deps = [src, os.path.join(os.path.dirname(HERE), "include", "kcg_b200.h"), os.path.join(root, "version.py")]
    if force or not _newer(out, deps):
        includes = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
                    os.path.join(CUDA_HOME, "include")]
        if os.path.exists(out):  # (one of an older source or torch must not be what is imported if this one does not compile)
            os.remove(out)
        try:
            subprocess.check_call(shlex.split(cxx) + ["-O2", "-std=c++17", "-shared", "-fPIC",
                                                      f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                                                      "-I" + sysconfig.get_paths()["include"]]
                                  + [f for i in includes for f in ("-isystem", i)]
                                  + ["-o", out, src, "-L" + os.path.join(root, "lib")]
                                  + ["-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10"])
        except subprocess.CalledProcessError as e:
            print(f"{src} does not compile here (status {e.returncode}): warm calls go through Python", file=sys.stderr)
            return None
    return out


def build_library(force: bool = False) -> str:
    """The C-ABI library. Needs nvcc alone; :func:`build_pycall` makes what Python callers launch through."""
    out = os.path.join(HERE, "libkcg_b200.so")
    srcs = [os.path.join(HERE, "csrc", "kcg_shim.cpp")]
    kdir = os.path.join(HERE, "csrc", "kernels")  # the allocation-free entry instantiates a kernel from these
    deps = srcs + [os.path.join(kdir, f) for f in sorted(os.listdir(kdir))] + [
        os.path.join(os.path.dirname(HERE), "include", "kcg_b200.h")]
    # device code linked into the library itself: the allocation-free split-K entry, the row softmax, the fused attention
    # and the split of fp32 operands
    extra = [os.path.join(HERE, "csrc", f) for f in ("kcg_noalloc.cu", "kcg_softmax.cu", "kcg_attention.cu", "kcg_f32split.cu")]
    deps += extra
    if not force and _newer(out, deps):
        return out
    nvcc = os.path.join(CUDA_HOME, "bin", "nvcc")
    cmd = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-shared",
           "-Xcompiler", "-fPIC", "-cudart", "static", "-I" + os.path.join(HERE, "csrc", "kernels"),
           "-o", out, *srcs, *extra, "-ldl", "-lpthread"]
    subprocess.check_call(cmd)
    return out


def prebuilt_configs():
    """Configs compiled ahead of time, so that a GPU box needs no nvcc for the smoke run and the bench."""
    from codegendemo_b200.kcg.matmul_op import default_config, tuned_config
    from codegendemo_b200.kcg.Utils import EnumKernelDType as E
    simt = dict(KERNEL_VARIANT=1, BLOCK_SIZE_M=128, BLOCK_SIZE_N=128, BLOCK_SIZE_K=16, THREAD_SIZE_M=8,
                THREAD_SIZE_N=8, BLOCK_LAYOUT_M=4, BLOCK_LAYOUT_N=2, WARP_LAYOUT_M=4, WARP_LAYOUT_N=8,
                WARP_SCATTER_WIDTH_A=4, WARP_SCATTER_WIDTH_B=4, THREAD_SCATTER_WIDTH_A=4, THREAD_SCATTER_WIDTH_B=4)
    cfgs = [tuned_config(1024, 1024, 1024, E.float32), tuned_config(4096, 4096, 4096, E.float32),
            default_config(4096, 4096, 4096, E.float32, **simt), tuned_config(8192, 8192, 8192, E.bfloat16)]
    # the rectangular sweep the benchmark line carries
    cfgs += [tuned_config(m, nk, nk, dt) for nk in (4096, 11008) for m in (128, 512, 2048)
             for dt in (E.float32, E.bfloat16)]
    for g in (1, 2, 4, 8):
        cfgs.append(tuned_config(32768 // g, 8192, 8192, E.bfloat16))
        if g > 1:  # tile of the bench's fused GEMM + all-gather leg (two TMEM accumulator buffers)
            cfgs.append(default_config(32768 // g, 8192, 8192, E.bfloat16))
    return cfgs


def prune_stale_cubins() -> None:
    """Cubins are cached under _cache/src-<hash of the kernel sources>; drop the directories of older sources."""
    import shutil
    from codegendemo_b200 import _lib
    cur = _lib.get_lib().kcg_cache_dir().decode()
    base = os.path.dirname(cur)
    if os.path.basename(base) != "_cache":
        return
    for d in os.listdir(base):
        full = os.path.join(base, d)
        if full != cur and (d.startswith("src-") or d.endswith(".cubin")):
            shutil.rmtree(full) if os.path.isdir(full) else os.remove(full)


def compile_many(kpms, workers: int = 0, verbose: bool = False):
    """Compiles a list of configs on a thread pool (the compile entry is reentrant and runs nvcc in a child
    process, so threads suffice); returns [(path, name)] in input order. Cached cubins cost nothing."""
    from concurrent.futures import ThreadPoolExecutor
    from codegendemo_b200.kcg.KCGCompiler import KCGCompiler

    def one(kpm):
        kpm.check()
        path, name = KCGCompiler().compileKernel(kpm)[0][:2]
        if verbose:
            print("cubin:", os.path.basename(path))
        return path, name

    workers = workers or min(16, os.cpu_count() or 1)
    with ThreadPoolExecutor(max_workers=workers) as pool:
        return list(pool.map(one, kpms))


def prebuild_kernels(verbose: bool = True) -> int:
    prune_stale_cubins()
    return len(compile_many(prebuilt_configs(), verbose=verbose))


if __name__ == "__main__":
    sys.path.insert(0, os.path.dirname(HERE))
    print(build_library(force="--force" in sys.argv))
    print(build_pycall(force="--force" in sys.argv))
    print(build_torchcall(force="--force" in sys.argv))
    if "--lib-only" not in sys.argv:
        prebuild_kernels()
