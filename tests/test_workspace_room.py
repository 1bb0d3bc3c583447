"""Who gets and who gives back the memory that the library takes for itself: the streams' workspaces, with the parts of large
fp32 products in them. On the CPU, against a stand-in for the driver's library that counts memory."""
import os
import re
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#include <map>
typedef unsigned long long u64;
static std::map<u64, u64> held;
static u64 next_address = 4096, in_use = 0, budget = ~0ull, calls = 0;
extern "C" {
void fake_budget(u64 bytes) { budget = bytes; }
u64 fake_in_use() { return in_use; }
u64 fake_calls() { return calls; }   // allocations asked for and memory freed
int NAME_cuMemAlloc(u64* p, u64 n) {
  ++calls;
  if (in_use + n > budget) return 2;
  *p = next_address;
  next_address += n + 4096;
  held[*p] = n;
  in_use += n;
  return 0;
}
int NAME_cuMemFree(u64 p) {
  ++calls;
  if (!held.count(p)) return 1;
  in_use -= held[p];
  held.erase(p);
  return 0;
}
int NAME_cuMemGetInfo(u64* free_bytes, u64* total) {
  *total = 64ull << 30;
  *free_bytes = (budget < *total ? budget : *total) - in_use;
  return 0;
}
int NAME_cuCtxGetCurrent(void** c) { *c = (void*)64; return 0; }
int NAME_cuDevicePrimaryCtxRetain(void** c, int) { *c = (void*)64; return 0; }
OTHERS
}
"""

PRELUDE = """
import ctypes, sys
fake = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)
fake.fake_in_use.restype = fake.fake_calls.restype = ctypes.c_uint64
fake.fake_budget.argtypes = [ctypes.c_uint64]
sys.path.insert(0, sys.argv[2])
from codegendemo_b200 import _lib
lib = _lib.get_lib()
lib.kcg_internal_reserve.argtypes = [ctypes.c_int] + [ctypes.c_uint64] * 3 + [ctypes.POINTER(ctypes.c_uint64)]
MB, GB = 1 << 20, 1 << 30
def reserve(stream, partials, need):
    out = (ctypes.c_uint64 * 2)()
    assert lib.kcg_internal_reserve(0, stream, partials, need, out) == 0, lib.kcg_last_error()
    return bool(out[0]), out[1]
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    """A libcuda.so.1 with every function that the library binds."""
    where = tmp_path_factory.mktemp("fake")
    source = open(os.path.join(ROOT, "codegendemo_b200", "csrc", "kcg_shim.cpp")).read()
    names = re.findall(r"X\((cu[A-Z]\w+)\)", source)
    (where / "names.c").write_text("#include <cuda.h>\n" + "".join(f"@@{n}={n}\n" for n in names).replace("=", " @ "))
    text = subprocess.run(["g++", "-E", "-P", "-x", "c", "-I/usr/local/cuda/include", str(where / "names.c")], capture_output=True,
                          text=True, check=True).stdout
    symbols = dict(zip(names, re.findall(r"@@\s*\w+\s*@\s*(\w+)", text)))
    assert len(symbols) == len(set(names)) and symbols["cuMemAlloc"] == "cuMemAlloc_v2"
    body = re.sub(r"NAME_(\w+)", lambda m: symbols[m.group(1)], FAKE)
    body = body.replace("OTHERS", "".join(f"int {s}() {{ return 0; }}\n" for n, s in symbols.items() if "NAME_" + n + "(" not in FAKE))
    (where / "fake.cpp").write_text(body)
    out = where / "libcuda.so.1"
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-Wl,-soname,libcuda.so.1", "-o", str(out), str(where / "fake.cpp")], check=True)
    return str(out)


def _run(fake, code):
    r = subprocess.run([sys.executable, "-c", PRELUDE + code, fake, ROOT], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def test_streams_that_alternate_keep_what_they_have(fake):
    """Three streams with 2 GiB of parts each: two have them, the third multiplies without until one has been idle."""
    _run(fake, """
assert reserve(1, MB, 2 * GB)[0] and reserve(2, MB, 2 * GB)[0]
assert reserve(3, MB, 2 * GB) == (False, MB)
calls = fake.fake_calls()
for _ in range(50):
    assert [reserve(s, MB, 2 * GB)[0] for s in (1, 2, 3)] == [True, True, False]
assert fake.fake_calls() == calls      # nobody took anybody's
for _ in range(300):
    reserve(1, MB, 2 * GB)
assert reserve(3, MB, 2 * GB) == (True, 2 * GB)
assert fake.fake_in_use() < 4 * GB + 16 * MB
assert reserve(2, MB, 2 * GB) == (False, MB)
""")


def test_no_memory_for_the_parts(fake):
    """The workspace that is there stays where it does not fit beside the parts, and the device is not asked on every call."""
    _run(fake, """
fake.fake_budget(GB + 100 * MB)
assert reserve(1, 64 * MB, 0)[1] == 64 * MB
assert reserve(1, MB, 2 * GB) == (False, MB)      # (asked again without the old one, which was in the way)
calls = fake.fake_calls()
for _ in range(100):
    assert reserve(1, MB, 2 * GB) == (False, MB)
    assert reserve(1, MB, 3 * GB) == (False, MB)
assert fake.fake_calls() == calls
assert reserve(1, MB, GB // 2) == (True, GB // 2)  # a smaller one may fit
fake.fake_budget(8 * GB)
for _ in range(1100):
    reserve(1, MB, MB)
assert reserve(1, MB, 2 * GB) == (True, 2 * GB)    # asked again in the end
""")


def test_partials_that_a_launch_cannot_do_without(fake):
    """They are had from other streams' parts, however lately used."""
    _run(fake, """
fake.fake_budget(3 * GB)
assert reserve(1, MB, 2 * GB)[0]
assert reserve(2, 2 * GB, 0) == (False, 2 * GB)
assert reserve(1, MB, 2 * GB) == (False, MB)
""")


def test_memory_given_back(fake):
    _run(fake, """
trim = lib.kcg_internal_trim_if_low
trim.restype = ctypes.c_bool
assert not trim(0) and not trim(99)                # no launch yet
reserve(1, MB, 2 * GB), reserve(2, MB, GB)
assert not trim(0) and fake.fake_in_use() > 3 * GB # most of the device is free
fake.fake_budget(12 * GB)
assert trim(0) and fake.fake_in_use() < MB
assert not trim(0)
assert reserve(1, MB, 2 * GB) == (True, 2 * GB)
assert lib.kcg_trim(0) == 0 and fake.fake_in_use() < MB
assert lib.kcg_trim(1) == 0 and lib.kcg_trim(-1) != 0
""")
