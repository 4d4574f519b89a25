"""What fn_download does to a large pageable destination before its copy, on the
CPU: missing pages are faulted in and bytes kept; a buffer whose pages are
there and an address that is not mapped are left alone (each in a process of
its own, since writing to either would end it)."""
import os
import subprocess
import sys

import pytest

HERE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "host_upload")

CHILD = r"""
import ctypes as C, mmap, sys
what, lib = sys.argv[1], C.CDLL(sys.argv[2])
lib.hp_touch.argtypes = [C.c_void_p, C.c_size_t]
libc = C.CDLL(None, use_errno=True)
libc.mmap.restype = C.c_void_p
libc.mmap.argtypes = [C.c_void_p, C.c_size_t, C.c_int, C.c_int, C.c_int, C.c_long]
for f in ("munmap", "mprotect", "mincore"):
    getattr(libc, f).argtypes = [C.c_void_p, C.c_size_t] + ([] if f == "munmap" else [C.c_void_p if f == "mincore" else C.c_int])
page, pages = mmap.PAGESIZE, 6000
size = page * pages
at = libc.mmap(None, size, mmap.PROT_READ | mmap.PROT_WRITE, mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS, -1, 0)
assert at not in (None, C.c_void_p(-1).value)

def missing():
    there = (C.c_ubyte * pages)()
    assert libc.mincore(at, size, there) == 0
    return sum(1 for v in there if not v & 1)

if what == "fresh":
    assert missing() > pages // 2
    lib.hp_touch(at + 24, size - 48)
    assert missing() == 0 and C.string_at(at, size) == bytes(size)
elif what == "half":
    C.memset(at, 7, size // 2)
    lib.hp_touch(at, size)
    assert missing() == 0 and C.string_at(at, size) == bytes([7]) * (size // 2) + bytes(size // 2)
elif what == "present":
    C.memset(at, 7, size)
    assert libc.mprotect(at, size, mmap.PROT_READ) == 0
    lib.hp_touch(at + 24, size - 48)
    assert C.string_at(at, size) == bytes([7]) * size
elif what == "unmapped":
    assert libc.munmap(at, size) == 0
    lib.hp_touch(at + 24, size - 48)
print("done")
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from fibrenet_b200 import build
    so = str(tmp_path_factory.mktemp("pages") / "libpages.so")
    out = subprocess.run([build.nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "-Xcompiler",
                          "-fPIC", "-include", os.path.join(HERE, "fake_cuda.h"), "-shared", "-o", so,
                          os.path.join(HERE, "pages_harness.cu")], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr[-3000:]
    return so


@pytest.mark.parametrize("what", ["fresh", "half", "present", "unmapped"])
def test_pages(lib, what):
    out = subprocess.run([sys.executable, "-c", CHILD, what, lib], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "done", (out.returncode, out.stderr[-2000:])
