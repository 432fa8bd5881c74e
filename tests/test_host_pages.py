"""Pages made before a download (ps3d_gb300/csrc/host_pages.h): all of a fresh
array's, contents kept, threads within the process's processors, and none where
the memory refuses the advice."""
import ctypes
import mmap
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "ps3d_gb300", "csrc")
SIZE = (20 << 20) + 4096 * 3
LIBC = ctypes.CDLL(None, use_errno=True)
PROT_READ, POPULATE_WRITE = 1, 23

CODE = """
import ctypes, mmap, os, sys
cpus = sorted(os.sched_getaffinity(0))[:int(sys.argv[2])]
os.sched_setaffinity(0, cpus)
L = ctypes.CDLL(sys.argv[1])
L.host_populate.argtypes = [ctypes.c_void_p, ctypes.c_ulonglong]
size = int(sys.argv[3])
m = mmap.mmap(-1, size, mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS, mmap.PROT_READ | mmap.PROT_WRITE)
m[size // 2] = 7
a = ctypes.addressof(ctypes.c_char.from_buffer(m))
n = L.host_populate(a + 8, size - 8)
vec = (ctypes.c_ubyte * (size // mmap.PAGESIZE))()
libc = ctypes.CDLL(None)
assert libc.mincore(ctypes.c_void_p(a), ctypes.c_size_t(size), vec) == 0
print(len(cpus), n, sum(v & 1 for v in vec), len(vec), m[size // 2], L.host_populate(a + 8, size - 8))
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("pages") / "libpages.so")
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-std=c++17", "-pthread", "-I", CSRC, "-o", so,
                    os.path.join(HERE, "host_pages.cpp")], check=True)
    return so


def advice_taken():
    m = mmap.mmap(-1, mmap.PAGESIZE)
    a = ctypes.addressof(ctypes.c_char.from_buffer(m))
    return LIBC.madvise(ctypes.c_void_p(a), ctypes.c_size_t(mmap.PAGESIZE), POPULATE_WRITE) == 0


@pytest.mark.parametrize("cpus", [1, 2, 4])
def test_fresh_array(lib, cpus):
    if not advice_taken():
        pytest.skip("this kernel does not make pages on advice")
    out = subprocess.run([sys.executable, "-c", CODE, lib, str(cpus), str(SIZE)], check=True, capture_output=True,
                         text=True).stdout
    allowed, started, made, pages, kept, again = map(int, out.split())
    assert started == min(allowed - 1, 7, 4)  # 20 MB are six parts of 4 MB, the caller's first among them
    assert made >= pages - 1 and kept == 7  # the first page is not whole
    assert again == 0  # the pages are there


def test_memory_that_refuses(lib):
    """a mapping without write permission: no thread, no fault"""
    m = mmap.mmap(-1, SIZE)
    a = ctypes.addressof(ctypes.c_char.from_buffer(m))
    assert LIBC.mprotect(ctypes.c_void_p(a), ctypes.c_size_t(SIZE), PROT_READ) == 0
    L = ctypes.CDLL(lib)
    L.host_populate.argtypes = [ctypes.c_void_p, ctypes.c_ulonglong]
    assert L.host_populate(a, SIZE) == 0


def test_small_arrays_are_left_alone(lib):
    L = ctypes.CDLL(lib)
    L.host_populate.argtypes = [ctypes.c_void_p, ctypes.c_ulonglong]
    assert L.host_populate(None, 4096) == 0
