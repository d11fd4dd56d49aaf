"""Pages of the arrays a read-back fills: asking for them changes no content,
inside or beside the ranges, whatever the alignment and the mapping."""
import ctypes
import mmap
import subprocess

import numpy as np
import pytest

from simp_b200 import build

_WRAP = """
#include "host_pages.h"
extern "C" void pages(const void *a, size_t na, const void *b, size_t nb) {
    const simp::HostRange r[] = {{a, na}, {nullptr, na}, {b, nb}};
    simp::make_resident(r, 3);
}
"""


@pytest.fixture(scope="module")
def pages(tmp_path_factory):
    d = tmp_path_factory.mktemp("pages")
    (d / "wrap.cpp").write_text(_WRAP)
    so = str(d / "pages.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-pthread", "-I", build.CSRC, "-o", so,
                    str(d / "wrap.cpp"), build.CSRC + "/host_pages.cpp"], check=True)
    lib = ctypes.CDLL(so)
    lib.pages.argtypes = [ctypes.c_void_p, ctypes.c_size_t] * 2
    return lib.pages


@pytest.mark.parametrize("nbytes", [0, 1, 262143, 262144, 1 << 20, (1 << 20) + 8, 9 << 20])
@pytest.mark.parametrize("offset", [0, 8, 4095, 4096])
@pytest.mark.parametrize("prot", ["fresh", "written", "read only"])
def test_contents_stay(pages, nbytes, offset, prot):
    m = mmap.mmap(-1, offset + nbytes + 8192, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS)
    a = np.frombuffer(m, dtype=np.uint8)
    want = np.zeros(a.size, np.uint8)
    if prot != "fresh":
        want = np.random.default_rng(nbytes).integers(0, 256, a.size, dtype=np.uint8)
        a[:] = want
    if prot == "read only":
        assert ctypes.CDLL(None).mprotect(ctypes.c_void_p(a.ctypes.data), ctypes.c_size_t(a.size), 1) == 0
    b = np.arange(nbytes // 8 + 1, dtype=np.float64)
    pages(a.ctypes.data + offset, nbytes, b.ctypes.data, b.nbytes)
    assert np.array_equal(a, want)
    assert np.array_equal(b, np.arange(nbytes // 8 + 1, dtype=np.float64))
