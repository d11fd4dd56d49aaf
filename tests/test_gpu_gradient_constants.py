"""The constants of the pair gradients where hsml is one value: (qscale / hsml)^2
and factor / hsml^4, each within one rounding (2^-53, and 2^-64 of the extended
arithmetic they are worked out in) of the exact rationals.  What they are off by
is the same for every pair, so that no sum averages it away."""
import ctypes
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from simp_b200 import basins, build
from simp_b200.params import SKF_CUBIC, SKF_WENDLAND_C6
from simp_b200.simp import Simp

pytestmark = pytest.mark.gpu

_SRC = """
#include "ctx.h"
extern "C" int constants(void *ctx, double *k, double *c) {
    simp_ctx *x = (simp_ctx *)ctx;
    simp::Inst I{};
    if (cudaStreamSynchronize(x->stream) != cudaSuccess) return 1;
    if (cudaMemcpy(&I, x->inst_dev, sizeof(I), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    *k = I.grad_k;
    *c = I.grad_c;
    return 0;
}
"""
PI = Fraction(3.1415926535897932)


@pytest.fixture(scope="module")
def constants(gpu_lib, tmp_path_factory):
    d = tmp_path_factory.mktemp("constants")
    (d / "c.cu").write_text(_SRC)
    so = str(d / "c.so")
    subprocess.run([build.nvcc(), "-shared", *build.ARCH, "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-I", build.INCLUDE,
                    "-I", build.CSRC, *build.host_compiler(), "-o", so, str(d / "c.cu")], check=True)
    lib = ctypes.CDLL(so)
    lib.constants.argtypes = [ctypes.c_void_p] * 3

    def look(sim):
        k, c = ctypes.c_double(), ctypes.c_double()
        assert lib.constants(sim.h, ctypes.byref(k), ctypes.byref(c)) == 0
        return k.value, c.value
    return look


@pytest.mark.parametrize("hsml", [600.0, 2400.0, 3000.0, 7.3, 1234.5, 5 ** 0.5 * 1e5])
@pytest.mark.parametrize("skf, qscale, factor", [(SKF_CUBIC, 2, Fraction(15) / (7 * PI) * 16),
                                                 (SKF_WENDLAND_C6, 1, Fraction(78) / (7 * PI))])
def test_rounded_once(constants, skf, qscale, factor, hsml):
    b = basins.make_basin(8, hsml / 2.4, 1, skf=skf)
    b.hsml = np.full(b.n, hsml)
    with Simp.from_basin(b) as g:
        k, c = constants(g)
    h = Fraction(hsml)
    for got, want in ((k, (Fraction(qscale) / h) ** 2), (c, factor / h ** 4)):
        assert abs(Fraction(got) / want - 1) < Fraction(2) ** -53 + Fraction(2) ** -61
