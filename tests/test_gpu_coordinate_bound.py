"""The bound on a basin's coordinates, which sets the margin of the FP32 search
that builds the lists: it follows the particles from sort to sort (it does not
add up the path of the fastest), and each basin of a batch has its own.
"""
import ctypes
import subprocess

import numpy as np
import pytest

from simp_b200 import basins, build
from simp_b200.simp import Batch, Simp

pytestmark = pytest.mark.gpu

_SRC = """
#include "ctx.h"
extern "C" double bound(void *ctx, int slot) {
    simp_ctx *c = (simp_ctx *)ctx;
    simp::Inst I{};
    if (cudaStreamSynchronize(c->stream) != cudaSuccess) return -1.0;
    if (cudaMemcpy(&I, c->inst_dev + slot, sizeof(I), cudaMemcpyDeviceToHost) != cudaSuccess) return -2.0;
    double v;
    memcpy(&v, &I.xabs_bits, sizeof(v));
    return v;
}
"""
SPEED = 60.0


@pytest.fixture(scope="module")
def bound(gpu_lib, tmp_path_factory):
    d = tmp_path_factory.mktemp("bound")
    (d / "b.cu").write_text("#include <cstring>\n" + _SRC)
    so = str(d / "b.so")
    subprocess.run([build.nvcc(), "-shared", *build.ARCH, "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-I", build.INCLUDE,
                    "-I", build.CSRC, *build.host_compiler(), "-o", so, str(d / "b.cu")], check=True)
    lib = ctypes.CDLL(so)
    lib.bound.argtypes = [ctypes.c_void_p, ctypes.c_int]
    lib.bound.restype = ctypes.c_double
    return lambda sim, slot=0: lib.bound(sim.h, slot)


def _drifting(nside, seed, far=0.0, speed=SPEED):
    """Towards the origin, so that the largest coordinate falls while the path grows."""
    b = basins.make_basin(nside, 1000.0, seed, walls="", dt=0.5)
    b.x = b.x + far
    b.vx = np.full((b.n, 2), -speed)
    b.params.wind_force = b.params.water_force = 0
    return b


def _check(got, x, speed=SPEED):
    """No less than the truth, and no more than the moves since the last sort (16 steps) above it."""
    top = float(np.abs(x).max())
    since = 17 * 0.5 * speed * np.sqrt(2.0)
    assert top <= got <= top + 2.0 * since, (top, got)


def test_single_basin(bound):
    b = _drifting(60, 3)
    with Simp.from_basin(b) as g:
        assert bound(g) == np.abs(b.x).max()
        for steps in (1, 15, 1, 40, 200):
            g.time_integration(steps)
            _check(bound(g), g.get_state()["x"])


def test_continued_state(bound):
    b = _drifting(60, 3)
    with Simp.from_basin(b) as g:
        for _ in range(40):
            g.time_integration(3)
            s = g.get_state()
            g.set_state(s["x"], s["vx"], s["mass"], s["rho"], s["hsml"], s["A"], s["h"], b.xb, b.massb, 0.5, 0.0)
        _check(bound(g), s["x"])


def test_each_basin_of_a_batch(bound):
    near, far = _drifting(60, 3), _drifting(45, 4, far=3.0e6, speed=2.0 * SPEED)
    with Batch(near.params, near.n + far.n, 0, 2) as g:
        a, z = g.add(near), g.add(far)
        g.step(50)
        _check(bound(g, a), g.get_state(a)["x"])
        _check(bound(g, z), g.get_state(z)["x"], 2.0 * SPEED)
        g.remove(z)
        g.step(20)
        _check(bound(g, a), g.get_state(a)["x"])
