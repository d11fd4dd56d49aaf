"""The pair passes' tiles where they can go wrong: tiles of a few particles and
around a full one, tiles that span several cell rows, sparse cell rows whose
halo has to be cut, more neighbours than a list holds, varying hsml with and
without the reference's bucket rule, and lists that motion outdates (built
again between sorts, over a wider stencil, and beyond the widest one).

One right-hand side at the state reached, against the oracle at that state.
The bars are those of the other right-hand-side tests: 1e-11 relative L2 in
FP64, where only the order of the sums differs, 2e-6 in mixed precision.
"""
import ctypes
import subprocess

import numpy as np
import pytest

from helpers import assert_same_pairs, rel_l2, smooth_velocity
from simp_b200 import basins, build
from simp_b200.params import PREC_FP64, PREC_MIXED
from simp_b200.simp import Batch, Simp

pytestmark = pytest.mark.gpu

TOL = {PREC_FP64: 1e-11, PREC_MIXED: 2e-6}


def _keep(b, mask):
    for k in ("x", "vx", "mass", "rho", "hsml", "A", "h"):
        setattr(b, k, np.ascontiguousarray(getattr(b, k)[mask]))
    return b


def _basin(name):
    b = basins.make_basin({"narrow": 120, "sparse": 150}.get(name, 40), 2000.0, 5, walls="+x-y", dt=1.0)
    rng = np.random.default_rng(3)
    b.vx = smooth_velocity(b.x, b.L, amp=0.3, seed=4)
    b.h = 1.0 + 0.5 * np.sin(b.x[:, 0] / 9000.0)
    b.A = 0.9 + 0.1 * np.cos(b.x[:, 1] / 7000.0)
    b.rho = 900.0 * b.h
    b.mass = b.rho * 4.0e6
    if name.startswith("n="):
        _keep(b, slice(0, int(name[2:])))
    elif name == "narrow":       # a tile holds several cell rows, whose ranges meet
        _keep(b, b.x[:, 0] < 5 * b.dx)
    elif name == "sparse":       # full rows under one of every seventh particle
        row = np.floor(b.x[:, 1] / b.dx)
        col = np.floor(b.x[:, 0] / b.dx)
        _keep(b, (row < 20) | ((row == 22) & (col % 7 == 0)))
    elif name == "dense":        # about 66 neighbours
        b.hsml = b.hsml * (4.6 / 2.4)
    elif name == "varied":
        b.hsml = b.hsml * rng.uniform(1.0, 1.3, size=b.n)
    elif name == "bucket rule":
        b.hsml = b.hsml * rng.uniform(0.6, 1.4, size=b.n)
    elif name == "drift of few":  # most tiles stay near their cells, a few particles do not
        b.vx[::97] += [60.0, 30.0]
        b.xb, b.massb = b.xb[:0], b.massb[:0]
        b.params.wind_force = b.params.water_force = 0
    elif name.startswith("drift="):
        b.vx = b.vx + np.array([float(name[6:]), 0.5 * float(name[6:])])
        b.xb, b.massb = b.xb[:0], b.massb[:0]
        b.params.wind_force = b.params.water_force = 0
    return b


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("name", ["n=1", "n=2", "n=127", "n=128", "n=129", "n=257", "narrow", "sparse", "dense",
                                  "varied", "bucket rule", "drift of few", "drift=60", "drift=250", "drift=900"])
def test_tile_right_hand_side(gpu_lib, oracle_mod, name, precision):
    b = _basin(name)
    prm = b.params.copy()
    prm.precision = precision
    with Simp.from_basin(b, prm) as g:
        if name.startswith("drift"):
            g.time_integration(13)   # 13 of the 16 steps between sorts
        s = g.get_state()
        r = g.single_step(600.0)
        pairs = g.nnps()
    o = oracle_mod.Oracle(b.params, b.n, max(b.nb, 1))
    o.set_state(s["x"], s["vx"], s["mass"], s["rho"], s["hsml"], s["A"], s["h"], b.xb, b.massb, 1.0, 600.0)
    assert_same_pairs(pairs, o.nnps())
    ro = o.single_step(600.0)
    for k in ("dvxdt", "dhdt", "dAdt"):
        assert rel_l2(r[k], ro[k]) < TOL[precision], (name, k)


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("bfa, pressure, friction", [(1, 1, 0), (1, 1, 1), (1, 0, 1), (3, 0, 1)])
@pytest.mark.parametrize("denser", [1, 3, 9])
def test_tile_walls(gpu_lib, oracle_mod, denser, bfa, pressure, friction, precision):
    """Wall pairs at the usual spacing, more of them in a tile than its table
    holds, and more walls than its list holds (corner tiles see all three)."""
    b = _basin("walls")
    b.params.bfa, b.params.boundary_pressure, b.params.boundary_friction = bfa, pressure, friction
    t = np.arange(0.5, denser) / denser
    along = np.where(np.abs(b.xb[:, :1] - b.xb[:, :1].max()) < 1.0, [[0.0, 1.0]], [[1.0, 0.0]])
    b.xb = (b.xb[:, None, :] + (t[None, :, None] - 0.5) * along[:, None, :] * b.params.b_length / 3.0).reshape(-1, 2)
    b.massb = np.full(len(b.xb), b.mass.mean())
    prm = b.params.copy()
    prm.precision = precision
    with Simp.from_basin(b, prm) as g:
        r = g.single_step(600.0)
    o = oracle_mod.Oracle(b.params, b.n, b.nb)
    o.set_state(b.x, b.vx, b.mass, b.rho, b.hsml, b.A, b.h, b.xb, b.massb, 1.0, 600.0)
    ro = o.single_step(600.0)
    for k in ("dvxdt", "dhdt", "dAdt"):
        assert rel_l2(r[k], ro[k]) < TOL[precision], k


_ROOTS = """
#include "pass_common.cuh"
__global__ void roots(int n, const double *u, double *g, double *h) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) simp::pass::root_pair(u[i], g[i], h[i]);
}
extern "C" int run(int n, const double *u, double *g, double *h) {
    double *d;
    const size_t b = n * sizeof(double);
    if (cudaMalloc(&d, 3 * b) != cudaSuccess) return 1;
    cudaMemcpy(d, u, b, cudaMemcpyHostToDevice);
    roots<<<(n + 127) / 128, 128>>>(n, d, d + n, d + 2 * n);
    cudaMemcpy(g, d + n, b, cudaMemcpyDeviceToHost);
    cudaMemcpy(h, d + 2 * n, b, cudaMemcpyDeviceToHost);
    return cudaFree(d) != cudaSuccess;
}
"""


def test_root_pair(gpu_lib, tmp_path):
    """sqrt(u) and 1 / (2 sqrt(u)) of the pair passes in FP64, in 80-bit arithmetic.

    The corrections leave errors of second order (2^-78) and one rounding each,
    2^-53 at most, plus that of the correction itself (2^-39 of it): 1.001 * 2^-53.
    """
    (tmp_path / "roots.cu").write_text(_ROOTS)
    so = str(tmp_path / "roots.so")
    subprocess.run([build.nvcc(), "-shared", *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-I", build.INCLUDE,
                    "-I", build.CSRC, *build.host_compiler(), "-o", so, str(tmp_path / "roots.cu")], check=True)
    rng = np.random.default_rng(7)
    u = np.concatenate([2.0 ** rng.uniform(-120.0, 120.0, 200000), rng.uniform(1.0, 4.0, 200000),
                        [1.0, 4.0, 2.0, np.nextafter(1.0, 0.0), np.nextafter(4.0, 5.0)]])
    g, h = np.empty_like(u), np.empty_like(u)
    p = [a.ctypes.data_as(ctypes.c_void_p) for a in (u, g, h)]
    assert ctypes.CDLL(so).run(len(u), *p) == 0
    root = np.sqrt(u.astype(np.longdouble))
    assert np.finfo(np.longdouble).nmant >= 63
    assert np.max(np.abs(g / root - 1)) < 1.001 * 2.0 ** -53
    assert np.max(np.abs(2 * h * root - 1)) < 1.001 * 2.0 ** -53


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
def test_alone_and_among_many(gpu_lib, precision):
    """A basin gives the same bits in its own context and in a batch of so many
    tiles that the passes take their other launch form."""
    bs = [basins.make_basin(n, 1000.0, 3 + n, walls="+x-x+y-y", precision=precision) for n in (40, 370)]
    batch = Batch(bs[0].params, sum(b.n for b in bs), sum(b.nb for b in bs), len(bs))
    slots = [batch.add(b) for b in bs]
    batch.step(12)
    got = batch.get_state(slots[0])
    alone = Simp.from_basin(bs[0])
    alone.time_integration(12)
    want = alone.get_state()
    for k in ("x", "vx", "mass", "rho", "hsml", "A", "h"):
        assert np.array_equal(got[k], want[k]), k
