"""Bounded waits for a tile's copies.

A wait that nothing ends gives up within its limit and marks block and context;
a context so marked steps no further and reports it until its state is set
anew.
"""
import ctypes
import subprocess

import numpy as np
import pytest

from simp_b200 import basins, build
from simp_b200.simp import SIMP_ERR_TIMEOUT, Batch, Simp, SimpError

pytestmark = pytest.mark.gpu

_SRC = """
#include "tile.cuh"
using namespace simp;
using namespace simp::pass;
// one block waits for 16 bytes: their copy is started (copy != 0) or never is
__global__ void wait(int copy, const double2 *src, double2 *got, Scalars *sc, int *out, unsigned long long *ns) {
    __shared__ __align__(16) double2 dst;
    __shared__ __align__(8) unsigned long long bar;
    __shared__ int failed;
    const int t = threadIdx.x;
    if (t == 0) bar_init(&bar);
    if (t == kTile - 1) failed = failed_before(sc);
    __syncthreads();
    const bool before = failed < 0;
    if (t == 0) {
        bar_expect(&bar, 16);
        if (copy) bulk_copy(&dst, src, 16, &bar);
    }
    unsigned long long a, b;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(a));
    const bool ok = copies_arrive(&bar, 0, 6, &failed, &sc->flags);
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(b));
    __syncthreads();
    out[t] = (before ? 1 : 0) | (ok ? 2 : 0) | (failed == 6 ? 4 : 0);
    ns[t] = b - a;
    if (t == 0 && ok) *got = dst;
}
extern "C" int run(int copy, int flags, double *got, int *out, unsigned long long *ns, int *flags_out) {
    struct Mem { double2 src, got; Scalars sc; int out[kTile]; unsigned long long ns[kTile]; } h{}, *d = nullptr;
    h.src = make_double2(1.5, -2.5);
    h.sc.flags = flags;
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess) return 1;
    cudaMemcpy(d, &h, sizeof(h), cudaMemcpyHostToDevice);
    wait<<<1, kTile>>>(copy, &d->src, &d->got, &d->sc, d->out, d->ns);
    if (cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    got[0] = h.got.x;
    got[1] = h.got.y;
    for (int t = 0; t < kTile; ++t) out[t] = h.out[t], ns[t] = h.ns[t];
    *flags_out = h.sc.flags;
    return cudaFree(d) != cudaSuccess;
}
// marks a context as a wait that gave up would
extern "C" int mark(void *ctx) {
    simp_ctx *c = (simp_ctx *)ctx;
    if (cudaStreamSynchronize(c->stream) != cudaSuccess) return 1;
    const int v = FLAG_TIMEOUT;
    return cudaMemcpy(&c->sc->flags, &v, sizeof(v), cudaMemcpyHostToDevice) != cudaSuccess;
}
"""


@pytest.fixture(scope="module")
def probe(gpu_lib, tmp_path_factory):
    d = tmp_path_factory.mktemp("wait")
    (d / "wait.cu").write_text(_SRC)
    so = str(d / "wait.so")
    subprocess.run([build.nvcc(), "-shared", *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-I", build.INCLUDE,
                    "-I", build.CSRC, *build.host_compiler(), "-o", so, str(d / "wait.cu")], check=True)
    lib = ctypes.CDLL(so)
    lib.mark.argtypes = [ctypes.c_void_p]
    return lib


@pytest.mark.parametrize("copy, flags", [(1, 0), (1, 4), (0, 0)])
def test_wait_is_bounded(probe, copy, flags):
    got, out = (ctypes.c_double * 2)(), (ctypes.c_int * 128)()
    ns, flags_out = (ctypes.c_ulonglong * 128)(), ctypes.c_int()
    assert probe.run(copy, flags, got, out, ns, ctypes.byref(flags_out)) == 0
    before = 1 if flags else 0
    if copy:
        assert set(out) == {before | 2} and list(got) == [1.5, -2.5] and flags_out.value == flags
        assert max(ns) < 1e8
    else:
        assert set(out) == {4} and flags_out.value == 4
        assert max(ns) < 2e10       # two waits, a second each


def test_marked_context_stops_and_recovers(probe):
    b = basins.make_basin(40, 1000.0, 3, walls="+x-x")
    with Simp.from_basin(b) as g:
        g.time_integration(3)
        s = g.get_state()
        assert probe.mark(g.h) == 0
        for _ in range(2):
            with pytest.raises(SimpError) as e:
                g.time_integration(2)
            assert e.value.code == SIMP_ERR_TIMEOUT
        with pytest.raises(SimpError) as e:
            g.single_step(1.0)
        assert e.value.code == SIMP_ERR_TIMEOUT
        now = g.get_state()
        for k in ("x", "vx", "h", "A"):
            assert np.array_equal(now[k], s[k]), k
        g.set_state(b.x, b.vx, b.mass, b.rho, b.hsml, b.A, b.h, b.xb, b.massb, b.params.dt, 0.0)
        g.time_integration(3)
        again = g.get_state()
        for k in ("x", "vx", "h", "A"):
            assert np.array_equal(again[k], s[k]), k


def test_marked_batch_stops(probe):
    b = basins.make_basin(40, 1000.0, 3, walls="+x-x")
    with Batch(b.params, b.n, b.nb, 1) as g:
        g.add(b)
        g.step(3)
        assert probe.mark(g.h) == 0
        for _ in range(2):
            with pytest.raises(SimpError) as e:
                g.step(1)
            assert e.value.code == SIMP_ERR_TIMEOUT
