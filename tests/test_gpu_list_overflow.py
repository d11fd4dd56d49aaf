"""Particles of more candidates than a list holds, among others of their tile
that have lists: they find their pairs in the tile's halo, and no tile is sent
to global memory for them.

The bars are those of the other comparisons: 1e-11 of a right-hand side in FP64
(2e-6 mixed), where only the order of the sums differs, and 1e-9 after ten steps
of the regularised and the summed-density forms.
"""
import ctypes
import subprocess

import numpy as np
import pytest

from helpers import rel_l2, smooth_velocity
from simp_b200 import basins, build
from simp_b200.params import ART_VISC_MON, PREC_FP64, PREC_MIXED
from simp_b200.simp import Simp

pytestmark = pytest.mark.gpu

_SRC = """
#include <vector>
#include "tile.cuh"
using namespace simp;
using namespace simp::pass;
// parts of the tiles in use by kind, and the particles whose list is too short
extern "C" int tiles(void *ctx, int *kinds, int *over) {
    simp_ctx *c = (simp_ctx *)ctx;
    constexpr int parts = kTile / kPartMin;
    if (cudaStreamSynchronize(c->stream) != cudaSuccess) return 1;
    std::vector<Chunk> ch(c->nchunks);
    std::vector<Halo> h((size_t)c->nchunks * parts);
    std::vector<int> cnt(c->n);
    Inst I;
    cudaMemcpy(ch.data(), c->chunks, ch.size() * sizeof(Chunk), cudaMemcpyDeviceToHost);
    cudaMemcpy(h.data(), c->halos, h.size() * sizeof(Halo), cudaMemcpyDeviceToHost);
    cudaMemcpy(cnt.data(), c->pair_count, cnt.size() * sizeof(int), cudaMemcpyDeviceToHost);
    if (cudaMemcpy(&I, c->inst_dev, sizeof(I), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    for (int k = 0; k < c->nchunks; ++k) {
        if (ch[k].spare >= I.spares) continue;
        for (int p = ch[k].p0; p < ch[k].p1;) {
            const Halo &r = h[(size_t)k * parts + (p - ch[k].p0) / kPartMin];
            if (r.size < 1 || r.kind < 0 || r.kind > 2) return 3;
            ++kinds[r.kind];
            p += r.size;
        }
    }
    for (int v : cnt) *over += v > kListRows;
    return 0;
}
"""


@pytest.fixture(scope="module")
def tiles(gpu_lib, tmp_path_factory):
    d = tmp_path_factory.mktemp("tiles")
    (d / "t.cu").write_text(_SRC)
    so = str(d / "t.so")
    subprocess.run([build.nvcc(), "-shared", *build.ARCH, "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-I", build.INCLUDE,
                    "-I", build.CSRC, *build.host_compiler(), "-o", so, str(d / "t.cu")], check=True)
    lib = ctypes.CDLL(so)
    lib.tiles.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]

    def look(sim):
        kinds, over = (ctypes.c_int * 3)(), ctypes.c_int(0)
        assert lib.tiles(sim.h, kinds, ctypes.byref(over)) == 0
        return list(kinds), over.value
    return look


def _basin(**kw):
    b = basins.make_basin(60, 2000.0, 5, walls="+x-y", dt=0.5, jitter=0.25)
    b.vx = smooth_velocity(b.x, b.L, amp=0.3, seed=4)
    b.h = 1.0 + 0.5 * np.sin(b.x[:, 0] / 9000.0)
    b.rho = 900.0 * b.h
    b.mass = b.rho * 4.0e6
    b.hsml = b.hsml * (3.55 / 2.4)
    for k, v in kw.items():
        setattr(b.params, k, v)
    return b


FORMS = {"plain": {}, "uneven": {},
         "continuity": dict(den_alg=2, xsph_regularization=1, artificial_visc=1, art_visc_alg=ART_VISC_MON),
         "summation": dict(den_alg=1)}


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("form", sorted(FORMS))
def test_long_lists(gpu_lib, tiles, oracle_mod, form, precision):
    b = _basin(**FORMS[form])
    if form == "uneven":
        b.hsml = b.hsml * np.random.default_rng(2).uniform(0.95, 1.05, size=b.n)
    prm = b.params.copy()
    prm.precision = precision
    o = oracle_mod.Oracle.from_basin(b, b.params)
    o.set_regularization_form(False)
    with Simp.from_basin(b, prm) as g:
        r, ro = g.single_step(600.0), o.single_step(600.0)
        kinds, over = tiles(g)
    for k in ("dvxdt", "dhdt", "dAdt"):
        assert rel_l2(r[k], ro[k]) < (1e-11 if precision == PREC_FP64 else 2e-6), k
    assert kinds[1] > 0 and kinds[0] == kinds[2] == 0, kinds
    assert 10 < over < 0.9 * b.n, over
    if precision == PREC_MIXED or form in ("plain", "uneven"):
        return
    o = oracle_mod.Oracle.from_basin(b, b.params)
    o.set_regularization_form(False)
    with Simp.from_basin(b, prm) as g:
        g.time_integration(10)
        s = g.get_state()
    o.step(10)
    so = o.get_state()
    for k in ("x", "vx", "h", "A", "rho"):
        ref = b.x if k == "x" else 0.0
        assert rel_l2(s[k] - ref, so[k] - ref) < 1e-9, k
