"""What once sent tiles, or parts of them, to global memory: particles of more
candidates than a list holds, which find their pairs in the tile's halo now,
among others of their tile that have lists; and sparse cell rows, whose tiles
are cut as short as their halo needs, also when other basins join the batch.

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
from simp_b200.simp import Batch, Simp

pytestmark = pytest.mark.gpu

_SRC = """
#include <vector>
#include "tile.cuh"
using namespace simp;
using namespace simp::pass;
// parts of the tiles in use by kind, and the particles whose list is too short
extern "C" int tiles(void *ctx, int slot, int *kinds, int *over) {
    simp_ctx *c = (simp_ctx *)ctx;
    if (cudaStreamSynchronize(c->stream) != cudaSuccess) return 1;
    std::vector<Chunk> ch(c->nchunks);
    std::vector<Halo> h((size_t)c->nchunks * kParts);
    std::vector<int> cnt(c->n);
    Inst I;
    cudaMemcpy(ch.data(), c->chunks, ch.size() * sizeof(Chunk), cudaMemcpyDeviceToHost);
    cudaMemcpy(h.data(), c->halos, h.size() * sizeof(Halo), cudaMemcpyDeviceToHost);
    cudaMemcpy(cnt.data(), c->pair_count, cnt.size() * sizeof(int), cudaMemcpyDeviceToHost);
    if (cudaMemcpy(&I, c->inst_dev + slot, sizeof(I), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    for (int k = 0; k < c->nchunks; ++k) {
        if (ch[k].q != slot || ch[k].spare >= I.spares) continue;
        for (int p = ch[k].p0; p < ch[k].p1;) {
            const Halo &r = h[(size_t)k * kParts + ((p - ch[k].p0) >> (ch[k].p1 - ch[k].p0 <= kParts ? 0 : 3))];
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
    lib.tiles.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]

    def look(sim, slot=0):
        kinds, over = (ctypes.c_int * 3)(), ctypes.c_int(0)
        assert lib.tiles(sim.h, slot, kinds, ctypes.byref(over)) == 0
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


def _sparse(every, seed=5):
    """Twelve full rows, one of every `every`-th particle, and full rows again above a gap."""
    b = basins.make_basin(300, 2000.0, seed, walls="+x-x", dt=0.5)
    b.vx = smooth_velocity(b.x, b.L, amp=0.3, seed=4)
    row, col = (np.floor(b.x[:, k] / b.dx).astype(int) for k in (1, 0))
    keep = (row < 12) | ((row == 14) & (col % every == every // 2)) | ((row >= 17) & (row < 24))
    for k in ("x", "vx", "mass", "rho", "hsml", "A", "h"):
        setattr(b, k, np.ascontiguousarray(getattr(b, k)[keep]))
    return b


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("every", [3, 25, 140, 290])
def test_sparse_rows(gpu_lib, tiles, oracle_mod, every, precision):
    b = _sparse(every)
    prm = b.params.copy()
    prm.precision = precision
    with Simp.from_basin(b, prm) as g:
        r = g.single_step(600.0)
        kinds, _ = tiles(g)
    assert kinds[1] > 0 and kinds[0] == kinds[2] == 0, kinds
    ro = oracle_mod.Oracle.from_basin(b, b.params).single_step(600.0)
    for k in ("dvxdt", "dhdt", "dAdt"):
        assert rel_l2(r[k], ro[k]) < (1e-11 if precision == PREC_FP64 else 2e-6), k


def test_sparse_rows_stay_cut_as_others_join(gpu_lib, tiles):
    b, other = _sparse(25), _sparse(140, seed=6)
    with Batch(b.params, b.n + other.n, b.nb + other.nb, 2) as g:
        slot = g.add(b)
        g.step(2)
        guest = g.add(other)
        g.step(2)
        for s in (slot, guest):
            kinds, _ = tiles(g, s)
            assert kinds[1] > 0 and kinds[0] == kinds[2] == 0, (s, kinds)
        got = g.get_state(slot)
    with Simp.from_basin(b) as alone:
        alone.time_integration(4)
        want = alone.get_state()
    for k in ("x", "vx", "h", "A"):
        assert np.array_equal(got[k], want[k]), k


def test_parts_after_motion(gpu_lib, tiles):
    """Five rows of cells of a large basin, whose tiles hold a halo of 576.  A cell
    is three lattice spacings wide: 15 lattice rows of 38 columns, some 14 of
    which lie beside the part.  A part then has 24 columns of the cell row's three
    lattice rows, 72 particles, so that a tile takes two parts, three at times."""
    b = basins.make_basin(384, 2000.0, 5, walls="", dt=1.0)
    b.vx = smooth_velocity(b.x, b.L, amp=0.3, seed=4) + np.array([60.0, 30.0])
    b.params.wind_force = b.params.water_force = 0
    with Simp.from_basin(b) as g:
        g.time_integration(14)          # (of 16 between sorts)
        kinds, _ = tiles(g)
    whole = -(-b.n // 128)
    assert kinds[0] == kinds[2] == 0, kinds
    assert 1.5 < kinds[1] / whole < 2.6, kinds[1] / whole
