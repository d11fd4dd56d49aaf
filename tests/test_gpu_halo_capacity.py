"""The same bits whatever a tile's halo holds: at the smallest capacities tiles
are cut short, taken in parts and, where there is no spare tile left, read
their neighbours from global memory; at the largest, every tile is whole.
Right-hand sides and steps, past a sort, of every pass that uses the tiles.
"""
import numpy as np
import pytest

from helpers import smooth_velocity
from simp_b200 import _lib, basins, build
from simp_b200.params import (ART_VISC_MON, PASSES_GATHER, PASSES_TILED, PREC_FP64, PREC_MIXED, SKF_CUBIC, SKF_GAUSSIAN,
                              SKF_WENDLAND_C6)
from simp_b200.simp import Simp

pytestmark = pytest.mark.gpu

FORMS = {
    "cubic": dict(skf=SKF_CUBIC),
    "wendland": dict(skf=SKF_WENDLAND_C6),
    "gaussian": dict(skf=SKF_GAUSSIAN),
    "varied": dict(skf=SKF_CUBIC),
    "continuity": dict(skf=SKF_GAUSSIAN, den_alg=2, xsph_regularization=1, artificial_visc=1, art_visc_alg=ART_VISC_MON),
    "summation": dict(skf=SKF_CUBIC, den_alg=1),
    "evolving": dict(skf=SKF_WENDLAND_C6, sle=2, tse=2),
}


def _basin(form, precision):
    b = basins.make_basin(48, 2000.0, 9, walls="+x-x+y-y", precision=precision, dt=0.5)
    b.vx = smooth_velocity(b.x, b.L, amp=2.0, seed=9)
    b.h = 1.0 + 0.5 * np.sin(b.x[:, 0] / 9000.0)
    b.rho = 900.0 * b.h
    b.mass = b.rho * 4.0e6
    if form == "varied":
        b.hsml = b.hsml * np.random.default_rng(9).uniform(1.0, 1.25, size=b.n)
    b.params.boundary_friction = 1
    for k, v in FORMS[form].items():
        setattr(b.params, k, v)
    return b


def _run(b, passes, lib=None):
    with Simp.from_basin(b, lib=lib) as g:
        g.set_passes(*passes)
        r = g.single_step(600.0)
        g.time_integration(20)
        return {**r, **g.get_state()}


def _same(got, want):
    for k, v in want.items():
        if isinstance(v, np.ndarray):
            assert np.isfinite(v).all(), k
        assert np.array_equal(got[k], v), k


@pytest.mark.parametrize("cap", [64, 96, 204, 528, 1344])
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("form", sorted(FORMS))
def test_same_bits_at_any_capacity(gpu_lib, form, precision, cap):
    b = _basin(form, precision)
    _same(_run(b, (PASSES_TILED, 128, cap)), _run(b, (PASSES_GATHER, 256, 1024)))


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
def test_capacity_changes_between_steps(gpu_lib, precision):
    b = _basin("cubic", precision)
    with Simp.from_basin(b) as g, Simp.from_basin(b) as h:
        for cap in (64, 1344, 96, 832, 64):
            g.set_passes(PASSES_TILED, 128, cap)
            g.time_integration(5)
            h.time_integration(5)
            _same(g.get_state(), h.get_state())
        g.set_passes(PASSES_GATHER)
        g.time_integration(5)
        h.time_integration(5)
        _same(g.get_state(), h.get_state())


@pytest.mark.parametrize("form", ["varied", "continuity", "summation"])
def test_checks_pass_at_the_smallest_capacity(gpu_lib, form):
    build.build(variant="checked")
    b = _basin(form, PREC_FP64)
    _same(_run(b, (PASSES_TILED, 128, 64), lib=_lib.load(build.LIB_CHECKED)), _run(b, (PASSES_GATHER, 256, 1024)))
