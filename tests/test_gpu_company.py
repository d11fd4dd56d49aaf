"""A basin's results do not depend on its company: bit for bit the same in its
own context and in a batch that another basin joins and leaves midway.  Among
the others is one whose hsml varies (the passes then read every neighbour's
hsml) and ones of so many tiles that the passes take their other launch form,
with fewer registers per thread and the walls from the cell lists.
"""
import numpy as np
import pytest

from helpers import smooth_velocity
from simp_b200 import basins
from simp_b200.params import PREC_FP64, PREC_MIXED, SKF_CUBIC, SKF_GAUSSIAN, SKF_WENDLAND_C6
from simp_b200.simp import Batch, Simp

pytestmark = pytest.mark.gpu

KEYS = ("x", "vx", "mass", "rho", "hsml", "A", "h")


def _basin(nside, seed, skf, precision, varied):
    b = basins.make_basin(nside, 1000.0, seed, walls="+x-x+y-y", precision=precision, skf=skf, dt=0.3)
    b.vx = smooth_velocity(b.x, b.L, amp=2.0, seed=seed)
    b.h = 1.0 + 0.5 * np.sin(b.x[:, 0] / 9000.0)
    b.A = 0.9 + 0.1 * np.cos(b.x[:, 1] / 7000.0)
    b.rho = 900.0 * b.h
    b.mass = b.rho * 1.0e6
    if varied:
        b.hsml = b.hsml * np.random.default_rng(seed).uniform(1.0, 1.25, size=b.n)
    b.params.boundary_friction = 1
    return b


@pytest.mark.parametrize("company", [(30, True), (380, False), (380, True)])
@pytest.mark.parametrize("varied", [False, True])
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("skf", [SKF_CUBIC, SKF_WENDLAND_C6, SKF_GAUSSIAN])
def test_same_bits_in_any_company(gpu_lib, skf, precision, varied, company):
    b = _basin(40, 7, skf, precision, varied)
    other = _basin(company[0], 8, skf, precision, company[1])
    with Batch(b.params, b.n + other.n, b.nb + other.nb, 2) as batch:
        slot = batch.add(b)
        batch.step(3)
        guest = batch.add(other)
        batch.step(17)              # past a sort
        batch.remove(guest)
        batch.step(4)
        got = batch.get_state(slot)
    with Simp.from_basin(b) as alone:
        alone.time_integration(24)
        want = alone.get_state()
    for k in KEYS:
        assert np.isfinite(want[k]).all()
        assert np.array_equal(got[k], want[k]), k
