"""A basin whose state turns non-finite.

It is flagged and carried without being searched any more (a batch) or
reported (a single basin).  Its walls are on all four sides, and its tiles
outnumber those resident at once, so that some of them start their stress
pass, with the wall sums' barriers, while others set the flag.
"""
import numpy as np
import pytest

from helpers import smooth_velocity
from simp_b200 import basins
from simp_b200.params import PREC_FP64, PREC_MIXED
from simp_b200.simp import SIMP_ERR_NONFINITE, Batch, Simp, SimpError

pytestmark = pytest.mark.gpu

KEYS = ("x", "vx", "mass", "rho", "hsml", "A", "h")
FLAG_NONFINITE = 1


def _basin(nside, seed, precision):
    b = basins.make_basin(nside, 1000.0, seed, walls="+x-x+y-y", precision=precision)
    b.vx = smooth_velocity(b.x, b.L, amp=0.4, seed=seed)
    b.params.dt = 0.25
    return b


def _overflowing(nside, seed, precision):
    """Its drag overflows in the first half step, at a particle in the first tile."""
    b = _basin(nside, seed, precision)
    b.vx[nside // 2, 0] = 1e200
    return b


@pytest.mark.parametrize("nside", [40, 330])
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
def test_batch_flags_the_basin_and_keeps_the_others(gpu_lib, precision, nside):
    good = [_basin(45, 3, precision), _basin(70, 4, precision)]
    bad = _overflowing(nside, 5, precision)
    order = [good[0], bad, good[1]]
    batch = Batch(bad.params, sum(b.n for b in order), sum(b.nb for b in order), 3)
    slots = [batch.add(b) for b in order]
    batch.step(1)
    assert [batch.info(s)["flags"] & FLAG_NONFINITE for s in slots] == [0, FLAG_NONFINITE, 0]
    batch.step(19)                  # past a sort
    for b, s in ((good[0], slots[0]), (good[1], slots[2])):
        got = batch.get_state(s)
        with Batch(b.params, b.n, b.nb, 1) as alone:
            sa = alone.add(b)
            alone.step(20)
            want = alone.get_state(sa)
        for k in KEYS:
            assert np.array_equal(got[k], want[k]), k
    batch.close()


def test_single_basin_reports_and_recovers(gpu_lib):
    bad, good = _overflowing(330, 5, PREC_FP64), _basin(330, 5, PREC_FP64)
    g = Simp.from_basin(bad)
    with pytest.raises(SimpError) as e:
        g.time_integration(2)
    assert e.value.code == SIMP_ERR_NONFINITE
    g.close()
    with Simp.from_basin(good) as h:
        h.time_integration(2)
        assert np.isfinite(h.get_state()["vx"]).all()
