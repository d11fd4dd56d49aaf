"""The pair passes' tiles where they can go wrong: tiles of a few particles and
around a full one, tiles that span several cell rows, sparse cell rows whose
halo has to be cut, more neighbours than a list holds, varying hsml with and
without the reference's bucket rule, and lists that motion outdates (built
again between sorts, over a wider stencil, and beyond the widest one).

One right-hand side at the state reached, against the oracle at that state.
The bars are those of the other right-hand-side tests: 1e-11 relative L2 in
FP64, where only the order of the sums differs, 2e-6 in mixed precision.
"""
import numpy as np
import pytest

from helpers import assert_same_pairs, rel_l2, smooth_velocity
from simp_b200 import basins
from simp_b200.params import PREC_FP64, PREC_MIXED
from simp_b200.simp import Simp

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
    elif name.startswith("drift="):
        b.vx = b.vx + np.array([float(name[6:]), 0.5 * float(name[6:])])
        b.xb, b.massb = b.xb[:0], b.massb[:0]
        b.params.wind_force = b.params.water_force = 0
    return b


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("name", ["n=1", "n=2", "n=127", "n=128", "n=129", "n=257", "narrow", "sparse", "dense",
                                  "varied", "bucket rule", "drift=60", "drift=250", "drift=900"])
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
