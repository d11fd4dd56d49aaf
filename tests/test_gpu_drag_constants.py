"""The drag factors c_wind rho_air / rho_ice and c_water rho_water / rho_ice, each
within one rounding (2^-53, and 2^-61 of the extended arithmetic they are worked
out in) of the exact rational.  What they are off by is the same for every
particle, so that no sum averages it away."""
from fractions import Fraction

import numpy as np
import pytest

from simp_b200 import basins
from simp_b200.simp import Simp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c, rho", [(1.2e-3, 1.3), (5.5e-3, 1026.0), (1.3e-3, 1.25), (2e-3, 1.3), (1e-3, 1.29)])
@pytest.mark.parametrize("rho_ice", [900.0, 910.0, 917.0])
@pytest.mark.parametrize("water", [False, True])
def test_rounded_once(gpu_lib, water, rho_ice, c, rho):
    """Particles too far apart for pairs, 1 m thick, at a relative velocity of 1 m/s: the rate is the factor."""
    b = basins.make_basin(3, 1000.0, 1, walls="")
    p = b.params
    p.rho_ice, p.wind_force, p.water_force = rho_ice, int(not water), int(water)
    if water:
        p.c_water, p.rho_water, p.current_u, p.current_v = c, rho, 1.0, -1.0
    else:
        p.c_wind, p.rho_air, p.wind_u, p.wind_v = c, rho, 1.0, -1.0
    b.x = b.x * 10.0
    b.vx, b.h, b.A, b.rho = np.zeros_like(b.x), np.ones(b.n), np.ones(b.n), np.full(b.n, rho_ice)
    with Simp.from_basin(b) as g:
        a = g.single_step(60.0)["dvxdt"]
    want = Fraction(c) * Fraction(rho) / Fraction(rho_ice)
    for k in range(b.n):
        assert a[k, 0] == -a[k, 1]
        assert abs(Fraction(float(a[k, 0])) / want - 1) < Fraction(2) ** -53 + Fraction(2) ** -61
