"""The served stream's memory budget: the tiles that the batch keeps for every
basin it may hold count towards it, beside what it keeps per particle."""
import numpy as np
import pytest

from simp_b200 import basins, serve
from simp_b200.simp import Batch, SimpError

pytestmark = pytest.mark.gpu

TILE_LISTS = 44 * 128 * 2      # bytes: a tile's lists, the largest part of what it keeps
PER_BASIN = 4                  # tiles kept per basin: a partial one and three spare ones


def _capacity(params, budget, instances, **kw):
    with serve.Server(params, budget, max_instances=instances, max_request_particles=1000, **kw) as s:
        return s.stats()["capacity_particles"]


def test_budget_counts_the_tiles_of_every_basin(gpu_lib):
    prm = basins.instance(0, 1000).params
    few, many = (_capacity(prm, 3.0e8, k) for k in (2, 1024))
    per = 3.0e8 / few              # bytes per particle, at least
    assert (few - many) * per > 1000 * PER_BASIN * TILE_LISTS
    assert many > 0.5 * few


@pytest.mark.parametrize("spot", [0, 2])
def test_a_tight_budget_holds_fewer_basins(gpu_lib, spot):
    """It would hold the largest request but not 1024 basins' tiles: still accepted, and served."""
    reqs = [serve.Request(basins.instance(k, 900), 6 + k, 0.0) for k in range(5)]
    budget = (1.3 + 2.6 * (spot > 0)) * 1000 * 1250.0
    with serve.Server(reqs[0].basin.params, budget, max_instances=1024, max_request_particles=1000, spot_every=spot) as s:
        assert s.stats()["capacity_particles"] * 600.0 < budget
        ids = [s.submit(r) for r in reqs]
        s.run()
        assert s.stats()["completed"] == len(reqs)
        for i, r in zip(ids, reqs):
            with Batch(r.basin.params, r.basin.n, max(r.basin.nb, 1), 1) as alone:
                slot = alone.add(r.basin)
                alone.step(r.nsteps)
                assert np.array_equal(s.outputs[i]["vx"], alone.get_state(slot)["vx"])


@pytest.mark.parametrize("instances", [2, 1024])
def test_a_budget_of_just_the_largest_request_is_accepted(gpu_lib, instances):
    """The tiles of the fewest basins a batch may hold refuse no budget that holds the largest request itself."""
    prm = basins.instance(0, 1000).params
    per = 3.0e8 / (_capacity(prm, 6.0e8, 2) - _capacity(prm, 3.0e8, 2))   # bytes per particle, to 1e-5
    n = 100_000
    with serve.Server(prm, per * n * (1.0 + 1e-4), max_instances=instances, max_request_particles=n) as s:
        assert s.stats()["capacity_particles"] == n
    with pytest.raises(SimpError):
        serve.Server(prm, per * n * (1.0 - 1e-4), max_instances=instances, max_request_particles=n)
