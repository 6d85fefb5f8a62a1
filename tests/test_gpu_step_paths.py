"""A run's records do not depend on which lane flies a secondary: plain and
batched runs, pools of different size and the adjoint's replay agree exactly.
"""
import numpy as np
import pytest

import nebula_b200 as nb

pytestmark = pytest.mark.gpu


def _sorted(rec):
    return np.sort(np.ascontiguousarray(rec).view(np.dtype((np.void, 36))).ravel())


def _records(g, mats, pri, **kw):
    sim = nb.Simulation(g, mats, seed=77, **kw)
    sim.push(pri)
    sim.run()
    rec, c = sim.flush_detected(), sim.counters()
    sim.close()
    assert c["primaries_started"] + c["spawned"] == c["detected"] + c["terminated"]
    return rec, c


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 65])
def test_secondaries_flown_in_ended_lanes(inputs, n):
    """Plain and batched runs pack their warps differently; so do pools of
    different size and the adjoint's replay."""
    from nebula_b200.synth import primaries
    g = nb.Geometry.from_tri_file(inputs["grating.tri"])
    mats = [nb.Material.load(inputs["si.nmat"]), nb.Material.load(inputs["pmma.nmat"])]
    pri = primaries.raster_scan(n, 1, 1, 0.5, 500.0, 40.0, seed=4)
    ref, c = _records(g, mats, pri)
    for kw in ({"capacity": 32}, {"adjoint": True, "tally": (n, 1)}, {"walk_cells": 7}, {"block_size": 32}):
        rec, c2 = _records(g, mats, pri, **kw)
        assert np.array_equal(_sorted(ref), _sorted(rec)), kw
        assert all(c[k] == c2[k] for k in ("flights", "boundary", "elastic", "inelastic", "spawned", "terminated")), kw
    batch = nb.Batch([g], mats, capacity=1 << 10, record_capacity=1 << 16)
    batch.set_jobs([(0, 77, pri)])
    batch.run()
    rec, _ = batch.records()
    batch.close()
    assert np.array_equal(_sorted(ref), _sorted(rec))
