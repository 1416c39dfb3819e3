"""The multigrid's smoothing tiles at their edges (needs a GPU): grids that the
tile shapes do not divide, rows whose length is not a multiple of 4 or is odd,
and smoothing counts that take one pass or several.  The solve equals the
oracle's bit for bit, as at every shape."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims, pre, post", [
    ((40, 36, 52), 2, 2), ((66, 34, 18), 2, 2), ((35, 64, 40), 2, 2), ((130, 20, 36), 1, 1), ((68, 36, 20), 3, 1), ((37, 44, 24), 2, 3),
    ((96, 40, 24), 4, 4), ((64, 64, 64), 1, 3)])
def test_multigrid_with_ragged_tiles_equals_the_oracle(pkg, abi, oracle_mod, dims, pre, post):
    p = abi.default_physics(*dims)
    p.mode, p.pressureTop = 1, 1
    d = (0.3 * np.random.default_rng(9).standard_normal(dims[::-1])).astype(np.float32)
    sim = pkg.FireSim(32, 16, *dims)
    sim.set_physics(p)
    sim.set_pressure_multigrid(2, pre, post)
    sim.set_pressure_tolerance(0.0, 1)
    sim.set("divergence", d)
    sim.set("pressure", np.zeros_like(d))
    sim.stages("pressure_sor", "pressure_sor", abi.FireSettings(), 0.0)
    o = oracle_mod.ConfigOracle(abi, 32, 16, *dims)
    o.set_physics(p)
    o.set_multigrid(2, pre, post, 0.0)
    o.set("divergence", d)
    o.set("pressure", np.zeros_like(d))
    o.stages("pressure_sor", "pressure_sor")
    a, b = sim.get("pressure"), o.get("pressure")
    sim.close()
    assert np.abs(b).max() > 0.0
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
