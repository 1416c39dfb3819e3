"""The multigrid's transfers on the smoothing's tiles (needs a GPU): levels that
halve every axis, some or one only, so that the correction and the residual are
taken on the tile or by a phase of their own; last passes of one to four half
sweeps; tiles that end inside the grid.  The solve equals the oracle's bit for
bit, as at every shape."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims, pre, post", [
    ((48, 40, 56), 1, 1), ((33, 32, 40), 1, 2), ((40, 33, 36), 2, 1), ((64, 48, 17), 2, 2), ((25, 27, 64), 1, 1), ((50, 36, 34), 4, 1),
    ((136, 24, 20), 3, 3)])
def test_multigrid_transfers_on_tiles_equal_the_oracle(pkg, abi, oracle_mod, dims, pre, post):
    p = abi.default_physics(*dims)
    p.mode, p.pressureTop = 1, 1
    d = (0.3 * np.random.default_rng(21).standard_normal(dims[::-1])).astype(np.float32)
    sim = pkg.FireSim(32, 16, *dims)
    sim.set_physics(p)
    sim.set_pressure_multigrid(3, pre, post)
    sim.set_pressure_tolerance(0.0, 1)
    sim.set("divergence", d)
    sim.set("pressure", np.zeros_like(d))
    sim.stages("pressure_sor", "pressure_sor", abi.FireSettings(), 0.0)
    o = oracle_mod.ConfigOracle(abi, 32, 16, *dims)
    o.set_physics(p)
    o.set_multigrid(3, pre, post, 0.0)
    o.set("divergence", d)
    o.set("pressure", np.zeros_like(d))
    o.stages("pressure_sor", "pressure_sor")
    a, b = sim.get("pressure"), o.get("pressure")
    sim.close()
    assert np.abs(b).max() > 0.0
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
