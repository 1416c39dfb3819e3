"""The raymarch's noise tables against hashing in place (needs a GPU).

A table holds the same function of the same lattice points, and a point
outside it is hashed in place, so the frame is the same bits with the tables
on and off: at times that put the lattice far from the origin (where a float
coordinate no longer resolves the table's margin), for every scene, with and
without a debug view, and on frames that the tiles do not divide.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene, debug, frame, time", [
    (0, 0, (97, 61), 0.0), (1, 0, (64, 48), 7.31), (2, 0, (33, 130), 1.0e4), (0, 4, (8, 4), 3.7), (1, 0, (96, 54), 2.5e6)])
def test_frame_with_and_without_tables(pkg, abi, scene, debug, frame, time):
    sim = pkg.FireSim(*frame, 40, 36, 28)
    for f in range(8):
        s = abi.validation_settings(f, scene=scene, width=frame[0], height=frame[1])
        sim.step(s)
    s.reset = 0
    s.renderDebugMode = debug
    frames = []
    for tables in (True, False):
        sim.set_hash_lattices(tables)
        sim.stages("light_build", "render", s, time)
        frames.append(sim.get("hdr"))
    sim.set_hash_lattices(True)
    sim.close()
    assert np.isfinite(frames[0]).all() and frames[0].max() > 0.0
    assert np.array_equal(frames[0].view(np.uint32), frames[1].view(np.uint32))
