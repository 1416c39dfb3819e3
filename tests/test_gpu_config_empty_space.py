"""The config physics' light and raymarch pass over empty bricks (needs a GPU):
grids that the bricks and the build's warps do not divide, matter at corners and
faces of the grid, nowhere and everywhere, negative zeros, and the values that a
sample of nothing may not be left out beside (an infinite transmittance or
remaining view); rays of several lanes each and, at the last size, of one.  The
same state with the smallest float as the heat of every cell that no hot cell
touches has hardly an empty brick, and that heat, which no sample interpolates
with another (it could break a rounding's tie), vanishes in every sum; the
pictures are equal bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(dims, kind, rng):
    f = {n: np.zeros(dims[::-1], np.float32) for n in ("heat", "fuel", "soot")}
    if kind == "corners":
        f["soot"][0, 0, 0] = f["soot"][-1, -1, -1] = 2.0
        f["heat"][-1, 0, 0] = f["fuel"][0, -1, -1] = 0.7
    elif kind != "nothing":
        mask = rng.random(dims[::-1]) < (1.0 if kind == "full" else 0.004)
        for a in f.values():
            a[mask] = rng.random(int(mask.sum())).astype(np.float32)
    if kind == "signed":
        f["soot"][f["soot"] == 0.0] = -0.0
        f["fuel"][f["fuel"] != 0.0] *= -1.0
    if kind == "overflow":
        f["soot"][f["soot"] != 0.0] = -3.0e4
    return f


def _pictures(sim, abi, frame, fields, light):
    s = abi.FireSettings(width=frame[0], height=frame[1])
    for n, a in fields.items():
        sim.set(n, a)
    out = []
    sim.stages("light_build", "render", s, 0.0)
    out += [sim.get("config_transmittance"), sim.get("hdr")]
    if light is not None:  # a render of its own, with the caller's transmittance
        sim.set("config_transmittance", light)
    sim.stages("render", "render", s, 0.0)
    return out + [sim.get("hdr")]


@pytest.mark.parametrize("kind", ["nothing", "corners", "sparse", "signed", "full", "overflow", "light"])
@pytest.mark.parametrize("dims, frame", [((8, 8, 8), (16, 16)), ((37, 29, 45), (72, 40)), ((61, 64, 10), (45, 33)), ((130, 20, 33), (72, 40)),
                                         ((104, 102, 101), (400, 330))])
def test_passing_over_empty_bricks_changes_no_bit(pkg, abi, dims, frame, kind):
    rng = np.random.default_rng(3)
    sim = pkg.FireSim(*frame, *dims)
    p = abi.default_physics(*dims)
    p.mode = 1
    sim.set_physics(p)
    sim.reset()
    fields = _state(dims, kind, rng)
    light = None
    if kind == "light":
        light = sim.get("config_transmittance")
        light.reshape(-1)[::7] = np.inf
    a = _pictures(sim, abi, frame, fields, light)
    pad = np.pad(fields["heat"] != 0.0, 1)
    near = np.zeros(dims[::-1], bool)
    for k in np.ndindex(3, 3, 3):
        near |= pad[tuple(slice(a, a + n) for a, n in zip(k, dims[::-1]))]
    dense = dict(fields, heat=np.where(near, fields["heat"], np.float32(1e-45)).astype(np.float32))
    b = _pictures(sim, abi, frame, dense, light)
    sim.close()
    for x, y in zip(a, b):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))


@pytest.mark.parametrize("kind", ["nothing", "corners", "sparse", "signed", "full", "overflow", "exit"])
@pytest.mark.parametrize("samples", [1, 10, 96])
def test_rays_of_four_lanes_equal_rays_of_one(pkg, abi, samples, kind):
    """A frame of 648 x 360 has more rays than get four lanes each; the middle
    pixels of its 9 x 9 blocks are the rays of the 72 x 40 frame.  exit: matter
    at the box's far wall only, where the view turns infinite at the last sample."""
    dims = (40, 33, 37)
    fields = _state(dims, "nothing" if kind == "exit" else kind, np.random.default_rng(5))
    if kind == "exit":
        fields["soot"][0] = fields["soot"][-1] = fields["soot"][:, :, 0] = fields["soot"][:, :, -1] = -3.0e4
    hdr = []
    for frame in ((72, 40), (648, 360)):
        sim = pkg.FireSim(*frame, *dims)
        p = abi.default_physics(*dims)
        p.mode, p.primarySamples = 1, samples
        sim.set_physics(p)
        sim.reset()
        for n, a in fields.items():
            sim.set(n, a)
        sim.stages("light_build", "render", abi.FireSettings(width=frame[0], height=frame[1]), 0.0)
        hdr.append(sim.get("hdr").reshape(frame[1], frame[0], 4))
        sim.close()
    few, many = hdr[0], np.ascontiguousarray(hdr[1][4::9, 4::9])
    assert np.array_equal(np.isnan(few), np.isnan(many))
    assert np.array_equal(np.where(np.isnan(few), 0.0, few), np.where(np.isnan(many), 0.0, many))
