"""The config physics' light and raymarch where their sample counts make the
brick flags worth building (needs a GPU): grids that the bricks and the build's
warps do not divide, from empty to largely full, with the cells that the build
looks at first set or clear against the rest.  As beside empty bricks, the same
state with the smallest float as the heat of every cell that no hot cell touches
takes every sample, and the pictures are equal bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_config_empty_space import _pictures, _state

pytestmark = pytest.mark.gpu


def _fill(dims, kind, rng):
    if kind in ("nothing", "corners", "sparse", "signed", "overflow"):
        return _state(dims, kind, rng)
    nx, ny, nz = dims
    first = np.zeros(dims[::-1], bool)  # the 64 cells that tell a largely full grid
    first[np.ix_(*[[(2 * k + 1) * n // 8 for k in range(4)] for n in (nz, ny, nx)])] = True
    mask = np.zeros(dims[::-1], bool)
    if kind == "lower half":
        mask[:, :ny // 2] = True
    elif kind == "most":
        mask[:, :, :] = rng.random(dims[::-1]) < 0.5
        mask &= ~first
    elif kind == "first cells":
        mask = first
    elif kind == "full but a corner":
        mask[:, :, :] = True
        mask[:nz // 3, :ny // 3, :nx // 3] = False
    f = {}
    for n in ("heat", "fuel", "soot"):
        f[n] = np.where(mask, rng.random(dims[::-1]), 0.0).astype(np.float32)
    return f


@pytest.mark.parametrize("kind", ["nothing", "corners", "sparse", "signed", "overflow", "lower half", "most", "first cells", "full but a corner"])
@pytest.mark.parametrize("dims, samples", [((8, 8, 8), 4096), ((37, 29, 45), 900), ((61, 64, 10), 900), ((130, 20, 33), 900)])
def test_full_and_empty_grids_with_many_samples(pkg, abi, dims, samples, kind):
    frame = (72, 40)
    sim = pkg.FireSim(*frame, *dims)
    p = abi.default_physics(*dims)
    p.mode, p.primarySamples, p.lightSamples = 1, samples, samples
    sim.set_physics(p)
    sim.reset()
    fields = _fill(dims, kind, np.random.default_rng(8))
    a = _pictures(sim, abi, frame, fields, None)
    pad = np.pad(fields["heat"] != 0.0, 1)
    near = np.zeros(dims[::-1], bool)
    for k in np.ndindex(3, 3, 3):
        near |= pad[tuple(slice(o, o + n) for o, n in zip(k, dims[::-1]))]
    every = dict(fields, heat=np.where(near, fields["heat"], np.float32(1e-45)).astype(np.float32))
    b = _pictures(sim, abi, frame, every, None)
    sim.close()
    for x, y in zip(a, b):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))


def test_a_frame_of_one_column(pkg, abi):
    """131,072 rays in one column: more rows than a grid of two-row blocks has."""
    sim = pkg.FireSim(1, 131072, 24, 20, 16)
    p = abi.default_physics(24, 20, 16)
    p.mode, p.primarySamples = 1, 128
    sim.set_physics(p)
    sim.reset()
    sim.set("soot", np.full((16, 20, 24), 0.5, np.float32))
    sim.stages("light_build", "render", abi.FireSettings(width=1, height=131072), 0.0)
    hdr = sim.get("hdr")
    sim.close()
    assert np.isfinite(hdr).all() and hdr[..., 3].max() > 0.5
