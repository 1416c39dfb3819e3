"""The multigrid solve where its largest tile (32 x 16 x 16 cells) carries the
finest level, and where a level exceeds the L2, so that the next tile's rows are
prefetched (needs a GPU): grids that the tile does not divide, odd rows, kept
axes, one to four sweeps, and a coarsest level in global memory, beside which
smaller tiles are taken.  The solve equals the oracle's bit for bit, as at
every shape, and scenes of a batch, whose levels share one tile, get the bits
that they have alone."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_batch import _bits_equal, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims, pre, post", [
    ((98, 88, 96), 2, 2), ((100, 90, 92), 1, 2), ((98, 90, 94), 2, 2), ((127, 96, 98), 2, 1), ((99, 110, 112), 1, 1), ((130, 120, 100), 3, 1), ((160, 72, 80), 4, 4), ((128, 80, 96), 1, 3),
    ((240, 232, 224), 2, 2), ((234, 224, 226), 1, 2), ((16, 1024, 800), 2, 3)])
def test_multigrid_on_large_tiles_equals_the_oracle(pkg, abi, oracle_mod, dims, pre, post):
    p = abi.default_physics(*dims)
    p.mode, p.pressureTop = 1, 1
    d = (0.3 * np.random.default_rng(33).standard_normal(dims[::-1])).astype(np.float32)
    sim = pkg.FireSim(32, 16, *dims)
    sim.set_physics(p)
    sim.set_pressure_multigrid(2, pre, post)
    sim.set_pressure_tolerance(0.0, 1)
    sim.set("divergence", d)
    sim.set("pressure", np.zeros_like(d))
    sim.stages("pressure_sor", "pressure_sor", abi.FireSettings(), 0.0)
    a = sim.get("pressure")
    sim.close()
    o = oracle_mod.ConfigOracle(abi, 32, 16, *dims)
    o.set_physics(p)
    o.set_multigrid(2, pre, post, 0.0)
    o.set("divergence", d)
    o.set("pressure", np.zeros_like(d))
    o.stages("pressure_sor", "pressure_sor")
    b = o.get("pressure")
    assert np.abs(b).max() > 0.0
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_batch_of_large_scenes_equals_each_alone(pkg, abi):
    sizes = [(98, 90, 94), (64, 40, 48), (130, 72, 66), (31, 64, 33)]
    settings = [abi.FireSettings(width=48, height=32, reset=int(k == 0)) for k in range(3)]
    alone = []
    for k, dims in enumerate(sizes):
        sc, hdr = _scene(pkg, abi, dims, k)
        for s in settings:
            sc.step(s, render=False)
        alone.append({n: sc.get(n) for n in ("heat", "pressure", "v")})
        sc.close()
    pairs = [_scene(pkg, abi, dims, k) for k, dims in enumerate(sizes)]
    scenes = [p[0] for p in pairs]
    batch = pkg.Batch(scenes)
    for s in settings:
        batch.run([s] * len(scenes), render=[False] * len(scenes))
    batch.synchronize()
    for k, sc in enumerate(scenes):
        for n, want in alone[k].items():
            _bits_equal(f"scene {k} {n}", sc.get(n), want)
    batch.close()
    for sc in scenes:
        sc.close()
