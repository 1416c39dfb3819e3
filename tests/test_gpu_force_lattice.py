"""The allocation-free force pass around the grid size from which it builds the
curl noise's hash lattices (needs a GPU).  A table holds the hashes that the
smaller grids evaluate in place, so at any size and time the outputs are the
regular pass's bits."""
from __future__ import annotations

import numpy as np
import pytest

from test_zz_no_alloc import _call, _no_alloc_fn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims, time", [((36, 36, 37), 1.3), ((40, 37, 36), 1.3), ((41, 35, 45), 4.0e5), ((2, 120, 300), 77.0)])
def test_force_pass_with_and_without_lattices(pkg, abi, dims, time):
    import torch

    nx, ny, nz = dims
    rng = np.random.default_rng(12)
    sim = pkg.FireSim(16, 8, *dims)
    f = {n: rng.uniform(0.0, 2.0, (nz, ny, nx)).astype(np.float32) for n in abi.SCALAR_FIELDS}
    f.update(u=rng.uniform(-2, 2, (nz, ny, nx + 1)).astype(np.float32), v=rng.uniform(-1, 3, (nz, ny + 1, nx)).astype(np.float32),
             w=rng.uniform(-2, 2, (nz + 1, ny, nx)).astype(np.float32))
    for n, a in f.items():
        sim.set(n, a)
    settings = abi.validation_settings(5, width=16, height=8)
    rec = [torch.tensor(np.stack([f[n] for n in names], axis=-1), device="cuda") for names in
           (("heat", "fuel", "oxygen", "soot"), ("char", "ash", "pyrolysis", "progress"), ("turbulence_energy", "soot_optics"))]
    faces = [torch.tensor(f[n], device="cuda") for n in ("u", "v", "w")]
    outs = [torch.full_like(t, np.nan) for t in faces] + [torch.full((nz, ny, nx), np.nan, device="cuda") for _ in range(2)]
    _call(_no_alloc_fn(pkg), pkg, settings, time, dims, [*rec, *faces], outs, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    sim.stages("force", "divergence", settings, time)
    for n, got in zip(("u", "v", "w", "divergence", "pressure"), outs):
        assert np.array_equal(got.cpu().numpy().view(np.uint32), sim.get(n).view(np.uint32)), n
    sim.close()
