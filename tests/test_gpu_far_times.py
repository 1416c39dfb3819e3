"""Hash lattices and noise tables at times beyond an int's lattice coordinates
(needs a GPU).  No table can hold those, so the hashes are evaluated in place,
and the outputs are the same bits with tables allowed and not."""
from __future__ import annotations

import numpy as np
import pytest

from test_zz_no_alloc import _call, _no_alloc_fn

pytestmark = pytest.mark.gpu

TIMES = [1.5e8, 3.0e8, 1.0e9, -3.0e9, 1.0e20]


def _fields(abi, dims):
    nx, ny, nz = dims
    rng = np.random.default_rng(12)
    f = {n: rng.uniform(0.0, 2.0, (nz, ny, nx)).astype(np.float32) for n in abi.SCALAR_FIELDS}
    f.update(u=rng.uniform(-2, 2, (nz, ny, nx + 1)).astype(np.float32), v=rng.uniform(-1, 3, (nz, ny + 1, nx)).astype(np.float32),
             w=rng.uniform(-2, 2, (nz + 1, ny, nx)).astype(np.float32))
    return f


def _same(a, b, what):
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), what


@pytest.mark.parametrize("time", TIMES)
def test_step_and_frame_with_and_without_tables(pkg, abi, time):
    sim = pkg.FireSim(48, 32, 40, 36, 28)
    f = _fields(abi, (40, 36, 28))
    settings = abi.validation_settings(5, width=48, height=32)
    got = []
    for tables in (True, False):
        sim.set_hash_lattices(tables)
        for n, a in f.items():
            sim.set(n, a)
        out = {}
        sim.stages("light_build", "render", settings, time)
        out["hdr"] = sim.get("hdr")
        sim.stages("advect_react", "divergence", settings, time)
        out.update({n: sim.get(n) for n in ("heat", "fuel", "u", "v", "w")})
        got.append(out)
    sim.set_hash_lattices(True)
    sim.close()
    for n in got[0]:
        _same(got[0][n], got[1][n], n)


@pytest.mark.parametrize("time", [*TIMES, float("inf"), float("nan")])
def test_force_pass_with_lattices_equals_hashing_in_place(pkg, abi, time):
    import torch

    dims = nx, ny, nz = (41, 35, 45)  # large enough for lattices
    f = _fields(abi, dims)
    settings = abi.validation_settings(5, width=16, height=8)
    rec = [torch.tensor(np.stack([f[n] for n in names], axis=-1), device="cuda") for names in
           (("heat", "fuel", "oxygen", "soot"), ("char", "ash", "pyrolysis", "progress"), ("turbulence_energy", "soot_optics"))]
    faces = [torch.tensor(f[n], device="cuda") for n in ("u", "v", "w")]
    outs = [torch.zeros_like(t) for t in faces] + [torch.zeros((nz, ny, nx), device="cuda") for _ in range(2)]
    _call(_no_alloc_fn(pkg), pkg, settings, time, dims, [*rec, *faces], outs, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    sim = pkg.FireSim(16, 8, *dims)
    sim.set_hash_lattices(False)
    for n, a in f.items():
        sim.set(n, a)
    sim.stages("force", "divergence", settings, time)
    want = [sim.get(n) for n in ("u", "v", "w", "divergence", "pressure")]
    sim.set_hash_lattices(True)
    sim.close()
    for n, got, ref in zip(("u", "v", "w", "divergence", "pressure"), outs, want):
        _same(got.cpu().numpy(), ref, n)
