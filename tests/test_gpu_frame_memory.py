"""The raymarch's noise tables count as a scene's memory from its making on (needs a
GPU): neither a step nor a frame changes what a scene reports, a served scene is
counted with them before it is admitted, and a scene of the config physics, which
has none, never allocates them."""
from __future__ import annotations

import pytest

from test_gpu_serving import _request

pytestmark = pytest.mark.gpu

DIMS = (32, 28, 24)


def _frame(pkg, abi, scene, hdr, reset):
    scene.set_hdr_buffer(hdr.data_ptr(), 64 * 16, 0)
    s = abi.validation_settings(0, width=64, height=48)
    s.reset = reset
    scene.step(s, render=True)
    scene.synchronize()


def test_no_frame_changes_what_a_scene_holds(pkg, abi):
    import torch

    hdr = torch.zeros((48, 64, 4), device="cuda")
    scene = pkg.Scene(64, 48, *DIMS)
    made = scene.device_bytes()
    s = abi.validation_settings(0, width=64, height=48)
    scene.step(s, render=False)
    assert scene.device_bytes() == made
    free = torch.cuda.mem_get_info()[0]
    _frame(pkg, abi, scene, hdr, 0)
    # (A kernel's first launch loads its code, a few MB; the tables are 23 MB.)
    assert free - torch.cuda.mem_get_info()[0] < 20_000_000
    assert scene.device_bytes() == made
    scene.close()


def test_the_config_physics_has_no_tables(pkg, abi):
    scene = pkg.Scene(64, 48, *DIMS)
    made = scene.device_bytes()
    p = abi.default_physics(*DIMS)
    p.mode = 1
    scene.set_physics(p)
    assert made - scene.device_bytes() > 20_000_000
    scene.step(abi.FireSettings(width=64, height=48, reset=1), render=False)
    assert scene.device_bytes() < made
    p.mode = 0
    scene.set_physics(p)
    assert scene.device_bytes() > made
    scene.close()


def test_the_tables_do_not_end_a_capture_elsewhere(pkg, abi):
    import numpy as np
    import torch

    frames = []
    x = torch.zeros(8, device="cuda")
    for capture in (False, True):
        sim = pkg.FireSim(64, 48, *DIMS)
        s = abi.validation_settings(3, width=64, height=48)
        if capture:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, capture_error_mode="global"):
                x += 1.0
                sim.stages("light_build", "render", s, 0.5, wait=False)
            graph.replay()
            torch.cuda.synchronize()
        else:
            sim.stages("light_build", "render", s, 0.5)
        sim.synchronize()
        frames.append(sim.get("hdr"))
        sim.close()
    assert float(x[0]) == 1.0
    assert np.array_equal(frames[0].view(np.uint32), frames[1].view(np.uint32))


def test_server_counts_a_scene_as_it_is_after_a_frame(pkg, abi):
    import torch

    hdr = torch.zeros((48, 64, 4), device="cuda")
    scene = pkg.Scene(64, 48, *DIMS)
    _frame(pkg, abi, scene, hdr, 1)
    rendered = scene.device_bytes() + 64 * 48 * 16
    scene.close()
    server = pkg.Server(budget_bytes=int(2.5 * rendered))
    for i in range(4):
        server.submit(_request(abi, i, DIMS, steps=6, arrival=0.0, scene=0, render_every=2))
    rep = server.run(60.0)
    server.close()
    assert rep["completed"] == 4
    assert rep["admittedPeak"] <= 2
    assert rep["deviceBytesPeak"] == rep["admittedPeak"] * rendered
