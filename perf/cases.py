"""The work that a user of firesim-b200 has it do, as measurable cases.

A case is one pass of a program that simulates and renders a fire:

  app    the singleton scene behind the reference's own entry points: a clip
         of frames from a reset, each stepped, rendered and copied to the host
         as BGRA8, the last one with its frame metrics;
  scene  one FireScene handle: a clip of steps with a frame into a device HDR
         buffer after every `every`-th step (and, with `fields`, a checkpoint
         of the state at its end); with `live`, the next steps of a running
         scene instead of a clip from a reset;
  batch  a FireBatch of scenes of mixed sizes, stepped and rendered together;
  force  the allocation-free force pass on buffers that the caller owns.

`physics` is "ref" (the reference's ten-scalar fire) or "cfg" (the T/F/S model
with disk emitters), `solver` the pressure solve: "sor" (a fixed count, or
until `tol`) or "mg" (multigrid, p = 0 on the top face), `precision` the
storage of the library that is loaded.  exact() restates the config physics
in 64 bits; the reference physics hashes sines of large arguments, so its
values have no meaning apart from the float arithmetic that produces them.
"""
import ctypes
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
CONTRACTS = ROOT / "tests" / "golden" / "scene_contracts"
STORAGE = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
# Frame metrics that are functions of the fields (the others are timings and counters).
METRICS = ("heatSum", "fuelSum", "oxygenSum", "sootSum", "charSum", "ashSum", "pyrolysisSum", "progressSum", "turbulenceEnergySum",
           "sootOpticalDepthSum", "maxHeat", "maxFuel", "maxSoot", "flameHeightMeters", "meanSceneLight", "meanSceneShadow",
           "divergenceBeforeL2", "divergenceAfterL2")
CHECKPOINT = ("heat", "fuel", "soot", "pressure", "u", "v", "w")


def package():
    if "firesim_b200" not in sys.modules:
        where = ROOT / "native-firesim_b200"
        spec = importlib.util.spec_from_file_location("firesim_b200", where / "__init__.py", submodule_search_locations=[str(where)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["firesim_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["firesim_b200"]


def case(kind, grid, frame, **more):
    c = {"kind": kind, "physics": "ref", "solver": "sor", "nx": grid[0], "ny": grid[1], "nz": grid[2], "fw": frame[0], "fh": frame[1],
         "sceneId": 0, "iterations": 40, "omega": 1.52, "tol": 0.0, "precision": "f32", "steps": 1, "every": 1, "live": False,
         "fields": False, "scenes": 1, "hdr16": False}
    c.update(more)
    return c


def listed():
    return [
        # The reference's API at its smallest window request: twelve frames of the validation harness, host BGRA each.
        case("app", (72, 80, 48), (320, 180), name="app-72x80x48", steps=12),
        # A small interactive scene, one step and one frame per call: latency and launches.
        case("scene", (48, 48, 48), (128, 128), name="live-48", live=True),
        # The reference's default: its 176x208x128 grid and 40 iterations, 1280x720, a frame per step (a campfire).
        case("scene", (176, 208, 128), (1280, 720), name="frames-176x208x128", sceneId=1, steps=36),
        # 128^3 with 60 iterations and a 512^2 frame every ten steps: the benchmark's workload.
        case("scene", (128, 128, 128), (512, 512), name="run-128", iterations=60, omega=1.8, steps=60, every=10),
        # An odd grid and a wide frame, half storage and an RGBA16F target (the gas burner).
        case("scene", (125, 99, 77), (640, 360), name="run-125x99x77-f16", sceneId=2, precision="f16", steps=24, every=2, hdr16=True),
        # A large grid, simulated for its fields more than its frames.
        case("scene", (256, 256, 256), (512, 512), name="run-256", steps=24, every=12),
        # The config physics at 64^3 with a checkpoint at the end.
        case("scene", (64, 64, 64), (256, 256), name="cfg-64", physics="cfg", omega=1.7, steps=40, every=40, fields=True),
        # 128^3 to |div u| <= 1e-4: wind, curl noise, multigrid, a frame every ten steps.
        case("scene", (128, 128, 128), (512, 512), name="cfg-128-mg", physics="cfg", solver="mg", tol=5e-5, steps=60, every=10),
        # 256^3 in bfloat16, SOR until the residual is small or 120 iterations.
        case("scene", (256, 256, 256), (512, 512), name="cfg-256-bf16", physics="cfg", iterations=120, omega=1.85, tol=1e-5,
             precision="bf16", steps=12, every=12),
        # The same grid with the multigrid solve, in half storage.
        case("scene", (256, 256, 256), (512, 512), name="cfg-256-mg-f16", physics="cfg", solver="mg", tol=5e-5, precision="f16",
             steps=32, every=16),
        # Twenty-four small scenes of mixed sizes stepped as one batch, 256^2 frames every ten steps.
        case("batch", (96, 96, 96), (256, 256), name="batch-24-f16", physics="cfg", solver="mg", tol=5e-5, precision="f16", steps=20,
             every=10, scenes=24),
        # The force pass of an engine that owns its memory.
        case("force", (120, 88, 96), (64, 64), name="force-120x88x96"),
    ]


def draw(rng):
    def size(lo, hi, step=1):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return max(lo, n // step * step)

    def grid(lo, hi, most, step=1):
        while True:
            g = tuple(size(lo, hi, step) for _ in range(3))
            if g[0] * g[1] * g[2] <= most:
                return g

    frame = (size(96, 1280), size(96, 720))
    precision = rng.choice(("f32", "f32", "f16", "bf16"))
    kind = rng.choice(("ref", "ref", "ref", "cfg", "cfg", "mg", "mg", "batch", "force", "app"))
    steps = rng.choice((4, 6, 8, 12))
    if kind == "ref":
        return case("scene", grid(24, 256, 10_000_000), frame, sceneId=rng.randrange(3), iterations=rng.choice((20, 40, 60)), steps=steps,
                    every=rng.choice((1, 2, steps)), precision=precision, hdr16=rng.random() < 0.3)
    if kind == "cfg":
        return case("scene", grid(24, 256, 10_000_000), frame, physics="cfg", iterations=rng.choice((40, 60)),
                    omega=rng.choice((1.7, 1.8)), steps=steps, every=steps, precision=precision)
    if kind == "mg":
        return case("scene", grid(32, 256, 12_000_000, 8), frame, physics="cfg", solver="mg", tol=5e-5, steps=steps, every=steps,
                    precision=precision)
    if kind == "batch":
        return case("batch", grid(32, 112, 900_000, 8), (size(64, 256), size(64, 256)), physics="cfg", solver="mg", tol=5e-5, steps=steps,
                    every=steps, precision=precision, scenes=rng.randint(3, 32))
    if kind == "force":
        return case("force", grid(16, 160, 1_000_000), (64, 64), precision=precision, sceneId=rng.randrange(3))
    return case("app", (rng.randint(72, 104), rng.randint(80, 112), rng.randint(48, 72)), (size(160, 960), size(90, 540)),
                sceneId=rng.randrange(3), steps=steps)


def batch_grids(c):
    """The scenes' grids: the case's own size and smaller and longer ones beside it."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    half = [max(16, n // 16 * 8) for n in (nx, ny, nz)]
    shapes = [(nx, ny, nz), (half[0], half[1], half[2]), (nx, half[1], half[2]), (nx, ny, half[2])]
    return [shapes[(5 * i + i // 4) % 4] for i in range(c["scenes"])]


def ref_settings(pkg, c, rng):
    """One FireSettings per step: the validation harness from a frame of its own on, seen from another side, with
    the scene's emitter contract."""
    first, gust, turn = rng.randrange(1000), 0.2 * rng.random(), rng.uniform(-0.3, 0.3)
    out = []
    for f in range(c["steps"]):
        s = pkg.abi.validation_settings(first + f, scene=c["sceneId"], width=c["fw"], height=c["fh"], fire_scenes_dir=CONTRACTS)
        s.reset = 1 if f == 0 and not c["live"] else 0
        s.wind += gust
        s.cameraYaw += turn
        out.append(s)
    return out


def cfg_physics(pkg, c, grid, rng, lib):
    nx, ny, nz = grid
    r = min(0.1 * min(nx, nz) + 2.0, 16.0)
    p = pkg.abi.config_scene(nx, ny, nz, nx * rng.uniform(0.4, 0.6), nz * rng.uniform(0.4, 0.6), r, rng.uniform(-0.5, 0.5),
                             rng.uniform(-0.5, 0.5), rng.randrange(1 << 20), lib)
    if c["kind"] == "scene":
        p.noiseSeed, p.noiseAmplitude, p.noisePeriod = rng.randrange(1 << 20), 0.4, 16.0
        p.primarySamples, p.lightSamples = 128, 48
    p.pressureTop = 1 if c["solver"] == "mg" else 0
    return p


def cfg_setup(scene, c, physics):
    scene.set_physics(physics)
    if c["solver"] == "mg":
        scene.set_pressure_multigrid(20, 2, 2)
        scene.set_pressure_tolerance(c["tol"], 1)
    elif c["tol"] > 0.0:
        scene.set_pressure_tolerance(c["tol"], 10)


def hdr_target(scene, c):
    hdr = torch.zeros((c["fh"], c["fw"] + c["fw"] % 2, 4), dtype=torch.float16 if c["hdr16"] else torch.float32, device="cuda")
    scene.set_hdr_buffer(hdr.data_ptr(), hdr.shape[1] * 4 * hdr.element_size(), 1 if c["hdr16"] else 0)
    return hdr


def prepare(c, seed):
    import random
    rng = random.Random(seed)
    pkg = package()
    grid = (c["nx"], c["ny"], c["nz"])
    lib = pkg.load_library(c["precision"])
    st = {"c": c, "pkg": pkg}
    if c["kind"] == "app":
        st["sim"] = pkg.FireSim(c["fw"], c["fh"], *grid, precision=c["precision"])
        st["sim"].set_pressure_solver(c["iterations"], c["omega"])
        st["settings"] = ref_settings(pkg, c, rng)
        return st
    if c["kind"] == "force":
        g = torch.Generator(device="cuda").manual_seed(seed)
        nx, ny, nz = grid
        dt = STORAGE[c["precision"]]

        def smooth(shape, lo, hi):
            coarse = torch.rand((1, 1, *[max(2, n // 8) for n in shape]), generator=g, device="cuda")
            x = torch.nn.functional.interpolate(coarse, size=shape, mode="trilinear", align_corners=True)[0, 0]
            return (lo + (hi - lo) * x * x).contiguous()

        cells = (nz, ny, nx)
        top = (("heat", 8.0), ("fuel", 4.0), ("oxygen", 1.0), ("soot", 5.0), ("char", 2.0), ("ash", 1.0), ("pyrolysis", 2.0),
               ("progress", 3.0), ("turbulence", 3.0), ("optics", 8.0))
        f = {n: smooth(cells, 0.0, m) for n, m in top}
        faces = [smooth((nz, ny, nx + 1), -2.0, 2.0), smooth((nz, ny + 1, nx), -0.9, 4.0), smooth((nz + 1, ny, nx), -2.0, 2.0)]
        st["in"] = [torch.stack([f[n] for n in names], -1).to(dt).contiguous() for names in
                    (("heat", "fuel", "oxygen", "soot"), ("char", "ash", "pyrolysis", "progress"), ("turbulence", "optics"))]
        st["in"] += [x.to(dt).contiguous() for x in faces]
        st["out"] = [torch.empty_like(x) for x in st["in"][3:]] + [torch.empty(cells, device="cuda") for _ in range(2)]
        fn = lib.fireCudaForceProjectNoAlloc
        fn.restype = ctypes.c_bool
        fn.argtypes = [ctypes.POINTER(pkg.abi.FireSettings), ctypes.c_float] + [ctypes.c_int] * 3 + [ctypes.c_void_p] * 12
        st["fn"], st["time"] = fn, rng.uniform(0.5, 20.0)
        st["settings"] = pkg.abi.validation_settings(rng.randrange(1, 1000), scene=c["sceneId"], fire_scenes_dir=CONTRACTS)
        return st
    if c["kind"] == "batch":
        st["scenes"], st["hdr"] = [], []
        for g in batch_grids(c):
            s = pkg.Scene(c["fw"], c["fh"], *g, precision=c["precision"])
            cfg_setup(s, c, cfg_physics(pkg, c, g, rng, lib))
            st["hdr"].append(hdr_target(s, c))
            st["scenes"].append(s)
        st["batch"] = pkg.Batch(st["scenes"])
        n = len(st["scenes"])
        st["settings"] = [[pkg.abi.FireSettings(width=c["fw"], height=c["fh"], reset=1 if k == 0 else 0) for _ in range(n)]
                          for k in range(c["steps"])]
        return st
    s = pkg.Scene(c["fw"], c["fh"], *grid, precision=c["precision"])
    s.set_pressure_solver(c["iterations"], c["omega"])
    st["scene"], st["hdr"] = s, hdr_target(s, c)
    if c["physics"] == "cfg":
        cfg_setup(s, c, cfg_physics(pkg, c, grid, rng, lib))
        st["settings"] = [pkg.abi.FireSettings(width=c["fw"], height=c["fh"], reset=1 if k == 0 else 0) for k in range(c["steps"])]
    else:
        st["settings"] = ref_settings(pkg, c, rng)
    if c["live"]:  # a scene that has been running for a while
        for f in range(100):
            q = pkg.abi.validation_settings(f, scene=c["sceneId"], width=c["fw"], height=c["fh"], fire_scenes_dir=CONTRACTS)
            q.wind = st["settings"][0].wind
            s.step(q, render=False)
        s.synchronize()
    return st


def renders(c, k):
    return (k + 1) % c["every"] == 0


def run(st):
    c = st["c"]
    if c["kind"] == "app":
        last = len(st["settings"]) - 1
        for k, s in enumerate(st["settings"]):
            bgra, m = st["sim"].step_and_render(s, metrics=k == last)
        return {"bgra": bgra, "metrics": np.array([getattr(m, n) for n in METRICS], dtype=np.float32)}
    if c["kind"] == "force":
        stream = torch.cuda.current_stream().cuda_stream
        if not st["fn"](ctypes.byref(st["settings"]), st["time"], c["nx"], c["ny"], c["nz"], *[t.data_ptr() for t in st["in"] + st["out"]],
                        stream):
            raise RuntimeError(st["pkg"].firesim.last_error(st["pkg"].load_library(c["precision"])))
        return {"u": st["out"][0], "v": st["out"][1], "w": st["out"][2], "divergence": st["out"][3], "pressure": st["out"][4]}
    if c["kind"] == "batch":
        n = len(st["scenes"])
        for k, s in enumerate(st["settings"]):
            st["batch"].run(s, render=[renders(c, k)] * n)
        return st["hdr"]
    for k, s in enumerate(st["settings"]):
        st["scene"].step(s, render=renders(c, k))
    out = {"hdr": st["hdr"]}
    if c["fields"]:
        out.update({n: st["scene"].get(n) for n in CHECKPOINT})
    return out


def work(c):
    """Per step the state is read and written once and every solver iteration's update is arithmetic that has to happen; a frame reads
    the state that it shows and writes its pixels.  Counts of operations are the models' own, by term."""
    grids = batch_grids(c) if c["kind"] == "batch" else [(c["nx"], c["ny"], c["nz"])]
    s = 4 if c["precision"] == "f32" else 2
    total = {"bytes": 0.0, "flops": 0.0}
    for g in grids:
        n = g[0] * g[1] * g[2]
        scalars = 10 if c["physics"] == "ref" else 4
        if c["kind"] == "force":
            total["bytes"] += n * (scalars * s + 6 * s + 8)
            total["flops"] += n * 400.0
            continue
        step_bytes = n * (2 * (scalars + 3) * s + 8)
        step_flops = n * (1500.0 if c["physics"] == "ref" else 500.0)
        if c["solver"] == "mg":
            step_flops += n * 3 * 60.0  # three V(2,2) cycles: 8/7 of (four sweeps, residual, interpolation)
        else:
            step_flops += n * 10.0 * c["iterations"]
        frames = sum(1 for k in range(c["steps"]) if renders(c, k))
        total["bytes"] += c["steps"] * step_bytes + frames * (n * scalars * s + c["fw"] * c["fh"] * (8 if c["hdr16"] else 16))
        total["flops"] += c["steps"] * step_flops + frames * c["fw"] * c["fh"] * 2.0e4
    return total


# ---- the config physics in 64 bits ---------------------------------------

def _i64(v):
    return v - (1 << 64) if v >= 1 << 63 else v


def _splitmix(z):
    z = z + _i64(0x9E3779B97F4A7C15)
    z = (z ^ ((z >> 30) & ((1 << 34) - 1))) * _i64(0xBF58476D1CE4E5B9)
    z = (z ^ ((z >> 27) & ((1 << 37) - 1))) * _i64(0x94D049BB133111EB)
    return z ^ ((z >> 31) & ((1 << 33) - 1))


def _top24(z):
    return (_splitmix(z) >> 40) & ((1 << 24) - 1)


def _sample(f, qx, qy, qz):
    """Trilinear at index-space positions, clamped to the grid (f is [z, y, x] or [z, y, x, channel])."""
    out, at = None, []
    for q, m in ((qz, f.shape[0]), (qy, f.shape[1]), (qx, f.shape[2])):
        q = q.clamp(0.0, m - 1.0)
        i = q.long()
        t = q - i
        at.append(((i, 1.0 - t), ((i + 1).clamp(max=m - 1), t)))
    for z, wz in at[0]:
        for y, wy in at[1]:
            for x, wx in at[2]:
                w = wz * wy * wx
                v = f[z, y, x] * (w[..., None] if f.dim() == 4 else w)
                out = v if out is None else out + v
    return out


class Exact:
    """One scene of the config physics, stepped in float64."""

    def __init__(self, c, grid, p):
        self.c, self.p, (self.nx, self.ny, self.nz) = c, p, grid
        nx, ny, nz = grid
        self.dev = torch.device("cuda")
        z = lambda *s: torch.zeros(s, dtype=torch.float64, device=self.dev)  # noqa: E731
        self.T, self.F, self.S = z(nz, ny, nx), z(nz, ny, nx), z(nz, ny, nx)
        self.u, self.v, self.w, self.pr = z(nz, ny, nx + 1), z(nz, ny + 1, nx), z(nz + 1, ny, nx), z(nz, ny, nx)
        self.step_index = 0
        self.noise = self.noise_field() if p.noiseAmplitude != 0.0 else None
        if c["solver"] == "mg":
            self.eigen = [self.laplacian(n, axis == 1) for axis, n in enumerate((nz, ny, nx))]
        x, y, zz = self.index(nx), self.index(ny), self.index(nz)
        parity = (x[None, None] + y[None, :, None] + zz[:, None, None]).long() % 2
        self.colour = [(parity == k) for k in range(2)]

    def index(self, n, offset=0.0):
        return torch.arange(n, dtype=torch.float64, device=self.dev) + offset

    def mesh(self, n, o):
        x, y, z = (self.index(n[k], o[k]) for k in range(3))
        return x[None, None, :], y[None, :, None], z[:, None, None]

    def laplacian(self, n, dirichlet_end):
        a = torch.zeros((n, n), dtype=torch.float64, device=self.dev)
        i = torch.arange(n - 1, device=self.dev)
        a[i, i + 1] = a[i + 1, i] = -1.0
        d = torch.full((n,), 2.0, dtype=torch.float64, device=self.dev)
        d[0], d[-1] = 1.0, 3.0 if dirichlet_end else 1.0
        return torch.linalg.eigh(a + torch.diag(d))

    def noise_field(self):
        p = self.p
        inv = float(np.float32(1.0) / np.float32(p.noisePeriod))
        x, y, z = self.mesh((self.nx, self.ny, self.nz), (0.5, 0.5, 0.5))
        f, cell, s, ds = [], [], [], []
        for q in (x * inv, y * inv, z * inv):
            q = q.expand(self.nz, self.ny, self.nx)
            cell.append(q.floor().long())
            f.append(q - q.floor())
            s.append(f[-1] * f[-1] * (3 - 2 * f[-1]))
            ds.append(6 * f[-1] * (1 - f[-1]))
        mult = (_i64(0x9E3779B97F4A7C15), _i64(0xC2B2AE3D27D4EB4F), 0x165667B19E3779F9)

        def gradient(comp):
            seed = _i64((((p.noiseSeed << 2) | comp) * 0xD1342543DE82EF95) & ((1 << 64) - 1))
            v = {(a, b, e): _top24(seed + (cell[0] + a) * mult[0] + (cell[1] + b) * mult[1] + (cell[2] + e) * mult[2]).double() / 8388608.0 - 1.0
                 for a in (0, 1) for b in (0, 1) for e in (0, 1)}
            mix = lambda a, b, t: a + (b - a) * t  # noqa: E731
            gx = ds[0] * mix(*[mix(v[1, 0, e] - v[0, 0, e], v[1, 1, e] - v[0, 1, e], s[1]) for e in (0, 1)], s[2])
            a = {(b, e): mix(v[0, b, e], v[1, b, e], s[0]) for b in (0, 1) for e in (0, 1)}
            gy = ds[1] * mix(a[1, 0] - a[0, 0], a[1, 1] - a[0, 1], s[2])
            gz = ds[2] * (mix(a[0, 1], a[1, 1], s[1]) - mix(a[0, 0], a[1, 0], s[1]))
            return gx * inv, gy * inv, gz * inv

        g0, g1, g2 = gradient(0), gradient(1), gradient(2)
        return [p.noiseAmplitude * d for d in (g2[1] - g1[2], g0[2] - g2[0], g1[0] - g0[1])]

    def velocity(self, x, y, z):
        return (_sample(self.u, x, y - 0.5, z - 0.5), _sample(self.v, x - 0.5, y, z - 0.5), _sample(self.w, x - 0.5, y - 0.5, z))

    def disk(self, e):
        x, _, z = self.mesh((self.nx, self.ny, self.nz), (0.0, 0.0, 0.0))
        inside = ((x - e.centerX) ** 2 + (z - e.centerZ) ** 2 <= e.radius * e.radius).expand(self.nz, self.ny, self.nx)
        row = torch.zeros(self.ny, dtype=torch.bool, device=self.dev)
        if 0 <= math.floor(e.centerY) < self.ny:
            row[math.floor(e.centerY)] = True
        return inside & row[None, :, None]

    def advance(self):
        p, nx, ny, nz = self.p, self.nx, self.ny, self.nz
        new = []
        for f, n, o in ((self.u, (nx + 1, ny, nz), (0.0, 0.5, 0.5)), (self.v, (nx, ny + 1, nz), (0.5, 0.0, 0.5)),
                        (self.w, (nx, ny, nz + 1), (0.5, 0.5, 0.0))):
            x, y, z = self.mesh(n, o)
            x, y, z = (q.expand(n[2], n[1], n[0]) for q in (x, y, z))
            a, b, d = self.velocity(x, y, z)
            new.append(_sample(f, x - a - o[0], y - b - o[1], z - d - o[2]))
        self.u, self.v, self.w = new
        x, y, z = (q.expand(nz, ny, nx) for q in self.mesh((nx, ny, nz), (0.5, 0.5, 0.5)))
        a, b, d = self.velocity(x, y, z)
        r = _sample(torch.stack((self.T, self.F, self.S), -1), x - a - 0.5, y - b - 0.5, z - d - 0.5)
        heat, fuel, soot = r.unbind(-1)
        burn = torch.where(heat > p.ignitionHeat, fuel * min(1.0, p.burnRate * p.dt), torch.zeros_like(fuel))
        fuel, heat, soot = fuel - burn, heat + p.heatRelease * burn, soot + p.sootYield * burn
        heat = heat - heat * min(1.0, p.cooling * p.dt)
        soot = soot - soot * min(1.0, p.sootDecay * p.dt)
        cell = torch.arange(nx * ny * nz, device=self.dev).reshape(nz, ny, nx)
        for e in range(p.emitterCount):
            em = p.emitters[e]
            key = _i64(((em.seed << 32) ^ (self.step_index * 0xD1B54A32D192ED03)) & ((1 << 64) - 1))
            j = 1.0 - em.jitterScale * (_top24(cell ^ key).double() / 16777216.0)
            hit = self.disk(em)
            fuel = torch.where(hit, torch.maximum(fuel, em.fuel * j), fuel)
            heat = torch.where(hit, torch.maximum(heat, em.heat * j), heat)
        self.T, self.F, self.S = heat, fuel, soot
        self.step_index += 1
        self.forces()
        self.project()

    def diff(self, f, dim):
        """Central difference (half the span) with clamped neighbours."""
        n = f.shape[dim]
        i = torch.arange(n, device=self.dev)
        return 0.5 * (f.index_select(dim, (i + 1).clamp(max=n - 1)) - f.index_select(dim, (i - 1).clamp(min=0)))

    def forces(self):
        p = self.p
        fx = fy = fz = torch.zeros_like(self.T)
        if p.vorticityEps != 0.0:
            cu, cv, cw = 0.5 * (self.u[..., 1:] + self.u[..., :-1]), 0.5 * (self.v[:, 1:] + self.v[:, :-1]), 0.5 * (self.w[1:] + self.w[:-1])
            o = (self.diff(cw, 1) - self.diff(cv, 0), self.diff(cu, 0) - self.diff(cw, 2), self.diff(cv, 2) - self.diff(cu, 1))
            mag = torch.sqrt(o[0] ** 2 + o[1] ** 2 + o[2] ** 2)
            e = (self.diff(mag, 2), self.diff(mag, 1), self.diff(mag, 0))
            length = torch.sqrt(e[0] ** 2 + e[1] ** 2 + e[2] ** 2)
            n = [torch.where(length > 1e-20, q / length.clamp(min=1e-20), torch.zeros_like(q)) for q in e]
            fx, fy, fz = (p.vorticityEps * q for q in (n[1] * o[2] - n[2] * o[1], n[2] * o[0] - n[0] * o[2], n[0] * o[1] - n[1] * o[0]))
        if self.noise is not None:
            fx, fy, fz = fx + self.noise[0], fy + self.noise[1], fz + self.noise[2]
        fy = fy + p.buoyancyHeat * (self.T - p.ambientHeat) - p.buoyancySoot * self.S
        u, v, w = self.u.clone(), self.v.clone(), self.w.clone()
        u[..., 1:-1] += p.dt * 0.5 * (fx[..., 1:] + fx[..., :-1]) + p.dt * p.windX
        v[:, 1:-1] += p.dt * 0.5 * (fy[:, 1:] + fy[:, :-1])
        v[:, -1] += p.dt * fy[:, -1]
        w[1:-1] += p.dt * 0.5 * (fz[1:] + fz[:-1]) + p.dt * p.windZ
        for k in range(p.emitterCount):
            hit = self.disk(p.emitters[k])
            face = torch.zeros_like(v, dtype=torch.bool)
            face[:, :-1] |= hit
            face[:, 1:] |= hit
            v[face] = p.emitters[k].upVelocity
        u[..., 0], u[..., -1], v[:, 0], w[0], w[-1] = 0.0, 0.0, 0.0, 0.0, 0.0
        self.u, self.v, self.w = u, v, w

    def project(self):
        u, v, w = self.u, self.v, self.w
        rhs = -((u[..., 1:] - u[..., :-1]) + (v[:, 1:] - v[:, :-1]) + (w[1:] - w[:-1]))
        if self.c["solver"] == "mg":
            (lz, ez), (ly, ey), (lx, ex) = self.eigen
            q = torch.einsum("zyx,za,yb,xc->abc", rhs, ez, ey, ex) / (lz[:, None, None] + ly[None, :, None] + lx[None, None, :])
            pr = torch.einsum("abc,za,yb,xc->zyx", q, ez, ey, ex)
        else:
            pr = torch.zeros_like(rhs)
            for k in range(2 * self.c["iterations"]):
                q = torch.nn.functional.pad(pr[None, None], (1,) * 6, mode="replicate")[0, 0]
                s = rhs + q[1:-1, 1:-1, :-2] + q[1:-1, 1:-1, 2:] + q[1:-1, :-2, 1:-1] + q[1:-1, 2:, 1:-1] + q[:-2, 1:-1, 1:-1] + q[2:, 1:-1, 1:-1]
                pr = torch.where(self.colour[k % 2], pr + self.c["omega"] * (s / 6.0 - pr), pr)
        u[..., 1:-1] -= pr[..., 1:] - pr[..., :-1]
        v[:, 1:-1] -= pr[:, 1:] - pr[:, :-1]
        w[1:-1] -= pr[1:] - pr[:-1]
        if self.c["solver"] == "mg":
            v[:, -1] += 2.0 * pr[:, -1]
        u[..., 0], u[..., -1], v[:, 0], w[0], w[-1] = 0.0, 0.0, 0.0, 0.0, 0.0
        self.pr = pr

    def frame(self):
        c, p = self.c, self.p
        rec = torch.stack((self.T, self.F, self.S), -1)
        lx, ly, lz = (self.nx + 1) // 2, (self.ny + 1) // 2, (self.nz + 1) // 2
        pos = [2.0 * q.expand(lz, ly, lx) + 1.0 for q in self.mesh((lx, ly, lz), (0.0, 0.0, 0.0))]
        d = [l - q for l, q in zip((p.lightX, p.lightY, p.lightZ), pos)]
        dist = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
        r = [q / dist.clamp(min=1e-6) for q in d]
        seg = dist
        for q, o, n in zip(r, pos, (self.nx, self.ny, self.nz)):
            seg = torch.where(q > 0, torch.minimum(seg, (n - o) / q), torch.where(q < 0, torch.minimum(seg, -o / q), seg))
        ds = seg.clamp(min=0.0) / p.lightSamples
        tau = torch.zeros_like(dist)
        for k in range(p.lightSamples):
            s = _sample(rec, *[o + q * (k + 0.5) * ds - 0.5 for o, q in zip(pos, r)])
            tau = tau + (p.extinction * s[..., 2] + p.fuelExtinction * s[..., 1]) * ds
        light = torch.where(dist > 1e-6, torch.exp(-tau), torch.ones_like(tau))
        eye = np.array([p.eyeX, p.eyeY, p.eyeZ], dtype=np.float64)
        fwd = np.array([p.targetX, p.targetY, p.targetZ]) - eye
        fwd = fwd / np.linalg.norm(fwd)
        right = np.array([-fwd[2], 0.0, fwd[0]])
        right = right / np.linalg.norm(right) if np.linalg.norm(right) > 0 else np.array([1.0, 0.0, 0.0])
        up = np.cross(right, fwd)
        half = math.tan(p.fovYDegrees * 0.00872664626)
        px, py = self.index(c["fw"], 0.5)[None, :], self.index(c["fh"], 0.5)[:, None]
        sx, sy = (2.0 * px / c["fw"] - 1.0) * half * (c["fw"] / c["fh"]), (1.0 - 2.0 * py / c["fh"]) * half
        ray = [fwd[k] + right[k] * sx + up[k] * sy for k in range(3)]
        length = torch.sqrt(ray[0] ** 2 + ray[1] ** 2 + ray[2] ** 2)
        ray = [q / length for q in ray]
        t0, t1 = torch.zeros_like(length), torch.full_like(length, 3e38)
        for q, o, n in zip(ray, eye, (self.nx, self.ny, self.nz)):
            a, b = -o / q, (n - o) / q
            t0, t1 = torch.maximum(t0, torch.minimum(a, b)), torch.minimum(t1, torch.maximum(a, b))
        hit = t1 > t0
        ds = torch.where(hit, (t1 - t0) / p.primarySamples, torch.zeros_like(t0))
        rgb, view = [torch.zeros_like(t0) for _ in range(3)], torch.ones_like(t0)
        for k in range(p.primarySamples):
            q = [o + e * (t0 + (k + 0.5) * ds) for o, e in zip(eye, ray)]
            s = _sample(rec, *[x - 0.5 for x in q])
            alpha = 1.0 - torch.exp(-(p.extinction * s[..., 2] + p.fuelExtinction * s[..., 1]) * ds)
            scatter = p.albedo * p.lightIntensity * _sample(light, *[x * 0.5 - 0.5 for x in q]) * alpha
            heat = s[..., 0].clamp(min=0.0)
            h, e = heat / (heat + 1.0), p.emission * heat * ds
            rgb[0] = rgb[0] + view * (scatter + e)
            rgb[1] = rgb[1] + view * (scatter + e * (0.35 + 0.45 * h))
            rgb[2] = rgb[2] + view * (scatter + e * (0.08 + 0.50 * h * h))
            view = view * (1.0 - alpha)
        out = torch.zeros((c["fh"], c["fw"] + c["fw"] % 2, 4), dtype=torch.float64, device=self.dev)
        for k, b in enumerate((0.015, 0.016, 0.020)):
            out[:, :c["fw"], k] = rgb[k] + view * b
        out[:, :c["fw"], 3] = 1.0
        return out


def exact(c, seed):
    import random
    if c["physics"] != "cfg" or c["kind"] not in ("scene", "batch"):
        return None  # chaotic hashes of float sines
    if c["nx"] * c["ny"] * c["nz"] * c["steps"] * c["scenes"] * (1 if c["solver"] == "mg" else 0.2 * c["iterations"]) > 1.2e9:
        return None  # too long
    rng = random.Random(seed)
    pkg = package()
    lib = pkg.load_library(c["precision"])
    frames = []
    for g in batch_grids(c) if c["kind"] == "batch" else [(c["nx"], c["ny"], c["nz"])]:
        scene = Exact(c, g, cfg_physics(pkg, c, g, rng, lib))
        shown = None
        for k in range(c["steps"]):
            scene.advance()
            shown = scene.frame() if renders(c, k) else shown
        frames.append(shown)
    if c["kind"] == "batch":
        return frames
    out = {"hdr": frames[0]}
    if c["fields"]:
        out.update({"heat": scene.T, "fuel": scene.F, "soot": scene.S, "pressure": scene.pr, "u": scene.u, "v": scene.v, "w": scene.w})
    return out
