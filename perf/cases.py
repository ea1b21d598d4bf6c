"""The work that programs using this library have it do, as timed cases.

A case is one call pattern of a host program at one size:

  step     the particle state kept in host memory, one frame of `substeps`
           simulation steps through Fluid.step_host (positions and velocities
           in and out)
  batch    many independent scenes stepped together through Batch.step_host
  multi    a two-phase scene with diffusion: Fluid.step, then the point buffer
           (positions and phase fractions) that a renderer reads
  predict  the warm-start network's forward pass on caller-owned buffers
  train    Adam steps of that network (forward and backward), with the
           gradients of the last one
  sph      the particle-only solvers (PBF, PCISPH) and their read-back state
  mesh     the surface mesh of a fluid into a device buffer
  draw     one whole headless frame of a fluid (mesh, point buffer, image)

Scenes are the pool plus falling ball of the tests and the benchmark, taken a
few steps into the fall.  The seed sets a small random velocity of every
particle before those steps.
"""
from __future__ import annotations

import math
import pathlib
import struct

import numpy as np
import torch

import aquarius_b200 as aq
from aquarius_b200 import _abi, scenes

WEIGHTS = pathlib.Path(aq.__file__).resolve().parent / "weights"
LAYERS = ((16, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (32, 32), (48, 16), (16, 16))


def _fluid_case(kind, size, **kw):
    c = dict(kind=kind, sx=size[0], sy=size[1], sz=size[2], pool=0.2, radius=0.15, ball=0.65, dt=0.01,
             init="carry", solve="fixed", sweeps=100, substeps=1, settle=5)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest grid of the tests: a frame is bound by launches and latency
        dict(_fluid_case("step", (16, 16, 16)), name="step_16"),
        # the reference's default grid and solver settings (100 sweeps, carried pressure)
        dict(_fluid_case("step", (50, 50, 50)), name="step_50"),
        # a container of unequal, odd sides, three steps to the frame
        dict(_fluid_case("step", (90, 61, 75), pool=0.3, substeps=3), name="step_ragged"),
        # the benchmark's scene: 5.2 M particles, zero-init solve to 1e-4 capped at 2000 sweeps
        dict(_fluid_case("step", (128, 128, 128), pool=0.3, radius=0.12, ball=0.7, dt=0.005, init="zero",
                         solve="residual", sweeps=2000), name="step_128"),
        # scenes of uneven sizes stepped together (data generation, ensembles)
        dict(kind="batch", scenes=40, set=2024, sweeps=2000, substeps=1, settle=3, name="batch_40"),
        # two phases that diffuse into each other
        dict(_fluid_case("multi", (96, 96, 96), pool=0.35, radius=0.12, ball=0.6, dt=0.0025, init="zero",
                         solve="residual", sweeps=400, substeps=2, diffusion=100, settle=4), name="multi_96"),
        # the learned warm start's inference on a caller's pressure system
        dict(_fluid_case("predict", (128, 128, 128), pool=0.3, radius=0.12, ball=0.7, dt=0.005), name="predict_128"),
        # fine-tuning steps of that network
        dict(_fluid_case("train", (64, 64, 64), pool=0.25, dt=0.01, pairs=2, steps=2), name="train_64"),
        # the reference's default PBF scene (four substeps to the step)
        dict(kind="sph", method="pbf", particles=300000, substeps=1, settle=4, name="pbf_300k"),
        # PCISPH at ten times the default budget, five of its short steps to the frame
        dict(kind="sph", method="pcisph", particles=3000000, substeps=5, settle=20, name="pcisph_3m"),
        # surface extraction for an external renderer
        dict(_fluid_case("mesh", (64, 64, 64), pool=0.25), name="mesh_64"),
        # one frame of the benchmark's scene in the window of the reference's application
        dict(_fluid_case("draw", (128, 128, 128), pool=0.3, radius=0.12, ball=0.7, dt=0.005, width=1728, height=864),
             name="draw_128"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["step", "step", "step", "batch", "multi", "predict", "train", "sph", "mesh", "draw"])
    pool, radius = round(rng.uniform(0.12, 0.38), 3), round(rng.uniform(0.08, 0.18), 3)
    common = dict(pool=pool, radius=radius, ball=0.7)
    if kind == "step":
        if rng.random() < 0.3:  # the benchmark's settings on a grid of sides divisible by 4
            size = tuple(4 * _log(rng, 6, 32) for _ in range(3))
            return _fluid_case(kind, size, **common, dt=round(0.64 / max(size), 5), init="zero", solve="residual",
                               sweeps=40 * rng.randint(5, 50))
        size = tuple(_log(rng, 12, 110) for _ in range(3))
        return _fluid_case(kind, size, **common, dt=round(0.5 / max(size), 5), sweeps=rng.randint(40, 300),
                           substeps=rng.randint(1, 4))
    if kind == "batch":
        return dict(kind=kind, scenes=_log(rng, 4, 40), set=rng.randint(1, 100000), sweeps=40 * rng.randint(5, 50),
                    substeps=1, settle=3)
    if kind == "multi":
        size = tuple(_log(rng, 16, 96) for _ in range(3))
        return _fluid_case(kind, size, **common, dt=round(0.24 / max(size), 5), sweeps=rng.randint(40, 300),
                           substeps=rng.randint(1, 3), diffusion=rng.randint(20, 100), settle=4)
    if kind == "predict":
        return _fluid_case(kind, tuple(4 * _log(rng, 4, 32) for _ in range(3)), **common, dt=0.005)
    if kind == "train":
        return _fluid_case(kind, tuple(4 * _log(rng, 4, 16) for _ in range(3)), **common, pairs=2,
                           steps=rng.randint(1, 3))
    if kind == "sph":
        if rng.random() < 0.5:
            return dict(kind=kind, method="pbf", particles=_log(rng, 8000, 600000), substeps=1, settle=4)
        return dict(kind=kind, method="pcisph", particles=_log(rng, 8000, 3000000), substeps=rng.randint(1, 5),
                    settle=20)
    size = tuple(_log(rng, 16, 120) for _ in range(3))
    if kind == "mesh":
        return _fluid_case(kind, size, **common)
    return _fluid_case(kind, size, **common, width=_log(rng, 320, 1728), height=_log(rng, 240, 864))


def _config(case):
    kind = case["kind"]
    vols = [dict(shape="box", min=(0, 0, 0), max=(1, case["pool"], 1), phase=0),
            dict(shape="sphere", center=(0.5, case["ball"], 0.5), radius=case["radius"],
                 phase=1 if kind == "multi" else 0)]
    kw = {}
    if kind == "multi":
        kw = dict(diffusion_iterations=case["diffusion"], diffusion_coeff=1e-4, phase_count=2)
    residual = case["solve"] == "residual"
    return _abi.make_config(
        (case["sx"], case["sy"], case["sz"]), vols, timestep=case["dt"], flip_coeff=0.95, particle_jitter=0.05,
        pressure_init=_abi.PRESSURE_ZERO if case["init"] == "zero" else _abi.PRESSURE_CARRY,
        solve_mode=_abi.SOLVE_RESIDUAL if residual else _abi.SOLVE_FIXED, pressure_iterations=case["sweeps"],
        rel_residual=1e-4, max_iterations=case["sweeps"], check_interval=40, **kw)


def _pinned(n):
    return torch.zeros((3, n), dtype=torch.float32, pin_memory=True).numpy()


def _velocity(n, seed):
    g = torch.Generator().manual_seed(seed)
    return (0.3 * torch.randn((3, n), generator=g)).numpy()


def prepare(case, seed):
    kind = case["kind"]
    st = dict(kind=kind, case=case)
    if kind == "batch":
        cfgs = scenes.batch_configs(case["scenes"], case["set"], max_iterations=case["sweeps"])
        b = st["batch"] = aq.Batch(cfgs)
        n = sum(b.particle_counts)
        st["in"], st["out"] = (_pinned(n), _pinned(n)), (_pinned(n), _pinned(n))
        b.step_host(case["settle"], None, _velocity(n, seed), *st["in"])
        return st
    if kind == "sph":
        cfg = _abi.sph_config(_abi.SPH_PBF if case["method"] == "pbf" else _abi.SPH_PCISPH,
                              max_particle_count=case["particles"])
        st["sph"] = aq.Sph(cfg)
        st["sph"].set_state({"velocity": _velocity(st["sph"].n, seed)})
        st["sph"].step(case["settle"])
        st["sph"].synchronize()
        return st
    f = aq.Fluid(_config(case))
    n = f.particleCount
    f.upload_state({"velocity_p": _velocity(n, seed)})
    if kind == "step":
        st["fluid"] = f
        st["in"], st["out"] = (_pinned(n), _pinned(n)), (_pinned(n), _pinned(n))
        f.step_host(case["settle"], None, None, *st["in"])
    elif kind == "multi":
        st["fluid"] = f
        f.step(case["settle"])
        f.synchronize()
        st["vbo"] = torch.zeros((n, 7), dtype=torch.float32, device="cuda")
    elif kind == "predict":
        st["size"] = f.size
        st["net"] = aq.UNet(0, weights=_weights_file(case))
        f.step(case["settle"])
        st["rhs"], st["type"] = _system(f)
        st["out"] = torch.zeros_like(st["rhs"])
    elif kind == "train":
        st["net"] = aq.UNet(0, weights=_weights_file(case))
        st["data"] = aq.Dataset(f.size, case["pairs"])
        for _ in range(case["pairs"]):
            f.step(case["settle"])
            st["data"].add_fluid(f)
        st["rms"] = st["data"].target_rms()
    elif kind == "mesh":
        st["fluid"] = f
        f.step(case["settle"])
        f.synchronize()
        st["records"] = torch.zeros((1 << 17, 15, 6), dtype=torch.float32, device="cuda")
    elif kind == "draw":
        st["fluid"] = f
        f.step(case["settle"])
        f.synchronize()
        st["renderer"] = aq.Renderer(0)
        st["renderer"].set_skybox(np.random.default_rng(seed).integers(0, 256, (6, 256, 256, 3), dtype=np.uint8))
        st["command"] = aq.draw_command_default(case["width"], case["height"], f.getContainerSize(), case["sy"])
        st["image"] = torch.zeros((case["height"], case["width"], 4), dtype=torch.uint8, device="cuda")
    else:
        raise ValueError(kind)
    return st


def _weights_file(case):
    return WEIGHTS / ("unet_128.bin" if max(case["sx"], case["sy"], case["sz"]) > 64 else "unet_64.bin")


def _system(f):
    """The fluid's current pressure system, as a program with its own solver would hold it."""
    s = f.download_state(["divergence", "density", "content"])
    sx, sy, sz = f.size
    fluid = s["content"].reshape(sx + 1, sy + 1, sz + 1)[:sx, :sy, :sz].reshape(-1) == 1
    rhs = np.where(fluid, -s["divergence"] * s["density"], np.float32(0)).astype(np.float32)
    return torch.from_numpy(rhs).cuda(), torch.from_numpy(fluid.astype(np.int8)).cuda()


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "step":
        state["fluid"].step_host(case["substeps"], *state["in"], *state["out"])
        return {"position": state["out"][0], "velocity": state["out"][1]}
    if kind == "batch":
        state["batch"].step_host(case["substeps"], *state["in"], *state["out"])
        return {"position": state["out"][0], "velocity": state["out"][1]}
    if kind == "multi":
        state["fluid"].step(case["substeps"])
        state["fluid"].points_vbo_into(state["vbo"].data_ptr())
        return {"points": state["vbo"]}
    if kind == "predict":
        state["net"].predict(state["size"], state["rhs"].data_ptr(), state["type"].data_ptr(), state["out"].data_ptr())
        return {"pressure": state["out"]}
    if kind == "train":
        state["net"].train(state["data"], 0, case["pairs"], case["steps"], lr=1e-4, seed=1, out_scale=state["rms"],
                           residual_weight=1.0, residual_sweeps=20)
        return {"gradients": state["net"].gradients()}
    if kind == "sph":
        state["sph"].step(case["substeps"])
        s = state["sph"].get_state(["position", "velocity"])
        return {"position": s["position"], "velocity": s["velocity"]}
    if kind == "mesh":
        cubes = state["fluid"].mesh_into(state["records"].data_ptr(), state["records"].shape[0])
        return {"cubes": cubes, "records": state["records"]}
    state["fluid"].draw(state["command"], state["renderer"], state["image"].data_ptr())
    return {"image": state["image"]}


def _cells(case):
    """Cells, and cells that hold fluid at the start."""
    c = case["sx"] * case["sy"] * case["sz"]
    ball = 4 / 3 * math.pi * (case["radius"] * case["sy"]) ** 3
    return c, min(c, c * case["pool"] + ball)


def _step_work(c, fluid, sweeps, exchanged):
    """One simulation step: 13 B of a cell's system in and out and 8 operations per
    cell and sweep; a particle's 48 B in and out, about 400 operations each."""
    n = 8 * fluid
    return n * (48 + exchanged) + 60 * c, fluid * 8 * sweeps + 400 * n


def work(case):
    kind = case["kind"]
    if kind == "batch":
        b = f = 0
        for cfg in scenes.batch_configs(case["scenes"], case["set"]):
            c = cfg.size_x * cfg.size_y * cfg.size_z
            db, df = _step_work(c, c * cfg.volumes[0].box_max[1], case["sweeps"], 48)
            b, f = b + db, f + df
        return {"bytes": b, "flops": f}
    if kind == "sph":
        n = 0.19 * case["particles"]
        per = (4 * 2 * 2 if case["method"] == "pbf" else 4 * 2) * case["substeps"]
        return {"bytes": n * 96 * case["substeps"], "flops": n * per * 34 * 20}
    c, fluid = _cells(case)
    if kind in ("step", "multi"):
        b, f = _step_work(c, fluid, case["sweeps"], 48 / case["substeps"])
        if kind == "multi":
            b, f = b + 32 * fluid * 8 + 32 * c, f + case["diffusion"] * fluid * 4 * 8
        return {"bytes": b * case["substeps"], "flops": f * case["substeps"]}
    if kind in ("predict", "train"):
        vox = [c, c, c / 8, c / 8, c / 64, c / 64, c / 8, c / 8, c, c]
        f = sum(2 * 27 * i * o * v for (i, o), v in zip(LAYERS, vox))
        if kind == "train":
            return {"bytes": 9 * c * case["steps"], "flops": 3 * f * case["steps"]}
        return {"bytes": 9 * c, "flops": f}
    # the mesher's samples are on a grid of half the cell; a particle reaches about 64 of them
    b, f = 8 * fluid * 12 + 8 * c * 4, 8 * fluid * 64 * 10
    if kind == "draw":
        return {"bytes": b + 4 * case["width"] * case["height"], "flops": f + 8 * fluid * 200}
    return {"bytes": b, "flops": f}


def exact(case, seed):
    """The network's forward pass in 64 bits; the simulations have no such
    value (a step branches on the cell that each rounded position falls in)."""
    if case["kind"] != "predict":
        return None
    st = prepare(case, seed)
    with open(_weights_file(case), "rb") as fp:
        raw = fp.read()
    scale, at, layers = struct.unpack_from("<f", raw, 8)[0], 12, []
    for cin, cout in LAYERS:
        at += 8
        w = np.frombuffer(raw, np.float32, 27 * cin * cout, at).reshape(3, 3, 3, cout, cin)
        at += w.nbytes
        b = np.frombuffer(raw, np.float32, cout, at)
        at += b.nbytes
        layers.append((torch.from_numpy(w.astype(np.float64)).permute(3, 4, 0, 1, 2).contiguous().cuda(),
                       torch.from_numpy(b.astype(np.float64)).cuda()))
    head = torch.from_numpy(np.frombuffer(raw, np.float32, 17, at).astype(np.float64)).cuda()

    def conv(l, x):
        return torch.relu(torch.nn.functional.conv3d(x, layers[l][0], layers[l][1], padding=1))

    def pool(x):
        return torch.nn.functional.avg_pool3d(x, 2)

    def up(x, skip):
        return torch.cat([x.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4), skip], 1)

    rhs, fluid = st["rhs"].double(), st["type"].double()
    top = rhs.abs().max()
    x = torch.zeros((1, 16, rhs.numel()), dtype=torch.float64, device="cuda")
    x[0, 0], x[0, 1] = rhs / (top if float(top) > 0 else 1.0), fluid
    x = x.reshape(1, 16, *st["size"])
    e1 = conv(1, conv(0, x))
    e2 = conv(3, conv(2, pool(e1)))
    b2 = conv(5, conv(4, pool(e2)))
    d2 = conv(7, conv(6, up(b2, e2)))
    d1 = conv(9, conv(8, up(d2, e1)))
    out = (d1[0].reshape(16, -1) * head[:16, None]).sum(0) + head[16]
    return {"pressure": out * top * scale * fluid}
