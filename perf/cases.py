"""The workloads whose speed this framework is judged by, each a call or a short sequence of calls that a program using it makes.

Families (the `kind` of a case), all through vtwin's public Python entry points over the C ABI:

  path    one path-traced camera image: poses set, rendered, radiance copied to pinned host memory
  twin    one frame of the twin's cameras: moved instruments, node radiosity, twin shading, sensor chain, 8-bit images read back
  batch   one pose sweep of three cameras with the sensor's raw frames
  calib   one calibration step: image loss and the gradient in albedos, lamps and intrinsics
  nodes   the scene's node radiosity solved after the lamps moved, its state read back
  solve   the dense node radiosity B = E + rho F B in FP32 or mixed precision
  lite    one frame of the raster live renderer: shadow maps, three cameras and SCOPE, display look, 8-bit images read back

The geometry of a dome depends on its level alone; a seed draws the albedos, poses, cameras, targets and light sources.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "veridien-twin_gb300"))

from vtwin import _abi as A  # noqa: E402
from vtwin import dome  # noqa: E402
from vtwin import sensor as sensor_mod  # noqa: E402
from vtwin.calibrate import Calibration  # noqa: E402
from vtwin.lite import LiteNodesRenderer  # noqa: E402
from vtwin.renderer import TwinRenderer, form_factors, solve_radiosity  # noqa: E402

#: The reference's presets of a twin frame (its DEFAULTS are "judge").
PRESETS = {"live": {"spp": 1, "lightSamples": 1, "refine": 0, "radiosityEvery": 2, "itersPerFrame": 1},
           "balanced": {"spp": 1, "lightSamples": 2, "refine": 2, "refineLightSamples": 1, "refineShadows": False, "radiosityEvery": 2,
                        "itersPerFrame": 1},
           "judge": {"spp": 1, "refine": 6, "lightSamples": 4, "refineLightSamples": 1, "refineShadows": True, "radiosityEvery": 1,
                     "itersPerFrame": 4}}
PRECISION = {"fp32": A.VT_PREC_FP32, "bf16": A.VT_PREC_BF16, "fp8": A.VT_PREC_FP8}
N_POSES = 8       # kinematic poses that a twin or raster program cycles through


def listed():
    return [
        # a thumbnail while someone drags a camera: a few thousand paths, so launches and latency
        {"name": "path_thumbnail", "kind": "path", "width": 160, "height": 120, "spp": 1, "light_samples": 1, "depth": 4, "level": 5, "tools": 0},
        # the benchmark's headline image
        {"name": "path_dome", "kind": "path", "width": 640, "height": 480, "spp": 16, "light_samples": 1, "depth": 4, "level": 5, "tools": 0},
        # a tracking camera's full frame with six instruments in view, an offline still
        {"name": "path_full_frame", "kind": "path", "width": 1920, "height": 1200, "spp": 8, "light_samples": 2, "depth": 6, "level": 6, "tools": 6},
        # the live feed: three cameras at the reference's size on a scene of its size, one sub-sample, no refinement
        {"name": "twin_live", "kind": "twin", "preset": "live", "width": 1280, "height": 720, "level": 8, "tools": 6},
        # the same feed at the reference's default quality
        {"name": "twin_judge", "kind": "twin", "preset": "judge", "width": 1280, "height": 720, "level": 8, "tools": 6},
        # training images for a tracker: three cameras over a sweep of instrument poses
        {"name": "batch_sweep", "kind": "batch", "width": 960, "height": 600, "spp": 8, "poses": 16, "depth": 6, "level": 5, "tools": 6},
        # one optimiser step of a twin calibration
        {"name": "calib_step", "kind": "calib", "width": 480, "height": 300, "spp": 16, "depth": 3, "nodes": 4096, "level": 5},
        # the lamps moved, the room solved anew: direct light and every transport step of a converge() at the reference's node count
        {"name": "nodes_converge", "kind": "nodes", "iters": 96, "level": 8},
        # one lighting state of a small room, plain FP32
        {"name": "solve_fp32_one", "kind": "solve", "n": 4096, "rhs": 1, "precision": "fp32", "tol": 1e-6, "reuse": False},
        # many lighting states of a large room, plain FP32
        {"name": "solve_fp32_many", "kind": "solve", "n": 32768, "rhs": 64, "precision": "fp32", "tol": 1e-5, "reuse": False},
        # the same room relit again and again in mixed precision: F's converted copies are kept between solves
        {"name": "solve_bf16_relight", "kind": "solve", "n": 32768, "rhs": 64, "precision": "bf16", "tol": 1e-5, "reuse": True},
        # the raster live renderer at its own scene's size
        {"name": "lite_frame", "kind": "lite", "width": 1280, "height": 720, "level": 7, "tools": 6},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _image(rng, lo, hi):
    """Width and height of about lo to hi pixels, any remainder, landscape to portrait."""
    px, aspect = _log(rng, lo, hi), rng.uniform(0.7, 1.9)
    return max(8, int(math.sqrt(px * aspect))), max(8, int(math.sqrt(px / aspect)))


def draw(rng):
    kind = rng.choice(["path", "path", "path", "twin", "twin", "batch", "calib", "nodes", "solve", "solve", "solve", "lite"])
    if kind == "path":
        w, h = _image(rng, 3e3, 2.2e6)
        spp = max(1, min(32, int(_log(rng, 1, 32)), int(1.2e7 / (w * h))))
        return {"kind": kind, "width": w, "height": h, "spp": spp, "light_samples": rng.randint(1, 3), "depth": rng.randint(2, 6),
                "level": rng.randint(4, 7), "tools": rng.choice([0, 1, 3, 6])}
    if kind == "twin":
        w, h = _image(rng, 5e4, 9e5)
        return {"kind": kind, "preset": rng.choice(sorted(PRESETS)), "width": w, "height": h, "level": rng.randint(5, 8), "tools": rng.randint(1, 6)}
    if kind == "batch":
        w, h = _image(rng, 1e4, 5e5)
        return {"kind": kind, "width": w, "height": h, "spp": max(1, min(16, int(3e6 / (w * h)))), "poses": rng.randint(2, 16), "depth": rng.randint(3, 6),
                "level": rng.randint(4, 6), "tools": rng.randint(1, 6)}
    if kind == "calib":
        w, h = _image(rng, 1e4, 1.4e5)
        return {"kind": kind, "width": w, "height": h, "spp": rng.randint(2, 16), "depth": rng.randint(2, 4), "nodes": rng.choice([512, 1000, 2048, 4096]),
                "level": 5}
    if kind == "nodes":
        return {"kind": kind, "iters": rng.randint(8, 96), "level": rng.randint(4, 8)}
    if kind == "solve":
        precision = rng.choice(["fp32", "fp32", "bf16", "fp8"])
        rhs = rng.choice([1, 4 * rng.randint(1, 15), 64])
        n = int(_log(rng, 500, 30000))
        return {"kind": kind, "n": n if precision == "fp32" else max(512, n // 16 * 16), "rhs": rhs, "precision": precision,
                "tol": rng.choice([1e-5, 1e-6]), "reuse": precision != "fp32" and rng.random() < 0.5}
    w, h = _image(rng, 5e4, 9e5)
    return {"kind": kind, "width": w, "height": h, "level": rng.randint(5, 7), "tools": rng.randint(1, 6)}


# ------------------------------------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=None)
def _dome(level, tools):
    return dome.make_dome_scene(seed=1, width=64, height=48, level=level, with_instruments=tools)


@functools.lru_cache(maxsize=None)
def _scope(level, tools, width, height):
    return dome.make_scope_scene(seed=2, level=level, n_tools=tools, width=width, height=height)


def _scene(case, seed, cameras):
    """The dome of the case's level with this seed's albedos and cameras."""
    sc = dict(_dome(case["level"], case.get("tools", 0)))
    rng = dome.Rng(seed)
    sc["materials"] = [dict(m, rho=[rng.uniform(0.2, 0.8) for _ in range(3)]) if m["name"].startswith("mat") else m for m in sc["materials"]]
    w, h = case.get("width", 64), case.get("height", 48)
    if cameras == 3:
        sc["cameras"] = dome.batched_cameras(seed=seed + 2, n=3, width=w, height=h)
    else:
        f = 300.0 * w / 640 * rng.uniform(0.9, 1.1)
        at = (rng.uniform(-0.3, 0.3), -3.0 + rng.uniform(-0.2, 0.2), 1.5 + rng.uniform(-0.2, 0.2))
        sc["cameras"] = [dome.kb4_camera("CAM1", (w, h), f, f, (w - 1) / 2.0, (h - 1) / 2.0, (0.05, -0.01, 0.002, -0.0003),
                                         dome.look_at(at, (0.0, 0.0, 0.6)))]
    return sc


def _poses(case, seed, n):
    return dome.batch_pose_array(dome.instrument_poses(n_poses=n, n_tools=case.get("tools", 0), seed=seed + 11))


def _patches(case, seed):
    """Dome patches, their form factors on the device, and the emission columns."""
    P = dome.dome_patches(case["n"], seed=seed + 2)
    F = torch.empty((case["n"], case["n"]), dtype=torch.float32, device="cuda")
    form_factors(P["centres"], P["normals"], P["areas"], out=F)
    E = dome.radiosity_rhs(case["n"], P["lamps"], case["rhs"], seed=seed + 5, single_value=50.0 + seed % 7)
    return F, P["rho"], E


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "turn": 0}
    if kind == "solve":
        s["F"], s["rho"], s["E"] = _patches(case, seed)
        if case["reuse"]:
            # a handle of its own keeps this F's converted copies
            s["r"], s["kept"] = TwinRenderer.create(_scene({"level": 4}, 1, 1), nodes=False), False
        return s
    if kind == "lite":
        sc = dict(_scope(case["level"], case["tools"], case["width"], case["height"]))
        rng = dome.Rng(seed)
        sc["materials"] = [dict(m, rho=[rng.uniform(0.6, 0.9) for _ in range(3)]) if m["name"].startswith("pla") else m for m in sc["materials"]]
        s["r"] = LiteNodesRenderer.create(sc)
        P = dome.scope_poses(N_POSES, case["tools"], seed=seed + 21)
        for k in range(N_POSES):
            P[k, 0] = P[k - k % 4, 0]          # the scope rests for four frames, the tools move in each
        s["poses"] = P
        return s
    sc = _scene(case, seed, 1 if kind in ("path", "nodes") else 3)
    if kind == "path":
        s["r"] = TwinRenderer.create(sc, nodes=False)
        s["poses"] = _poses(case, seed, 1)[0]
        s["image"] = torch.zeros((case["height"], case["width"], 4), dtype=torch.float32).pin_memory().numpy()
        s["seed"] = seed
    elif kind == "twin":
        s["r"] = TwinRenderer.create(sc, **PRESETS[case["preset"]])
        s["poses"] = _poses(case, seed, N_POSES)
    elif kind == "batch":
        s["r"] = TwinRenderer.create(sc, nodes=False)
        s["poses"] = _poses(case, seed, case["poses"])
        s["sensor"] = sensor_mod.unit_radiance_sensor()
        s["raw"] = torch.zeros(3 * case["poses"] * case["height"] * case["width"], dtype=torch.int16).pin_memory()
    elif kind == "calib":
        r = s["r"] = TwinRenderer.create(sc, nodes=False)
        info = r.calib_setup(n_nodes=case["nodes"], lamp_samples=16)
        rng = np.random.default_rng(seed)
        albedo = np.clip(np.array([m["rho"] for m in sc["materials"]], np.float64), 0.05, 1.0)
        lamp = 50.0 * (1.0 + 0.2 * (rng.random(info["n_lamps"]) - 0.5))
        _, targets = r.calib_forward([0, 1, 2], albedo, lamp, spp=case["spp"], max_depth=case["depth"])
        d = rng.normal(size=(200, 3))
        d[:, 2] = np.abs(d[:, 2])
        points = 4.0 * d / np.linalg.norm(d, axis=1, keepdims=True)     # fiducials on the dome
        uv = np.stack([np.where(r.observed(c, points, margin=2.0)[:, None], r.project(c, points), np.nan) for c in range(3)])
        s["model"] = Calibration(r, [0, 1, 2], targets, fiducials=points, uv_targets=uv, w_reproj=1e-3, spp=case["spp"], max_depth=case["depth"],
                                 image_intrinsics=True)
        K = np.stack([r.get_intrinsics(c) for c in range(3)])
        s["x"] = s["model"].pack(np.clip(albedo * (1 + 0.1 * (2 * rng.random(albedo.shape) - 1)), 0.01, 1.0),
                                 lamp * (1 + 0.1 * (2 * rng.random(lamp.shape) - 1)), K * (1 + 0.002 * (2 * rng.random(K.shape) - 1)))
    elif kind == "nodes":
        s["r"] = TwinRenderer.create(sc)
        s["poses"] = _poses(case, seed, N_POSES)
        rng = dome.Rng(seed + 31)
        s["poses"][:, 0, 12:15] = [[rng.uniform(-0.2, 0.2) for _ in range(3)] for _ in range(N_POSES)]      # the lamps move
    return s


# ------------------------------------------------------------------------------------------------ a pass

def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "path":
        s["r"].set_pose_array(s["poses"])
        s["r"].renderCamera(0, out=s["image"], spp=case["spp"], lightSamples=case["light_samples"], seed=s["seed"] % 1000, mode=A.VT_SHADE_PATH,
                            max_depth=case["depth"])
        return s["image"]
    if kind in ("twin", "lite"):
        r = s["r"]
        r.set_pose_array(s["poses"][s["turn"] % N_POSES])
        s["turn"] += 1
        if kind == "lite":
            for c in r.cameras:
                r.renderCamera(c)
                r.sensor(c, gain=2.0)
            return [r.readback(c, "rgb8") for c in r.cameras]
        r.renderFrame(sensor=True, sensorOpts={"exposure_s": 2e-3, "gain": 1.0})
        return [r.readback(c, "rgb8") for c in range(3)]
    if kind == "batch":
        s["r"].render_batch([0, 1, 2], s["poses"], spp=case["spp"], max_depth=case["depth"], sensor=s["sensor"], raw_out=s["raw"])
        return s["raw"]
    if kind == "calib":
        loss, gradient = s["model"].loss_and_grad(s["x"])
        return loss, gradient
    if kind == "nodes":
        r = s["r"]
        r.set_pose_array(s["poses"][s["turn"] % N_POSES])
        s["turn"] += 1
        summary = r.converge(case["iters"])
        state, slot = r.get_node_state()
        return [summary[k] for k in ("area", "meanIndirect", "meanDirect", "meanLout", "eAvg")] + [state, slot]
    if case["reuse"]:
        B, _ = s["r"].solve_radiosity(s["F"], s["rho"], s["E"], precision=PRECISION[case["precision"]], tol=case["tol"], max_iters=400,
                                      reuse_f=s["kept"])
        s["kept"] = True
        return B
    B, _ = solve_radiosity(s["F"], s["rho"], s["E"], precision=PRECISION[case["precision"]], tol=case["tol"], max_iters=400)
    return B


# ------------------------------------------------------------------------------------------------ what a pass needs

#: Jacobi sweeps to 1e-5 of the residual on these rooms (albedos 0.1 to 0.9, rows of F summing to one or less).
SWEEPS = 16


def _ray_flops(case):
    """A ray's least arithmetic: two slab tests (24 operations) at each level of a balanced tree and one triangle test (40)."""
    return 24.0 * math.log2(len(_dome(case["level"], case.get("tools", 0))["static"]["I"])) + 40.0


def work(case):
    kind = case["kind"]
    if kind == "solve":
        n, r = case["n"], case["rhs"]
        per = {"fp32": 4, "bf16": 2, "fp8": 1}[case["precision"]] if case["reuse"] else 4
        return {"bytes": float(per) * n * n + 4.0 * n * (2 * r + 1), "flops": 2.0 * n * n * r * SWEEPS}
    if kind == "nodes":
        n = len(_dome(case["level"], 0)["static"]["P"])
        return {"bytes": n * (64.0 * 16 + 16 * 8 + 64 * 2), "flops": n * 64 * 6.0 * case["iters"]}
    px = case["width"] * case["height"]
    if kind == "lite":
        return {"bytes": 4 * px * 3.0 + 64.0 * 2 * len(_scope(case["level"], case["tools"], case["width"], case["height"])["static"]["I"]),
                "flops": 4 * px * 24 * 60.0}
    sc = _dome(case["level"], case.get("tools", 0))["static"]
    scene = 64.0 * 2 * len(sc["I"]) + 32.0 * len(sc["P"])
    if kind == "path":
        rays = px * case["spp"] * case["depth"] * (1 + 0.5 * case["light_samples"])
        return {"bytes": scene + 16.0 * px, "flops": rays * _ray_flops(case)}
    if kind == "twin":
        p = PRESETS[case["preset"]]
        # the camera rays' static hits and the settled occlusion are kept between frames: one ray to the light per sub-sample
        rays = 3 * px * p["spp"] * p["lightSamples"]
        return {"bytes": scene + 3 * px * 3.0, "flops": rays * _ray_flops(case)}
    if kind == "batch":
        rays = 3 * px * case["spp"] * case["depth"] * 1.5
        return {"bytes": scene + 3 * px * case["poses"] * 2.0, "flops": rays * _ray_flops(case)}
    rays = 3 * px * case["spp"] * case["depth"] * 1.5
    return {"bytes": scene + 3 * px * 16.0 + 4.0 * case["nodes"] ** 2, "flops": rays * _ray_flops(case) + 96 * 2 * 6.0 * case["nodes"] ** 2}


# ------------------------------------------------------------------------------------------------ in 64 bits

def exact(case, seed):
    """The dense solves in 64 bits (the other families have no closed value: sampled images, bytes)."""
    if case["kind"] != "solve":
        return None
    F, rho, E = _patches(case, seed)
    rho = torch.from_numpy(rho).cuda().double()[:, None]
    E = torch.from_numpy(E).cuda().double()
    B = E.clone()
    rows = 4096
    for _ in range(200):
        new = torch.empty_like(B)
        for i in range(0, len(F), rows):
            new[i:i + rows] = E[i:i + rows] + rho[i:i + rows] * (F[i:i + rows].double() @ B)
        done = float((new - B).norm()) <= 1e-13 * float(new.norm())
        B = new
        if done:
            break
    return B.cpu().numpy()
