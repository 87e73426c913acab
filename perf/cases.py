"""The work a user of this framework has it do, as timed cases.

Four kinds of pass, each through the package's public entry points:

* ``frame``   - one ``Renderer.render_frame`` of a prepared scene, every camera
  of the rig in one call, the next frame of a running sequence (history,
  reservoirs, moving cameras). With ``denoise`` the U-Net runs inside the
  frame; with ``download`` every camera's AOVs are copied to host memory.
* ``animate`` - ``Renderer.prepare_scene`` with the same scene moved (the
  acceleration structure is refitted), then a frame.
* ``load``    - ``Renderer.prepare_scene`` with another scene (a full build),
  then its first frame.
* ``train``   - one ``rtgb_trainer_step`` of the denoiser on a batch of crops,
  and its parameter gradients.

Scenes, rigs and profiles are the package's own; cameras orbit and the sample
stream starts where the seed says.
"""
from __future__ import annotations

import ctypes as C
from functools import lru_cache

import numpy as np
import torch

from ray_tracing_gb300 import abi, denoiser, scenes
from ray_tracing_gb300.renderer import Renderer

# per scene: the degrees a rig may be turned about the scene's centre by the
# seed (the acceptance scene is only seen from the front)
SCENES = {
    "restir_acceptance": 4.0, "smoke": 360.0, "final_room": 360.0, "bouncing_spheres": 360.0, "cornell_box": 12.0,
    "random_spheres": 360.0, "openpbr_gallery": 12.0, "triangle_terrain": 360.0, "triangle_terrain_pbr": 360.0,
    "textured_room": 360.0,
}
CENTER = {"cornell_box": (278.0, 278.0, 278.0), "openpbr_gallery": (0.0, 1.0, 6.0)}
ORBIT = 2.0       # degrees per frame of a moving rig
POSES = 8         # frames after which a moving rig starts over
FRAME = {"kind": "frame", "seeded": False, "detail": 0, "cameras": 4, "width": 0, "height": 0, "spp": 1, "bounces": 4,
         "restir": True, "candidates": 4, "spatial": 1, "emissive": False, "denoise": False, "orbit": False,
         "download": False}


def listed():
    """Twelve cases from the smallest call to the largest."""
    def frame(name, scene, **kw):
        return dict(FRAME, name=name, scene=scene, **kw)

    return [
        # the ReSTIR acceptance scene: one small camera, launch and latency bound
        frame("acceptance_128", "restir_acceptance", cameras=1, bounces=1, candidates=8),
        # the published realtime protocol: trivial scene, two bounces, denoised
        frame("smoke_realtime_4x640x480", "smoke", width=640, height=480, bounces=2, denoise=True),
        # the headline frame: 1024 area lights, 32-candidate ReSTIR, denoised
        frame("spheres_restir_4x640x480", "random_spheres", detail=1024, width=640, height=480, candidates=32,
              denoise=True),
        # offline-quality settings on a tiny scene: many samples, deep paths
        frame("cornell_256_64spp", "cornell_box", cameras=1, width=256, height=256, spp=64, bounces=8, restir=False),
        # OpenPBR features at an odd size, two cameras, downloaded to the host
        frame("gallery_333x217_4spp", "openpbr_gallery", seeded=True, detail=24, cameras=2, width=333, height=217,
              spp=4, bounces=8, download=True),
        # an ordinary plain render with media-free legacy materials, one HD camera
        frame("final_room_1280x720_4spp", "final_room", cameras=1, width=1280, height=720, spp=4, bounces=8,
              restir=False),
        # a million OpenPBR triangles seen by two pinhole and two fisheye cameras
        frame("terrain_1m_mixed_rig", "triangle_terrain_pbr", detail=1000000),
        # the largest: four million triangles, mixed 1080p rig on an orbit, denoised
        frame("room_4m_4x1080p_orbit", "textured_room", bounces=6, candidates=32, denoise=True, orbit=True),
        # a deforming mesh: refit, then a frame
        dict(FRAME, name="animate_200k", kind="animate", scene="triangle_terrain", detail=200000, cameras=1, width=640,
             height=480, bounces=2),
        # a scene switch: full build of a million triangles, then the first frame
        dict(FRAME, name="load_1m", kind="load", scene="triangle_terrain_pbr", detail=1000000, cameras=1, width=640,
             height=480, bounces=2),
        # denoiser training: the recipe's batch, and a small odd one
        {"name": "train_16x256x256", "kind": "train", "batch": 16, "height": 256, "width": 256},
        {"name": "train_3x100x76", "kind": "train", "batch": 3, "height": 100, "width": 76},
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    kind = rng.choice(("frame",) * 6 + ("animate", "load", "train", "train"))
    if kind == "train":
        h, w = 4 * int(_log(rng, 8, 65)), 4 * int(_log(rng, 8, 65))
        return {"kind": "train", "batch": max(1, min(16, int(_log(rng, 1, 17)))), "height": h, "width": w}
    case = dict(FRAME, kind=kind)
    if kind == "frame":
        case["scene"] = rng.choice(tuple(SCENES))
    else:
        case["scene"] = rng.choice(("triangle_terrain", "triangle_terrain_pbr", "textured_room"))
    scene = case["scene"]
    if scene == "random_spheres":
        case["detail"] = int(_log(rng, 16, 2049))
        case["seeded"] = True
    elif scene == "openpbr_gallery":
        case["detail"] = int(_log(rng, 8, 97))
        case["seeded"] = True
    elif scene.startswith("triangle_terrain"):
        case["detail"] = int(_log(rng, 2000, 1000001))
        case["seeded"] = True
    elif scene == "textured_room":
        case["detail"] = int(_log(rng, 200000, 2000001))
        case["seeded"] = True
    case["cameras"] = 1 if scene == "restir_acceptance" else rng.randint(1, 4)
    case["bounces"] = rng.choice((1, 2, 4, 6, 8))
    case["restir"] = rng.random() < 0.7
    case["candidates"] = rng.choice((4, 8, 32))
    case["spatial"] = rng.choice((0, 1, 2))
    case["emissive"] = bool(case["restir"] and scene not in ("restir_acceptance", "random_spheres") and rng.random() < 0.25)
    if case["emissive"]:  # each candidate costs a BSDF evaluation
        case["candidates"] = 4
    case["denoise"] = kind == "frame" and rng.random() < 0.4
    case["orbit"] = rng.random() < 0.5
    case["download"] = kind == "frame" and rng.random() < 0.15
    pixels = _log(rng, 10000, 2100000)
    if scene != "restir_acceptance":
        case["width"] = max(33, int((pixels * rng.choice((1.0, 4.0 / 3.0, 16.0 / 9.0))) ** 0.5))
        case["height"] = max(17, int(pixels / case["width"]))
    else:
        case["width"] = case["height"] = 128
    # no more path segments than the smaller scenes' largest listed case
    room = 3.0e7 / (case["width"] * case["height"] * case["cameras"] * case["bounces"])
    case["spp"] = 1 if case["denoise"] else int(_log(rng, 1, 16))
    while case["spp"] > 1 and case["spp"] > room:
        case["spp"] //= 2
    if room < 1:
        case["cameras"], case["bounces"] = 1, min(case["bounces"], 4)
    return case


@lru_cache(maxsize=3)
def _host_scene(name, seed, detail):
    return scenes.HostScene(name, seed=seed, detail=detail)


def _rigs(case, rng):
    rig = scenes.default_rig(case["scene"], case["cameras"], case["width"], case["height"])
    turn = SCENES[case["scene"]]
    start = (rng.random() - 0.5) * turn
    center = CENTER.get(case["scene"], (0.0, 0.0, 0.0))
    n = POSES if case["orbit"] else 1
    step = min(ORBIT, turn / (4 * POSES))
    return [scenes.orbit_rig(rig, start + step * i, center) for i in range(n)]


def _profile(case):
    return scenes.profile("balanced", samples_per_pixel=case["spp"], max_bounces=case["bounces"],
                          enable_denoise=int(case["denoise"]), enable_restir_di=int(case["restir"]),
                          restir_initial_candidates=case["candidates"], restir_spatial_neighbors=case["spatial"],
                          restir_emissive=int(case["emissive"]))


class _DeviceArray:
    """A frame view's device buffer, as torch reads foreign arrays; tensors over
    it keep this object, and with it the renderer that owns the buffer."""

    def __init__(self, renderer, ptr, shape):
        self.renderer = renderer
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f4", "version": 3}


def _views(state, views):
    """The frame's AOVs as tensors over the renderer's two ping-pong buffer
    sets, made once per set."""
    key = views.cameras[0].beauty
    got = state["views"].get(key)
    if got is None:
        got = []
        for c in range(views.camera_count):
            v = views.cameras[c]
            for field, ch in (("beauty", 4), ("normal", 4), ("denoiser_normal", 4), ("albedo", 4), ("depth", 1),
                              ("flow", 2), ("flow_trustworthiness", 1)):
                array = _DeviceArray(state["renderer"], getattr(v, field), (v.height, v.width, ch))
                got.append(torch.as_tensor(array, device="cuda"))
        state["views"][key] = got
    return got


def _moved(view, rng):
    """Two copies of a triangle scene whose points wave up and down."""
    n = view.triangle_count
    words = C.sizeof(abi.Triangle) // 4
    base = np.frombuffer((C.c_float * (words * n)).from_address(C.addressof(view.triangles.contents)),
                         dtype=np.float32).reshape(n, words)
    out = []
    for _ in range(2):
        tris = base.copy()
        phase, amp = 6.28 * rng.random(), 0.05 + 0.05 * rng.random()
        for k in range(3):
            x, z = tris[:, 3 * k], tris[:, 3 * k + 2]
            tris[:, 3 * k + 1] += np.float32(amp) * np.sin(np.float32(0.7) * x + np.float32(0.9) * z + np.float32(phase))
        moved = abi.Scene()
        C.pointer(moved)[0] = view
        moved.triangles = C.cast(tris.ctypes.data, C.POINTER(abi.Triangle))
        out.append((moved, tris))
    return out


def _train_data(case, seed):
    """Network inputs and targets as the tracer's frames have them: albedo and
    normals of piecewise flat surfaces, noisy radiance, its clean counterpart."""
    n, h, w = case["batch"], case["height"], case["width"]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def patches(ch, cell):
        x = torch.rand((n, ch, -(-h // cell), -(-w // cell)), generator=g, device="cuda")
        return x.repeat_interleave(cell, 2).repeat_interleave(cell, 3)[:, :, :h, :w]

    albedo = patches(3, 12)
    normal = patches(3, 20) * 2.0 - 1.0
    normal = normal / normal.norm(dim=1, keepdim=True).clamp_min(1e-3)
    depth = 1.0 + 12.0 * patches(1, 24)
    clean = albedo * (0.1 + 2.0 * patches(3, 32) ** 2)
    noise = torch.rand((n, 1, h, w), generator=g, device="cuda")
    noisy = clean * torch.where(noise < 0.35, 0.0, 1.0 / 0.65) * (
        0.5 + torch.rand((n, 3, h, w), generator=g, device="cuda"))
    x = torch.cat([torch.log1p(noisy), albedo, normal, torch.log1p(depth)], 1)
    target = torch.log1p(clean).permute(0, 2, 3, 1).contiguous()
    torch.manual_seed(seed)
    flat = denoiser.flatten(denoiser.build_model())
    return denoiser.blocked_input(x), target, flat


class _Trainer:
    def __init__(self, case, flat):
        self.lib, self.h = abi.load(), C.c_void_p()
        abi.check(self.lib.rtgb_trainer_create(case["batch"], case["height"], case["width"], flat.ctypes.data, flat.size,
                                               C.byref(self.h)), what="rtgb_trainer_create")

    def __del__(self):
        if self.h:
            self.lib.rtgb_trainer_destroy(self.h)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "train":
        x, target, flat = _train_data(case, seed)
        torch.cuda.synchronize()  # the trainer has a stream of its own
        return {"case": case, "trainer": _Trainer(case, flat), "x": x, "target": target,
                "grads": np.empty(flat.size, np.float32)}
    scene_seed = 1 + seed % 1009 if case["seeded"] else 0
    host = _host_scene(case["scene"], scene_seed, case["detail"])
    state = {"case": case, "rigs": _rigs(case, rng), "profile": _profile(case), "views": {}, "i": 0, "host": host}
    r = state["renderer"] = Renderer()
    if case["kind"] == "animate":
        state["scenes"] = _moved(host.view, rng)
    elif case["kind"] == "load":
        other = _host_scene(case["scene"], scene_seed + 1, case["detail"] - case["detail"] // 50)
        state["other"] = other
        state["scenes"] = [(other.view, None), (host.view, None)]
    r.prepare_scene(state["scenes"][1][0] if "scenes" in state else host.view)
    if case["denoise"]:
        r.set_denoiser(denoiser.load_weights())
    r.reset_sequence(1 + seed)
    # the sequence is running: the first frames carry the graph's capture
    for _ in range(2):
        _views(state, r.render_frame(state["rigs"][0], state["profile"], case["cameras"]))
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "train":
        t = state["trainer"]
        loss = C.c_float()
        abi.check(t.lib.rtgb_trainer_step(t.h, state["x"].data_ptr(), state["target"].data_ptr(), 1e-3, C.byref(loss)),
                  what="rtgb_trainer_step")
        abi.check(t.lib.rtgb_trainer_gradients(t.h, state["grads"].ctypes.data), what="rtgb_trainer_gradients")
        return {"grads": state["grads"], "loss": np.float32(loss.value)}
    r, i = state["renderer"], state["i"]
    state["i"] = i + 1
    if "scenes" in state:
        r.prepare_scene(state["scenes"][i % 2][0])
    views = r.render_frame(state["rigs"][i % len(state["rigs"])], state["profile"], case["cameras"])
    out = _views(state, views)
    if case["download"]:
        out = [a for c in range(case["cameras"]) for f in (r.download(c),)
               for a in (f.beauty_rgba, f.normal_rgba, f.albedo_rgba, f.depth)]
    return {"aovs": out, "rays": int(views.rays_traced)}


def exact(case, seed):
    """The training step's loss and gradients by autograd in 64 bits. A path
    tracer's frame has no 64-bit value: its decisions (lobes, light picks,
    Russian roulette) follow the single-precision arithmetic."""
    if case["kind"] != "train":
        return None
    x, target, flat = _train_data(case, seed)
    n, h, w = case["batch"], case["height"], case["width"]
    model = denoiser.build_model()
    denoiser.unflatten(model, flat)
    model = model.double().cuda()
    y = model(x.permute(0, 1, 4, 2, 3).reshape(n, 16, h, w)[:, :10].double())
    loss = torch.nn.functional.l1_loss(y, target.double().permute(0, 3, 1, 2))
    loss.backward()
    grads = torch.cat([p.grad.reshape(-1) for conv in model.convs for p in (conv.weight, conv.bias)])
    return {"grads": grads, "loss": loss.detach()}


def _sizes(case):
    """(width, height) of every camera."""
    rig = scenes.default_rig(case["scene"], case["cameras"], case["width"], case["height"])
    return [(rig.cameras[c].width, rig.cameras[c].height) for c in range(case["cameras"])]


def _unet_flops(pixels):
    scale = (1, 1, 4, 4, 16, 16, 4, 4, 1, 1, 1)
    return sum(2.0 * 9 * i * o * pixels / s for (i, o), s in zip(denoiser.LAYERS, scale))


def work(case):
    """Bytes: the scene's primitives and triangles read (on a scene change from
    the host: uploaded) once, the AOVs written once, the history a frame of a
    running sequence reads; ReSTIR's reservoirs read and written. Operations:
    per path segment a closest-hit and a shadow ray of 2 log2(primitives)
    box tests and a few hundred for shading; the denoiser's convolutions."""
    if case["kind"] == "train":
        pixels = case["batch"] * case["height"] * case["width"]
        params = denoiser.param_count()
        return {"bytes": pixels * (32.0 + 12.0) + params * 4.0 * 8, "flops": 3.0 * _unet_flops(pixels)}
    pixels = float(sum(w * h for w, h in _sizes(case)))
    triangles = case["scene"].startswith(("triangle", "textured"))
    if triangles:
        prims = case["detail"] or 4000000
    else:
        prims = {"random_spheres": 485, "restir_acceptance": 129}.get(case["scene"], 20)
    restir = case["restir"] and (case["emissive"] or case["scene"] in ("restir_acceptance", "random_spheres",
                                                                       "openpbr_gallery"))
    changed = 0.0 if case["kind"] == "frame" else 108.0 + 64.0 + 128.0
    bytes_ = pixels * (80.0 + 36.0 + (192.0 if restir else 0.0)) + prims * (64.0 + (108.0 if triangles else 0.0) + changed)
    segments = pixels * case["spp"] * (1.0 + 0.6 * (case["bounces"] - 1))
    flops = segments * (2 * 2 * np.log2(prims + 2) * 12.0 + 400.0)
    if case["denoise"]:
        flops += _unet_flops(pixels)
    return {"bytes": bytes_, "flops": float(flops)}
