"""The work a user of this framework has it do, as timed cases.

Each case goes through the public entry points: `Renderer` frames with a moving
camera read back to the host (forward and deferred, plain and learned ambient
occlusion), the frame's TGA files, many views as one `Batch`, and the
learned-AO network's forward and training step. Scenes, resolutions and sample
counts are those of the benchmark and the tests, or generic ones around them.

A case's scene has one set of model and texture files (generated once into the
temporary directory); the seed places the models and the camera.
"""

from __future__ import annotations

import math
import os
import random
import tempfile

import numpy as np
import torch

import forkerrenderer_gb300 as fr
from forkerrenderer_gb300 import _native as N
from forkerrenderer_gb300 import output, scenegen
from forkerrenderer_gb300.aonet import AONet
from forkerrenderer_gb300.batch import Batch, directional_light, point_light, view

WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(fr.__file__)), "weights", "aonet_field20_ssao16.f32")
PROBE_THRESHOLD = 0.01377  # the shipped model's: the learned AO stays in use
INPUT_SAMPLES = 16

# ---- scenes -------------------------------------------------------------------------

# name -> (generator, arguments, model files, triangles and vertices of a model, texels of all textures in bytes)
ASSETS = {
    "sphere": ("sphere", dict(seed=0, lon=64, lat=32, tex=256), 1, 4032, 2145, 256 * 256 * 3),
    "small": ("field", dict(seed=2, n_spheres=4, subdiv=2, tex=64), 4, 320, 162, 5 * 64 * 64 * 8),
    "field": ("field", dict(seed=0, n_spheres=20, subdiv=5, tex=1024), 20, 20480, 10242, 21 * 1024 * 1024 * 8),
}


def _assets(name: str) -> str:
    kind, kw = ASSETS[name][:2]
    out = os.path.join(tempfile.gettempdir(), "fr_perf_%s_%d" % (name, os.getuid()))
    if not os.path.exists(os.path.join(out, "scene.scene")):
        tmp = out + ".tmp%d" % os.getpid()
        (scenegen.forward_sphere_scene if kind == "sphere" else scenegen.deferred_field_scene)(tmp, **kw)
        try:
            os.rename(tmp, out)
        except OSError:
            pass  # another process wrote the same files
    return out


def _scene(case: dict, seed: int) -> fr.Scene:
    """The case's scene with its models placed by the seed."""
    assets = case["assets"]
    folder = _assets(assets)
    rng = random.Random(seed)
    if assets == "sphere":
        models = [("sphere.obj", False, (rng.uniform(-0.3, 0.3), 0.0, rng.uniform(-2.3, -1.7)), rng.uniform(0, 360), 1.0),
                  ("plane.obj", False, (0, 0, 0), 0, 1)]
        light, eye, target = (2, 5, 5), (-1, 1, 1), (0, 0, -1)
    else:
        models = [("ground.obj", True, (0.0, 0.0, 0.0), 0.0, 1.0)]
        for i in range(case["models"]):
            scale = rng.uniform(0.3, 1.0)
            models.append(("ico%d.obj" % (i % ASSETS[assets][2]), True, (rng.uniform(-5, 5), scale, rng.uniform(-5, 5)),
                           rng.uniform(0, 360), scale))
        light, eye, target = (3, 9, 6), (0, 7, 11), (0, 0, 0)
    spec = scenegen.SceneSpec(case["width"], case["height"], case["deferred"], case["deferred"], True,
                              case.get("ssaa", 0), light, (1, 1, 1), eye, target, models)
    path = os.path.join(folder, "perf_%d_%d.scene" % (os.getpid(), rng.getrandbits(40)))
    spec.write(path)
    try:
        return fr.Scene(path)
    finally:
        os.unlink(path)


def _triangles(case: dict) -> int:
    return 2 + (case["models"] if case["assets"] != "sphere" else 1) * ASSETS[case["assets"]][3]


def _vertices(case: dict) -> int:
    return 4 + (case["models"] if case["assets"] != "sphere" else 1) * ASSETS[case["assets"]][4]


def _network(seed: int = 0) -> AONet:
    net = AONet(0, seed)
    net.set_params(np.fromfile(WEIGHTS, "<f4"))
    return net


def _renderer(case: dict, scene: fr.Scene, **more) -> fr.Renderer:
    cfg = dict(shadow_mode=case["shadow"], shadow_size=case["shadow_size"], pcf_samples=case["pcf"],
               blocker_samples=case["blocker"], ssao_samples=case["ssao"], ssao_radius=case["radius"],
               blur_mode=case.get("blur", N.FR_BLUR_REFERENCE), texture_wrap=case.get("wrap", 0),
               texture_filter=case.get("filter", 0))
    cfg.update(more)
    r = fr.Renderer(**cfg)
    r.Preconfigure(scene)
    return r


# ---- network inputs -----------------------------------------------------------------


def _smooth(g, B, C, H, W, cells):
    low = torch.rand((B, C, cells, cells), generator=g, device="cuda")
    return torch.nn.functional.interpolate(low, (H, W), mode="bicubic", align_corners=False).clamp(0, 1)


def _views(case: dict, seed: int):
    """(input channels (B, 4, H, W), label (B, H, W)): view depth / 8, view normal x and y and
    a 16-sample ambient occlusion of smooth surfaces in front of an empty background, and
    the occlusion itself (-1 where there is only background)."""
    B, H, W = case["batch"], case["height"], case["width"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    depth = 0.4 + 0.9 * _smooth(g, B, 1, H, W, 7)
    dx = torch.nn.functional.pad(depth[..., 1:] - depth[..., :-1], (0, 1)) * 120
    dy = torch.nn.functional.pad(depth[..., 1:, :] - depth[..., :-1, :], (0, 0, 0, 1)) * 120
    n = torch.rsqrt(1 + dx * dx + dy * dy)
    ao = _smooth(g, B, 1, H, W, 11) ** 0.5
    hits = torch.floor(16 * (1 - ao) + torch.rand((B, 1, H, W), generator=g, device="cuda")).clamp(0, 16)
    covered = (_smooth(g, B, 1, H, W, 3) > 0.2).float()
    x = torch.cat([depth, -dx * n, -dy * n, (1 - hits / 16) ** 3], 1) * covered
    label = torch.where(covered > 0, ao, torch.full_like(ao, -1.0))[:, 0].contiguous()
    return x.to(torch.bfloat16), label


def _packed(x: torch.Tensor) -> torch.Tensor:
    B, C, H, W = x.shape
    out = torch.zeros((B, 1, H, W, 8), dtype=torch.bfloat16, device="cuda")
    out[:, 0, :, :, :C] = x.permute(0, 2, 3, 1)
    return out


# ---- the cases ----------------------------------------------------------------------

_BENCH = dict(shadow=N.FR_SHADOW_PCSS, shadow_size=2048, pcf=25, blocker=16, ssao=64, radius=0.5)
_REFERENCE = dict(shadow=N.FR_SHADOW_PCSS, shadow_size=0, pcf=64, blocker=32, ssao=32, radius=0.075)


def listed():
    return [
        # a thumbnail or a test image of a small model under the reference's own settings, launch by launch
        dict(name="frame_small_161x97", kind="frame", assets="small", models=4, width=161, height=97, deferred=True,
             graph=False, ao="ssao", **_REFERENCE),
        # the forward Blinn-Phong frame with a hard shadow map: the reference's plain mode
        dict(name="frame_forward_640x400", kind="frame", assets="sphere", models=1, width=640, height=400,
             deferred=False, graph=False, ao="ssao", **dict(_BENCH, shadow=N.FR_SHADOW_HARD, shadow_size=1024)),
        # the headline frame: an interactive viewer or a camera path, frame after frame
        dict(name="frame_1280x800", kind="frame", assets="field", models=20, width=1280, height=800, deferred=True,
             graph=True, ao="ssao", **_BENCH),
        # a window of odd size with the quality options set otherwise: PCF, bilinear textures, repeat, parallel blur
        dict(name="frame_options_1917x1071", kind="frame", assets="field", models=20, width=1917, height=1071,
             deferred=True, graph=False, ao="ssao", blur=N.FR_BLUR_SEPARABLE, wrap=1, filter=1,
             **dict(_BENCH, shadow=N.FR_SHADOW_PCF, shadow_size=3000)),
        # a final picture: two million triangles, 2x2 supersampling, a 4096^2 shadow map
        dict(name="frame_ssaa_2560x1600", kind="frame", assets="field", models=100, width=1280, height=800, ssaa=2,
             deferred=True, graph=False, ao="ssao", **dict(_BENCH, shadow_size=4096)),
        # the headline frame with the learned ambient occlusion
        dict(name="frame_learned_1280x800", kind="frame", assets="field", models=20, width=1280, height=800,
             deferred=True, graph=True, ao="learned", **_BENCH),
        # the TGA files of a frame, as the reference's main writes them after it
        dict(name="files_1280x800", kind="files", assets="field", models=20, width=1280, height=800, deferred=True,
             rle=True, **_BENCH),
        # a few odd-sized views under a point and a directional light: thumbnails of one scene from several sides
        dict(name="batch_5_views", kind="batch", assets="field", models=20, width=1280, height=800, deferred=True,
             views=5, sizes="odd", size_seed=1, lights=2, point=True, learned=False, **_BENCH),
        # a data set's views in one go: uneven sizes, four directional lights, learned AO where the size allows it
        dict(name="batch_64_views", kind="batch", assets="field", models=20, width=1280, height=800, deferred=True,
             views=64, sizes="mixed", size_seed=4, lights=4, point=False, learned=True,
             **dict(_BENCH, shadow=N.FR_SHADOW_PCF)),
        # the network by itself on a frame's worth of input
        dict(name="network_1280x800", kind="network", batch=1, width=1280, height=800),
        # the network on a single small crop: latency only
        dict(name="network_96x64", kind="network", batch=1, width=96, height=64),
        # one training step at the trainer's batch and crop
        dict(name="train_16x256", kind="train", batch=16, width=256, height=256),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "files", "batch", "network", "train"])
    if kind in ("network", "train"):
        B = _log_int(rng, 1, 16)
        W, H = 32 * _log_int(rng, 1, 40), 32 * _log_int(rng, 1, 25)
        while B * W * H > 16 * 256 * 256 * (4 if kind == "network" else 1):
            B, W = max(1, B // 2), W if B > 1 else W // 64 * 32
        return dict(kind=kind, batch=B, width=W, height=H)
    assets = rng.choice(["sphere", "small", "field", "field"])
    models = 1 if assets == "sphere" else rng.randint(1, ASSETS[assets][2]) if rng.random() < 0.5 else \
        _log_int(rng, 1, 100 if assets == "field" else 20)
    width = _log_int(rng, 64, 2200)
    height = max(40, min(1400, int(width * rng.uniform(0.5, 0.8))))
    config = dict(shadow=rng.randrange(3), shadow_size=rng.choice([0, 512, 1024, 2048, _log_int(rng, 256, 4096)]),
                  pcf=rng.choice([16, 25, 64]), blocker=rng.choice([16, 32]), ssao=rng.choice([16, 32, 64, 128]),
                  radius=rng.choice([0.075, 0.5]), blur=rng.choice([0, 0, 1]), wrap=rng.randrange(4),
                  filter=rng.choice([0, 0, 1]))
    if kind == "files":
        return dict(kind=kind, assets=assets, models=models, width=width, height=height, deferred=rng.random() < 0.7,
                    rle=rng.random() < 0.7, **config)
    if kind == "batch":
        config["shadow_size"] = config["shadow_size"] or 1024
        return dict(kind=kind, assets=assets, models=min(models, 20), width=1280, height=800, deferred=True,
                    views=_log_int(rng, 1, 24), sizes=rng.choice(["odd", "mixed"]), size_seed=rng.randrange(1000),
                    lights=rng.randint(1, 4), point=rng.random() < 0.5, learned=rng.random() < 0.5,
                    **dict(config, ssao=min(config["ssao"], 64)))
    ao = rng.choice(["ssao", "ssao", "learned"])
    deferred = ao == "learned" or rng.random() < 0.7
    if ao == "learned":
        width, height = max(64, width // 32 * 32), max(64, height // 32 * 32)
    ssaa = 0 if ao == "learned" or width > 1280 else rng.choice([0, 0, 2, 3 if width <= 640 else 2])
    return dict(kind=kind, assets=assets, models=models, width=width, height=height, ssaa=ssaa, deferred=deferred,
                graph=rng.random() < 0.5, ao=ao, **config)


_MIXED = [(256, 256), (640, 400), (1280, 800), (1920, 1080)]


def _view_sizes(case: dict):
    rng = random.Random(case["size_seed"])
    if case["sizes"] == "mixed":
        return [rng.choice(_MIXED) for _ in range(case["views"])]
    return [(rng.randint(50, 1100), rng.randint(50, 800)) for _ in range(case["views"])]


def _batch(case: dict, seed: int) -> dict:
    scene = _scene(case, seed)
    r = _renderer(case, scene, ao_probe_threshold=1e9, ao_input_samples=INPUT_SAMPLES)
    net = _network()
    r.set_ao_net(net)
    rng = random.Random(seed + 1)
    views = []
    for w, h in _view_sizes(case):
        # a camera on the hemisphere around the scene, with the view's own viewport
        rad, ct, ph = rng.uniform(4, 8), rng.uniform(0.25, 0.95), rng.uniform(0, 2 * math.pi)
        st = math.sqrt(1 - ct * ct)
        eye = (rad * st * math.cos(ph), rad * ct, rad * st * math.sin(ph))
        m = scene.view_matrices(eye, (0, 0, 0), case["shadow_size"])
        m.width, m.height = w, h
        m.viewport[:] = [w / 2, 0, 0, w / 2, 0, h / 2, 0, h / 2, 0, 0, 0.5, 0.5, 0, 0, 0, 1]
        learned = case["learned"] and w % 32 == 0 and h % 32 == 0
        views.append(view(m, eye, N.FR_AO_LEARNED if learned else N.FR_AO_SSAO))
    lights = [directional_light((rng.uniform(-0.6, 0.6), -1.0, rng.uniform(-0.6, 0.6)), (0.6, 0.55, 0.5),
                                case["shadow_size"], 6.0) for _ in range(case["lights"])]
    if case["point"]:
        lights[0] = point_light((3.0, 9.0, 6.0), (0.9, 0.9, 0.8), case["shadow_size"])
    return dict(batch=Batch(r, views, lights), renderer=r, network=net, scene=scene, views=len(views))


def _camera(state: dict):
    """The next camera of the state's orbit: (frame matrices, eye)."""
    state["step"] += 1
    a = state["angle"] + math.radians(0.5 * state["step"])
    c, rad, y = state["centre"], state["distance"], state["eye_y"]
    eye = (c[0] + rad * math.sin(a), y, c[2] + rad * math.cos(a))
    return state["scene"].view_matrices(eye, c, state["shadow_size"]), eye


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("network", "train"):
        x, label = _views(case, seed)
        state = dict(net=_network(), x=_packed(x), label=label, B=case["batch"], H=case["height"], W=case["width"])
        state["ao"] = torch.empty((case["batch"], case["height"], case["width"]), device="cuda")
    elif kind == "batch":
        state = _batch(case, seed)
    else:
        scene = _scene(case, seed)
        more = {}
        if kind == "frame":
            more = dict(frame_graph=int(case["graph"]), pass_timings=int(not case["graph"]))
            if case["ao"] == "learned":
                more.update(ao_mode=N.FR_AO_LEARNED, ao_probe_threshold=PROBE_THRESHOLD, ao_input_samples=INPUT_SAMPLES)
        r = _renderer(case, scene, **more)
        state = dict(renderer=r, scene=scene, step=0, shadow_size=case["shadow_size"])
        if more.get("ao_mode"):
            r.set_ao_net(_network())
        eye, centre = scene.info.eye, scene.info.target
        state["centre"] = tuple(centre)
        state["distance"] = math.hypot(eye[0] - centre[0], eye[2] - centre[2])
        state["angle"] = math.atan2(eye[0] - centre[0], eye[2] - centre[2]) + random.Random(seed + 1).uniform(-0.5, 0.5)
        state["eye_y"] = eye[1]
        if kind == "frame":
            ssaa = bool(case.get("ssaa", 0))
            state["buffer"] = N.FR_BUF_SSAA_U8 if ssaa else N.FR_BUF_FRAME_U8
            state["image"] = torch.empty(case["width"] * case["height"] * 3, dtype=torch.uint8, pin_memory=True).numpy()
        else:
            m, eye = _camera(state)
            r.set_matrices(m, eye)
            r.Render()
            state["rle"] = case["rle"]
            state["files"] = torch.zeros(output.max_bytes(r), dtype=torch.uint8, pin_memory=True).numpy()
    state["kind"] = kind
    return state


def run(state):
    kind = state["kind"]
    if kind == "frame":
        # a viewer's frame: new camera matrices in, the 8-bit picture out
        m, eye = _camera(state)
        r = state["renderer"]
        r.set_matrices(m, eye)
        r.Render()
        return r.download(state["buffer"], state["image"])
    if kind == "files":
        sizes, _ = output.encode_all_into(state["renderer"], state["files"], state["rle"])
        return {"sizes": sizes, "files": state["files"]}  # the files one after the other, then untouched bytes
    if kind == "batch":
        b = state["batch"]
        b.render()
        return [b.download(i, N.FR_BUF_FRAME_U8) for i in range(state["views"])]
    if kind == "network":
        state["net"].forward(state["x"], state["B"], state["H"], state["W"], state["ao"])
        return state["ao"]
    loss = state["net"].train_step(state["x"], state["label"], state["B"], state["H"], state["W"])
    return {"loss": loss, "grads": state["net"].get_grads()}


# ---- what a pass cannot do without --------------------------------------------------

# (input channels, output channels, level) of the network's 3x3 convolutions; each level is 4x coarser,
# level 0 works on 2x2 pixel blocks
LAYERS = [(16, 16, 0), (16, 16, 0), (16, 32, 1), (32, 32, 1), (32, 64, 2), (64, 64, 2), (96, 32, 1), (32, 32, 1),
          (48, 16, 0), (16, 16, 0)]
NUM_PARAMS = sum(ci * co * 9 + co for ci, co, _ in LAYERS) + 68


def _network_flops(pixels: int) -> int:
    blocks = pixels // 4
    return sum(blocks // 16 ** lv * ci * co * 9 * 2 for ci, co, lv in LAYERS) + blocks * 16 * 4 * 2


def work(case):
    kind = case["kind"]
    if kind in ("network", "train"):
        P = case["batch"] * case["width"] * case["height"]
        if kind == "network":
            return {"bytes": P * (16 + 4) + 4 * NUM_PARAMS, "flops": _network_flops(P)}
        # parameters and both moments in and out, the gradient out; forward, data and weight gradients
        return {"bytes": P * (16 + 4) + 7 * 4 * NUM_PARAMS, "flops": 3 * _network_flops(P)}
    T, V = _triangles(case), _vertices(case)
    # positions, normals, tangents, texture coordinates and three index triples, once
    scene = V * (12 + 12 + 12 + 8) + T * 36
    S = case["shadow_size"] ** 2 if case["shadow_size"] else case["width"] * case["height"]
    if kind == "files":
        P = case["width"] * case["height"]
        # the frame, shadow map, depth, AO and G-buffer fields in, about a byte of file per sample out
        return {"bytes": P * (4 + 4 + (4 + 5 * 12 if case["deferred"] else 0)) + 4 * S + 12 * P + S, "flops": 0}
    taps = {0: 1, 1: case["pcf"], 2: case["pcf"] + case["blocker"]}[case["shadow"]]
    if kind == "batch":
        P = sum(w * h for w, h in _view_sizes(case))
        texels = min(ASSETS[case["assets"]][5], 8 * P)
        return {"bytes": scene + texels + 3 * P,
                "flops": P * (30 * case["ssao"] + case["lights"] * (15 * taps + 150) + 200) +
                (V * 60 + T * 60) * (case["views"] + case["lights"])}
    k = case.get("ssaa", 0) or 1
    P = case["width"] * case["height"] * k * k
    texels = min(ASSETS[case["assets"]][5], 8 * P)
    ao = 0 if not case["deferred"] else 30 * case["ssao"] if case["ao"] == "ssao" else \
        30 * INPUT_SAMPLES + _network_flops(P) // P
    return {"bytes": scene + texels + 3 * case["width"] * case["height"],
            "flops": P * (ao + 15 * taps + 350) + (V * 60 + T * 60) * 2}


# ---- the network in 64 bits ---------------------------------------------------------


def _up4(x):
    return torch.nn.functional.interpolate(x, scale_factor=4, mode="bilinear", align_corners=False)


def _forward64(p, x):
    """The U-Net on (B, 4, H, W) in 64 bits; its 3x3 weights are BF16 numbers."""
    conv, at = [], 0
    for ci, co, _ in LAYERS:
        w = p[at:at + ci * co * 9].view(co, ci, 3, 3)
        conv.append((w + (w.detach().to(torch.bfloat16).double() - w.detach()), p[at + ci * co * 9:at + ci * co * 9 + co]))
        at += ci * co * 9 + co
    head, bias = p[at:at + 64].view(4, 16, 1, 1), p[at + 64:]

    def layer(i, v):
        return torch.relu(torch.nn.functional.conv2d(v, conv[i][0], conv[i][1], padding=1))

    # space to depth: channel 8 r + 4 c + k of a block is channel k of its pixel (r, c)
    x = torch.cat([x[:, :, r::2, c::2] for r in range(2) for c in range(2)], 1)
    s0 = layer(1, layer(0, x))
    s1 = layer(3, layer(2, torch.nn.functional.avg_pool2d(s0, 4)))
    b = layer(5, layer(4, torch.nn.functional.avg_pool2d(s1, 4)))
    d1 = layer(7, layer(6, torch.cat([_up4(b), s1], 1)))
    d0 = layer(9, layer(8, torch.cat([_up4(d1), s0], 1)))
    return torch.pixel_shuffle(torch.sigmoid(torch.nn.functional.conv2d(d0, head, bias)), 2)[:, 0]


def exact(case, seed):
    if case["kind"] not in ("network", "train"):
        return None  # pictures and files: whole numbers
    x, label = _views(case, seed)
    p = torch.from_numpy(np.fromfile(WEIGHTS, "<f4")).double().cuda()
    if case["kind"] == "network":
        with torch.no_grad():
            return _forward64(p, x.double())
    p.requires_grad_(True)
    ao = _forward64(p, x.double())
    diff = torch.where(label >= 0, ao - label.double(), torch.zeros_like(ao))
    loss = diff.square().sum() / diff.numel()
    loss.backward()
    return {"loss": float(loss.detach()), "grads": p.grad.cpu().numpy()}
