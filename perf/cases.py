"""The work that users of this package have it do, as cases that can be timed.

A case is a dict of plain values. Kinds:

* frame   one frame of the path tracer: (bake a slice of the probe grid) -> (move the instances)
          -> rt pass -> reproject pass -> compose pass -> history hand-over -> (output stage), through
          PathTracingRenderer, on a camera that orbits by half a degree per frame;
* rays    a ray-query call on device buffers (line of sight, picking, baking tools);
* unet    the learned denoiser's forward on a batch of 1-spp inputs;
* train   steps of the denoiser's training, then the new weights read back;
* adjoint a step of a material fit: differentiable render, image loss, gradients;
* conv    one 3 x 3 convolution of the denoiser, with bias and ReLU;
* wgrad   that convolution's weight gradient.

listed() holds the sizes of the package's own scenes and training runs, draw() more of the same ranges.
"""
import ctypes
import math

import numpy as np
import torch

from gknextengine_gb300 import abi, autograd, camera, denoiser, native, scenes
from gknextengine_gb300.renderer import PathTracingRenderer

FRAMES = 16          # frames a state holds; the camera swings forth and back over them
CITY_FRAMES = 4      # instance tables a moving scene's state holds


def listed():
    return [
        # the smallest frame: the Cornell box at 256 x 256, where launches and latency count
        frame("frame-cornell-256", "cornell", 256, 256, bounces=4),
        # the headline: a million triangles at 1080p, TAA, a-trous denoising
        frame("frame-bricks-1080p", "bricks", 1920, 1080, bounces=8, taa=True, denoiser=abi.DENOISE_ATROUS),
        # the largest: ten million triangles at 4K, spheres that move, emissive-triangle lights
        frame("frame-city-4k", "city", 3840, 2160, bounces=8, taa=True, nee=abi.NEE_EMISSIVE),
        # an editor's viewport of an odd size at the reference's own settings (8 samples, 5 bounces),
        # textured, under an HDR sky and a sun, upscaled for presentation
        frame("frame-textured-odd", "textured", 1277, 713, samples=8, bounces=5, taa=True, sun=True,
              present_width=1920, present_height=1072),
        # a game's frame on the probe grid: a slice of probes baked, paths ending at their first bounce
        frame("frame-probes-720p", "yard", 1280, 720, bounces=4, taa=True, sun=True, probes=True, fast_gather=True),
        # line-of-sight queries of an offline tool: two million incoherent rays
        {"name": "rays-city-2m", "kind": "rays", "scene": "city", "count": 2097143, "any": False},
        # picking and gameplay queries: a thousand rays
        {"name": "rays-cornell-1k", "kind": "rays", "scene": "cornell", "count": 1000, "any": False},
        # the denoiser on a 1080p frame
        {"name": "unet-1080p", "kind": "unet", "batch": 1, "height": 1080, "width": 1920},
        # its training on batches of 8 crops of 256 x 256
        {"name": "train-8x256", "kind": "train", "batch": 8, "height": 256, "width": 256, "steps": 2},
        # the fit of 256 materials at 512 x 512 and 16 samples per pixel
        {"name": "adjoint-512", "kind": "adjoint", "height": 512, "width": 512, "spp": 16, "bounces": 4},
        # a half-resolution layer of the denoiser on an odd image, and a wide layer's weight gradient
        {"name": "conv-64-odd", "kind": "conv", "batch": 1, "height": 539, "width": 963, "cin": 64, "cout": 64},
        {"name": "wgrad-96-32", "kind": "wgrad", "batch": 2, "height": 509, "width": 517, "cin": 96, "cout": 32},
    ]


def frame(name, scene, width, height, samples=1, bounces=4, taa=False, denoiser=abi.DENOISE_JBF,
          nee=abi.NEE_REFERENCE, sun=False, probes=False, fast_gather=False, present_width=0, present_height=0):
    return {"name": name, "kind": "frame", "scene": scene, "width": width, "height": height, "samples": samples,
            "bounces": bounces, "taa": taa, "denoiser": denoiser, "nee": nee, "sun": sun, "probes": probes,
            "fast_gather": fast_gather, "present_width": present_width, "present_height": present_height}


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["frame"] * 5 + ["rays"] * 2 + ["unet", "train", "adjoint", "conv", "wgrad"])
    if kind == "frame":
        scene = rng.choice(["cornell", "bricks", "city", "textured", "yard"])
        width = spread(96, 3840)
        height = max(64, min(2160, int(width * rng.uniform(0.5, 1.0))))
        samples = 1 if scene == "city" else rng.choice([s for s in (1, 2, 4, 8) if s * width * height <= 8000000])
        c = frame("", scene, width, height, samples=samples, bounces=rng.randint(2, 8), taa=rng.random() < 0.7,
                  denoiser=rng.choice([abi.DENOISE_JBF, abi.DENOISE_ATROUS]),
                  nee=abi.NEE_EMISSIVE if scene == "city" else rng.choice([abi.NEE_REFERENCE, abi.NEE_EMISSIVE]),
                  sun=rng.random() < 0.5, probes=scene == "yard", fast_gather=scene == "yard" and rng.random() < 0.5)
        if rng.random() < 0.4:
            c["present_width"], c["present_height"] = (width * 3 // 2, height * 3 // 2)
    elif kind == "rays":
        c = {"kind": kind, "scene": rng.choice(["cornell", "bricks", "city"]), "count": spread(64, 4000000) | 1,
             "any": rng.random() < 0.5}
    elif kind == "unet":
        c = {"kind": kind, "batch": rng.randint(1, 2), "height": 8 * spread(2, 135), "width": 8 * spread(2, 240)}
    elif kind == "train":
        c = {"kind": kind, "batch": rng.randint(1, 8), "height": 8 * spread(4, 40), "width": 8 * spread(4, 40),
             "steps": rng.randint(1, 2)}
    elif kind == "adjoint":
        c = {"kind": kind, "height": spread(48, 512), "width": spread(48, 512), "spp": rng.randint(1, 16),
             "bounces": rng.randint(2, 6)}
    elif kind == "conv":
        c = {"kind": kind, "batch": rng.randint(1, 2), "height": spread(16, 700), "width": spread(16, 1000),
             "cin": 32 * rng.randint(1, 5), "cout": 32 * rng.randint(1, 4)}
    else:
        c = {"kind": kind, "batch": rng.randint(1, 4), "height": spread(16, 512), "width": spread(16, 512),
             "cin": 32 * rng.randint(1, 5), "cout": 32 * rng.randint(1, 4)}
    c.pop("name", None)
    return c


# ---- scenes ----

def yard(seed):
    """A field of 16 x 16 bricks around the origin, inside the probe grid, under a sky."""
    sc, _, st = scenes.bricks(seed, grid=16, emissive=16)
    inst = sc.instances.copy()
    for axis, shift in ((3, -17.6), (11, -9.6)):      # the bricks are scaled along y only
        inst["world"][:, axis] += np.float32(shift)
        inst["world_inv"][:, axis] = -inst["world"][:, axis]
    sc = abi.SceneArrays(sc.positions, sc.normals, sc.material_slots, sc.indices, sc.meshes, sc.materials, inst,
                         name="yard")
    st.has_sky, st.sky_color = True, (0.5, 0.7, 1.0, 1.0)
    return sc, camera.Camera(eye=(0.0, 9.0, 22.0), center=(0.0, 2.0, 0.0), fov_deg=40.0), st


def make_scene(name, seed):
    """(SceneArrays, Camera, Settings, CityMotion or None)"""
    if name == "city":
        return scenes.city(seed)
    made = {"cornell": scenes.cornell, "bricks": scenes.bricks, "textured": scenes.cornell_textured, "yard": yard}
    return made[name](seed) + (None,)


# Ray origins of the ray-query cases: a box inside each scene.
RAY_BOX = {"cornell": ((-0.49, 0.01, -0.49), (0.49, 0.99, 0.49)), "bricks": ((0.0, 0.0, 0.0), (140.0, 12.0, 76.0)),
           "city": ((0.0, 0.5, 0.0), (850.0, 160.0, 850.0))}


def generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


# ---- device images as tensors ----

class Views:
    """Tensors over a renderer's device images, made once per image buffer (history buffers swap)."""

    def __init__(self, renderer):
        self.r = renderer
        self.made = {}

    def __call__(self, image_id):
        v = self.r.image_view(image_id)
        key = (image_id, v.device_ptr)
        if key not in self.made:
            dt, ch = abi.IMAGE_FORMATS[image_id]
            words = device_tensor(self.r, v.device_ptr, v.height * (v.pitch_bytes // 4),
                                  "<f4" if dt == np.float32 else "<i4")
            t = words.view(v.height, v.pitch_bytes // (4 * ch), ch)[:, :v.width]
            self.made[key] = t
        return self.made[key]


def device_tensor(renderer, ptr, words, typestr):
    """A tensor over a buffer of the renderer's; it keeps the renderer, which owns the buffer, alive."""
    class A:
        __cuda_array_interface__ = {"shape": (words,), "typestr": typestr, "data": (ptr, False), "version": 3}

    a = A()
    a.owner = renderer
    return torch.as_tensor(a, device="cuda")


# ---- preparation: what a program has in hand before the call ----

def prepare(case, seed):
    return {"frame": prepare_frame, "rays": prepare_rays, "unet": prepare_unet, "train": prepare_train,
            "adjoint": prepare_adjoint, "conv": prepare_conv, "wgrad": prepare_wgrad}[case["kind"]](case, seed)


def prepare_frame(case, seed):
    sc, cam, st, motion = make_scene(case["scene"], seed)
    W, H = case["width"], case["height"]
    st.samples, st.bounces, st.taa = case["samples"], case["bounces"], case["taa"]
    st.max_bounces = max(st.max_bounces, st.bounces)
    st.denoiser, st.nee_mode, st.fast_gather = case["denoiser"], case["nee"], case["fast_gather"]
    if case["sun"]:
        st.has_sun, st.sun_intensity, st.sun_direction = True, 2.0, (0.3, 0.8, 0.5)
    start = float(np.random.default_rng(seed).uniform(-10.0, 10.0))
    fb = camera.FrameBuilder(W, H, st)
    frames = []
    for k in range(FRAMES + 1):
        swing = k % FRAMES
        frames.append(fb.build(cam.orbit(start + 0.5 * min(swing, FRAMES - swing)), k + 1))
    r = PathTracingRenderer(0)
    r.load_scene(sc)
    r.create_swap_chain(W, H)
    if case["present_width"]:
        r.output_resize(case["present_width"], case["present_height"])
    if case["probes"]:
        r.probe_voxelize()
    tables = [motion.instances(k + 1) for k in range(CITY_FRAMES)] if motion is not None else None
    return {"case": case, "r": r, "views": Views(r), "frames": frames[1:], "tables": tables, "next": 0}


def prepare_rays(case, seed):
    sc = make_scene(case["scene"], seed)[0]
    r = PathTracingRenderer(0)
    r.load_scene(sc)
    rays = random_rays(case, seed)
    hits = torch.empty((case["count"], 8), dtype=torch.float32, device="cuda")
    return {"case": case, "r": r, "rays": rays, "hits": hits}


def random_rays(case, seed):
    g = generator(seed)
    n = case["count"]
    lo, hi = (torch.tensor(v, device="cuda") for v in RAY_BOX[case["scene"]])
    rays = torch.empty((n, 8), dtype=torch.float32, device="cuda")
    rays[:, 0:3] = lo + (hi - lo) * torch.rand((n, 3), device="cuda", generator=g)
    rays[:, 3] = 1e-3
    d = torch.randn((n, 3), device="cuda", generator=g)
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    rays[:, 7] = 1000.0
    return rays


def network_input(case, seed):
    """1-spp radiance (a few bright samples on a dark image), albedo, normal and depth of smooth surfaces."""
    g = generator(seed)
    B, H, W = case["batch"], case["height"], case["width"]
    x = torch.empty((B, H, W, 10), dtype=torch.float32, device="cuda")
    yy = torch.linspace(0.0, 9.0, H, device="cuda")[:, None]
    xx = torch.linspace(0.0, 16.0, W, device="cuda")[None, :]
    phase = 6.0 * torch.rand((B, 10, 1, 1), device="cuda", generator=g)
    wave = torch.sin(xx + phase) * torch.cos(yy - phase)                                  # (B, 10, H, W)
    smooth = wave.permute(0, 2, 3, 1)
    lit = torch.rand((B, H, W, 3), device="cuda", generator=g)
    x[..., 0:3] = torch.where(lit > 0.9, 8.0 * lit, 0.3 * lit) * (0.6 + 0.4 * smooth[..., 0:3])
    x[..., 3:6] = 0.55 + 0.35 * smooth[..., 3:6]
    n = smooth[..., 6:9] + 0.01
    x[..., 6:9] = n / n.norm(dim=-1, keepdim=True)
    x[..., 9] = 0.9 + 0.09 * smooth[..., 9]
    target = (0.4 * (1.0 + smooth[..., 0:3])).contiguous()
    return x, target


def prepare_unet(case, seed):
    r = PathTracingRenderer(0)
    net = denoiser.load_c5(r)
    x, _ = network_input(case, seed)
    shape = (case["batch"], case["height"], case["width"], 4)
    return {"case": case, "net": net, "x": x, "linear": torch.empty(shape, device="cuda"),
            "raw": torch.empty(shape, device="cuda")}


def prepare_train(case, seed):
    r = PathTracingRenderer(0)
    net = denoiser.load_c5(r)
    batches = [network_input(case, seed * 16 + k) for k in range(case["steps"])]
    return {"case": case, "net": net, "batches": batches}


def prepare_adjoint(case, seed):
    sc, cam, st = scenes.cornell_materials(seed)
    st.bounces = st.max_bounces = case["bounces"]
    W, H = case["width"], case["height"]
    r = PathTracingRenderer(0)
    r.load_scene(sc)
    r.create_swap_chain(W, H)
    fc = camera.FrameBuilder(W, H, st).build(cam, 1 + seed % 1000)
    n = 256
    albedo = torch.as_tensor(sc.materials["diffuse"][:n, :3].copy(), device="cuda").requires_grad_()
    rough = torch.as_tensor(sc.materials["fuzziness"][:n].copy(), device="cuda").requires_grad_()
    target = torch.rand((H, W, 3), device="cuda", generator=generator(seed))
    return {"case": case, "r": r, "fc": fc, "albedo": albedo, "rough": rough, "target": target}


def prepare_conv(case, seed):
    g = generator(seed)
    B, H, W, ci, co = (case[k] for k in ("batch", "height", "width", "cin", "cout"))
    x = torch.relu(torch.randn((B, H, W, ci), device="cuda", generator=g)).bfloat16()
    w = (torch.randn((co, 3, 3, ci), device="cuda", generator=g) * math.sqrt(2.0 / (9 * ci))).bfloat16()
    bias = 0.1 * torch.randn((co,), device="cuda", generator=g)
    return {"case": case, "lib": native.load(), "x": x, "w": w, "bias": bias,
            "y": torch.empty((B, H, W, co), dtype=torch.bfloat16, device="cuda")}


def prepare_wgrad(case, seed):
    g = generator(seed)
    B, H, W, ci, co = (case[k] for k in ("batch", "height", "width", "cin", "cout"))
    x = torch.relu(torch.randn((B, H, W, ci), device="cuda", generator=g)).bfloat16()
    dy = torch.randn((B, H, W, co), device="cuda", generator=g).bfloat16()
    return {"case": case, "lib": native.load(), "x": x, "dy": dy,
            "dw": torch.zeros((co, 3, 3, ci), dtype=torch.float32, device="cuda")}


# ---- one pass ----

def run(state):
    return {"frame": run_frame, "rays": run_rays, "unet": run_unet, "train": run_train, "adjoint": run_adjoint,
            "conv": run_conv, "wgrad": run_wgrad}[state["case"]["kind"]](state)


def run_frame(s):
    case, r, view = s["case"], s["r"], s["views"]
    k = s["next"]
    s["next"] = k + 1
    fc = s["frames"][k % FRAMES]
    if case["probes"]:
        r.probe_bake_slice(fc, k + 4)      # the slices just above the ground come first
    if s["tables"] is not None:
        r.update_instances(s["tables"][k % CITY_FRAMES])
    r.render(fc)
    out = {"denoised": view(abi.IMG_DENOISED), "linear": view(abi.IMG_DENOISED_LINEAR),
           "history": [view(i) for i in (abi.IMG_PREV_DIFFUSE, abi.IMG_PREV_SPECULAR, abi.IMG_PREV_ALBEDO)],
           "ids": view(abi.IMG_OBJECT_ID_PREV), "normal": view(abi.IMG_NORMAL), "motion": view(abi.IMG_MOTION)}
    if case["present_width"]:
        r.output_pass(abi.OUTPUT_FSR)
        if "present" not in s:
            v = abi.GkrtImageView()
            r._check(r._lib.gkrt_get_output(r._h, ctypes.byref(v)))
            s["present"] = device_tensor(r, v.device_ptr, v.width * v.height, "<i4")
        out["present"] = s["present"]
    return out


def run_rays(s):
    rays, hits = s["rays"], s["hits"]
    s["r"].trace_rays_device(rays.data_ptr(), hits.data_ptr(), rays.shape[0],
                             abi.TRACE_ANY if s["case"]["any"] else abi.TRACE_CLOSEST)
    ids = hits.view(torch.int32)[:, 3:5]
    if s["case"]["any"]:
        return {"occluded": ids[:, 0] >= 0}   # any-hit: which triangle was met is not part of the answer
    return {"t": hits[:, 0], "b": hits[:, 1:3], "ids": ids}


def run_unet(s):
    s["net"].forward(s["x"], s["linear"], s["raw"])
    return {"linear": s["linear"], "raw": s["raw"][..., :3]}


def run_train(s):
    losses = [s["net"].train_step(x, target, 5e-5) for x, target in s["batches"]]
    return {"loss": losses, "weights": s["net"].params()}


def run_adjoint(s):
    s["albedo"].grad = s["rough"].grad = None
    img = autograd.render_materials(s["r"], s["fc"], s["case"]["spp"], s["albedo"], s["rough"])
    loss = ((img - s["target"]) ** 2).mean()
    loss.backward()
    return {"image": img.detach(), "albedo": s["albedo"].grad, "rough": s["rough"].grad}


def check(rc):
    if rc != abi.GKRT_OK:
        raise native.GkrtError(rc, "convolution")


def run_conv(s):
    c = s["case"]
    check(s["lib"].gkrt_conv3x3_bf16(s["x"].data_ptr(), c["batch"], c["height"], c["width"], c["cin"],
                                     s["w"].data_ptr(), s["bias"].data_ptr(), c["cout"], s["y"].data_ptr(), c["cout"],
                                     0, c["cout"], 1, None))
    return s["y"]


def run_wgrad(s):
    c = s["case"]
    s["dw"].zero_()
    check(s["lib"].gkrt_conv3x3_wgrad_bf16(s["dy"].data_ptr(), s["x"].data_ptr(), c["batch"], c["height"], c["width"],
                                           c["cin"], c["cout"], s["dw"].data_ptr(), None))
    return s["dw"]


# ---- what a pass cannot do without ----

# Multiply-adds per pixel of the network's convolutions, over the resolutions' pixel shares.
UNET_MACS = 9 * (16 * 32 + 32 * 32 + 96 * 32 + 32 * 32 + 32 * 4
                 + (32 * 64 + 64 * 64 + 160 * 64 + 64 * 64) / 4
                 + (64 * 96 + 96 * 96 + 224 * 96 + 96 * 96) / 16
                 + (96 * 128 + 128 * 128) / 64)
UNET_PARAMS = 952_000

# Triangles a scene's instances stand for, and of its distinct meshes.
TRIANGLES = {"cornell": (36, 36), "textured": (36, 36), "yard": (64_514, 254), "bricks": (1_032_194, 254),
             "city": (10_480_002, 2062)}
RAY_FLOPS = 18      # two slab tests per tree level and axis, six flops each
TRI_FLOPS = 50      # one ray / triangle test


def ray_flops(scene):
    return RAY_FLOPS * math.log2(TRIANGLES[scene][0]) + TRI_FLOPS


def work(case):
    k = case["kind"]
    if k == "frame":
        px = case["width"] * case["height"]
        # history in and out (three colours), ids in and out, normals and motion out, two final images
        nbytes = px * (2 * 3 * 16 + 2 * 4 + 16 + 8 + 2 * 16) + 4 * case["present_width"] * case["present_height"]
        nbytes += 48 * TRIANGLES[case["scene"]][1] + (25_001 * 224 if case["scene"] == "city" else 0)
        rays = px * (1 + 2 * case["samples"])
        if case["probes"]:
            rays += 14_720 * 6 * 16 // 8
        return {"bytes": nbytes, "flops": rays * ray_flops(case["scene"])}
    if k == "rays":
        return {"bytes": 64 * case["count"] + 48 * TRIANGLES[case["scene"]][1],
                "flops": case["count"] * ray_flops(case["scene"])}
    if k in ("unet", "train"):
        px = case["batch"] * case["height"] * case["width"]
        if k == "unet":
            return {"bytes": px * (40 + 32) + 2 * UNET_PARAMS, "flops": 2 * UNET_MACS * px}
        return {"bytes": case["steps"] * (px * 52 + 7 * 4 * UNET_PARAMS), "flops": case["steps"] * 3 * 2 * UNET_MACS * px}
    if k == "adjoint":
        px = case["height"] * case["width"]
        rays = 2 * px * (1 + 2 * case["spp"])
        return {"bytes": px * (16 + 12 + 12 + 16), "flops": rays * (RAY_FLOPS * math.log2(5000) + TRI_FLOPS)}
    px = case["batch"] * case["height"] * case["width"]
    weights = 9 * case["cin"] * case["cout"]
    return {"bytes": 2 * px * (case["cin"] + case["cout"]) + (2 if k == "conv" else 4) * weights,
            "flops": 2 * weights * px}


# ---- the same answers in 64 bits, for the cases whose outputs are sums that can be written down ----

def exact(case, seed):
    if case["kind"] == "conv":
        s = prepare_conv(case, seed)
        y = torch.nn.functional.conv2d(s["x"].double().permute(0, 3, 1, 2), s["w"].double().permute(0, 3, 1, 2),
                                       s["bias"].double(), padding=1)
        return torch.relu(y).permute(0, 2, 3, 1)
    if case["kind"] == "wgrad":
        s = prepare_wgrad(case, seed)
        x = s["x"].double().permute(0, 3, 1, 2)
        dw = torch.nn.grad.conv2d_weight(x, (case["cout"], case["cin"], 3, 3), s["dy"].double().permute(0, 3, 1, 2),
                                         padding=1)
        return dw.permute(0, 2, 3, 1)
    if case["kind"] == "rays" and case["scene"] == "cornell" and not case["any"]:
        return exact_rays(case, seed)
    return None


def exact_rays(case, seed):
    """Closest hits over every triangle of the scene: t, and the barycentrics of vertices 1 and 2."""
    sc = scenes.cornell(seed)[0]
    tris = []
    for inst in sc.instances:
        m = sc.meshes[inst["mesh_id"]]
        idx = sc.indices[m["index_offset"]:m["index_offset"] + m["index_count"]].astype(np.int64) + int(m["vertex_offset"])
        p = sc.positions[idx, :3].astype(np.float64)
        w = np.linalg.inv(np.vstack([inst["world_inv"].astype(np.float64).reshape(3, 4), [0.0, 0.0, 0.0, 1.0]]))
        tris.append((p @ w[:3, :3].T + w[:3, 3]).reshape(-1, 3, 3))
    tri = torch.as_tensor(np.concatenate(tris), device="cuda")
    e1, e2, v0 = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0], tri[:, 0]
    rays = random_rays(case, seed).double()
    out_t, out_b = [], []
    for part in rays.split(65536):
        o, d = part[:, None, 0:3], part[:, None, 4:7]
        p = torch.cross(d.expand(-1, tri.shape[0], -1), e2[None].expand(part.shape[0], -1, -1), dim=-1)
        det = (p * e1).sum(-1)
        t0 = o - v0
        b1 = (t0 * p).sum(-1) / det
        q = torch.cross(t0, e1[None].expand_as(t0), dim=-1)
        b2 = (d * q).sum(-1) / det
        t = (e2 * q).sum(-1) / det
        ok = (det != 0) & (b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (t >= part[:, None, 3]) & (t <= part[:, None, 7])
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        best, at = t.min(dim=1)
        hit = torch.isfinite(best)
        pick = torch.stack([b1.gather(1, at[:, None])[:, 0], b2.gather(1, at[:, None])[:, 0]], 1)
        out_t.append(torch.where(hit, best, torch.full_like(best, -1.0)))
        out_b.append(torch.where(hit[:, None], pick, torch.zeros_like(pick)))
    return {"t": torch.cat(out_t), "b": torch.cat(out_b), "ids": None}
