"""What a user of this framework has it do, as cases that can be timed.

A program of this framework loads a scene (upload, acceleration structure),
renders it (a preview of a few samples, a progressive chunk, a final image),
denoises a low-sample render, renders many small jobs as one batch, or trains
the denoiser.  Every case goes through `pt_gb300.Context`, `pt_gb300.HostScene`
or `pt_gb300.denoise.UNet`, with host buffers where a program has host
buffers: scenes come from host memory and images go back to it (into pinned
memory that the program keeps).

Scenes are the distributions of pt_gb300.scenes, generated from the seed as raw
arrays: `small` (a ground quad, icospheres and one light), `mid` (displaced
grids, icospheres and some hundred rotated boxes, 32 emitters, thin lens),
`heavy` (displaced grids and spheres in up to 10,000 rotated instances, a tenth
of them transmissive, 256 emitters), `textured` (every texture path) and
`glass` (refractive dielectrics).
"""
import math

import numpy as np
import torch

import pt_gb300 as P
from pt_gb300 import abi, scenes
from pt_gb300.denoise import WEIGHTS_DIR, UNet

# ---------------------------------------------------------------- cases


def listed():
    return [
        # a thumbnail while a scene is being set up: one sample, tone-mapped; launches and latency
        {"name": "preview_160x120", "kind": "render", "scene": "small", "detail": 8, "width": 160, "height": 120, "spp": 1,
         "bounces": 8, "rr_start": 1, "fp64": False, "tonemap": True},
        # the small configuration of the benchmark: a quick look at a simple scene
        {"name": "small_256", "kind": "render", "scene": "small", "detail": 8, "width": 256, "height": 256, "spp": 16,
         "bounces": 8, "rr_start": 1, "fp64": False, "tonemap": False},
        # an odd-sized frame of a fully textured scene with FP64 sums (a chunk of a reference image)
        {"name": "textured_333x217_fp64", "kind": "render", "scene": "textured", "detail": 0, "width": 333, "height": 217,
         "spp": 9, "bounces": 6, "rr_start": 1, "fp64": True, "tonemap": False},
        # one step of a progressive view of an ordinary scene at a common window size
        {"name": "mid_1280x720_2spp", "kind": "render", "scene": "mid", "detail": 196, "width": 1280, "height": 720, "spp": 2,
         "bounces": 8, "rr_start": 1, "fp64": False, "tonemap": False},
        # the benchmark's image: a final frame
        {"name": "mid_1024_128spp", "kind": "render", "scene": "mid", "detail": 196, "width": 1024, "height": 1024, "spp": 128,
         "bounces": 8, "rr_start": 1, "fp64": False, "tonemap": False},
        # a full-HD chunk of the heavy configuration: two million triangles, ten thousand instances
        {"name": "heavy_1920x1080_4spp", "kind": "render", "scene": "heavy", "detail": 10000, "width": 1920, "height": 1080,
         "spp": 4, "bounces": 12, "rr_start": 4, "fp64": False, "tonemap": False},
        # a new ordinary scene: upload, acceleration structure, first preview
        {"name": "load_mid", "kind": "load", "scene": "mid", "detail": 196, "width": 320, "height": 240, "spp": 1, "bounces": 8,
         "rr_start": 1},
        # a new large scene
        {"name": "load_heavy", "kind": "load", "scene": "heavy", "detail": 10000, "width": 320, "height": 240, "spp": 1,
         "bounces": 12, "rr_start": 4},
        # a denoised frame: few samples with features and the noise estimate, then the network
        {"name": "denoised_mid_1024_3spp", "kind": "denoise", "scene": "mid", "detail": 196, "width": 1024, "height": 1024,
         "spp": 3, "bounces": 8, "rr_start": 1},
        # a render farm's queue of small jobs as one batch
        {"name": "batch_16_jobs", "kind": "batch", "jobs": 16, "side_lo": 128, "side_hi": 256, "spp_lo": 4, "spp_hi": 16,
         "tris_lo": 1000, "tris_hi": 50000, "bounces": 8},
        # the denoiser network alone on a full-HD frame (a program with its own feature buffers)
        {"name": "unet_forward_1080x1920", "kind": "unet_forward", "batch": 1, "height": 1080, "width": 1920},
        # the denoiser's training at its shipped recipe: loss and gradients of one batch
        {"name": "unet_gradients_16x256x256", "kind": "unet_gradients", "batch": 16, "height": 256, "width": 256},
    ]


def _logu(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


# paths (width x height x samples) of one pass at most, per scene: a drawn pass costs less than the largest listed one
_MOST_PATHS = {"small": 1 << 24, "mid": 1 << 26, "heavy": 1920 * 1080 * 4, "textured": 1 << 23, "glass": 1 << 23}


def _draw_render(rng):
    scene = rng.choice(["small", "mid", "mid", "heavy", "textured", "glass"])
    most = _MOST_PATHS[scene]
    width = int(_logu(rng, 64, 1920))
    height = max(48, min(1080, int(width * rng.uniform(0.5, 1.1))))
    spp = max(1, int(_logu(rng, 1, 128)))
    spp = max(1, min(spp, most // (width * height)))
    detail = {"small": lambda: rng.randint(3, 16), "mid": lambda: int(_logu(rng, 40, 400)),
              "heavy": lambda: int(_logu(rng, 500, 10000))}.get(scene, lambda: 0)()
    heavy = scene == "heavy"
    return {"kind": "render", "scene": scene, "detail": detail, "width": width, "height": height, "spp": spp,
            "bounces": rng.randint(4, 12 if heavy else 8), "rr_start": rng.choice([1, 4]) if heavy else 1,
            "fp64": rng.random() < 0.25, "tonemap": rng.random() < 0.25}


def draw(rng):
    kind = rng.choice(["render", "render", "render", "render", "load", "denoise", "batch", "unet_forward", "unet_gradients"])
    if kind == "render":
        return _draw_render(rng)
    if kind == "load":
        scene = rng.choice(["small", "mid", "heavy", "textured"])
        detail = {"small": lambda: rng.randint(3, 16), "mid": lambda: int(_logu(rng, 40, 400)),
                  "heavy": lambda: int(_logu(rng, 500, 10000))}.get(scene, lambda: 0)()
        return {"kind": "load", "scene": scene, "detail": detail, "width": rng.randint(64, 400), "height": rng.randint(48, 300),
                "spp": rng.randint(1, 2), "bounces": rng.randint(4, 8), "rr_start": 1}
    if kind == "denoise":
        return {"kind": "denoise", "scene": rng.choice(["small", "mid"]), "detail": rng.randint(8, 196),
                "width": 8 * rng.randint(12, 160), "height": 8 * rng.randint(10, 120), "spp": rng.randint(2, 8), "bounces": 8,
                "rr_start": 1}
    if kind == "batch":
        lo, n = int(_logu(rng, 64, 200)), rng.randint(3, 16)
        return {"kind": "batch", "jobs": n, "side_lo": lo, "side_hi": rng.randint(lo + 8, 264), "spp_lo": rng.randint(1, 4),
                "spp_hi": rng.randint(5, 16), "tris_lo": 1000, "tris_hi": int(_logu(rng, 4000, 50000)), "bounces": rng.randint(4, 8)}
    if kind == "unet_forward":
        return {"kind": "unet_forward", "batch": rng.choice([1, 1, 2]), "height": 8 * int(_logu(rng, 6, 135)),
                "width": 8 * int(_logu(rng, 6, 120))}
    side = 8 * rng.randint(6, 32)
    return {"kind": "unet_gradients", "batch": rng.randint(1, 16), "height": side, "width": 8 * rng.randint(6, 32)}


# ---------------------------------------------------------------- scenes

_MESHES = {}


def _mesh(key, make):
    """Unit meshes that do not depend on the seed, made once per process."""
    if key not in _MESHES:
        _MESHES[key] = make()
    return _MESHES[key]


def _sphere(subdiv):
    return _mesh(("sphere", subdiv), lambda: scenes.icosphere(subdiv))


def _at(scale, pos, rot=None):
    M = np.eye(4)
    M[:3, :3] = (np.eye(3) if rot is None else rot) * scale
    M[:3, 3] = pos
    return M


def _rotations(rng, n):
    """n random rotations (axis uniform in a cube, angle U(1e-5, 2 pi)), [n, 3, 3]."""
    a = rng.uniform(-1, 1, (n, 3))
    a /= np.maximum(np.linalg.norm(a, axis=1, keepdims=True), 1e-9)
    ang = rng.uniform(1e-5, 2 * math.pi, n)
    c, s = np.cos(ang), np.sin(ang)
    K = np.zeros((n, 3, 3))
    K[:, 0, 1], K[:, 0, 2], K[:, 1, 2] = -a[:, 2], a[:, 1], -a[:, 0]
    K[:, 1, 0], K[:, 2, 0], K[:, 2, 1] = a[:, 2], -a[:, 1], a[:, 0]
    return np.eye(3) * c[:, None, None] + s[:, None, None] * K + (1 - c)[:, None, None] * a[:, :, None] * a[:, None, :]


def _material(rng, alpha=1.0):
    return scenes.material_row(rng.uniform(0.1, 0.9, 3), float(rng.uniform(0.05, 1.0)), 1.0 if rng.random() < 0.3 else 0.0,
                               alpha=alpha)


def _emitter(rng, centre, size):
    cx, cy, cz = centre
    tri = scenes.triangle((cx - size, cy, cz - size * 0.5), (cx, cy, cz + size), (cx + size, cy, cz - size * 0.5))
    return tri, scenes.material_row((0, 0, 0), 1.0, 0.0, float(math.exp(rng.uniform(0.0, math.log(100.0))))), [np.eye(4)]


def _camera(eye, target, fov, **more):
    eye, target = np.asarray(eye, np.float64), np.asarray(target, np.float64)
    return {"position": tuple(-eye), "lookdir": tuple(eye - target), "fov_degrees": fov, **more}


def _small(rng, spheres):
    ms = []
    for _ in range(spheres):
        s = rng.uniform(0.5, 1.5)
        ms.append(_at(s, (rng.uniform(-4, 4), s, rng.uniform(-4, 4))))
    meshes = [(scenes.quad(20.0, 0.0, False), scenes.material_row(rng.uniform(0.2, 0.8, 3), 1.0), [np.eye(4)]),
              (_sphere(3), scenes.material_row(rng.uniform(0.2, 0.8, 3), 1.0), ms),
              (scenes.quad(2.0, 6.0, True), scenes.material_row((0, 0, 0), 1.0, 0.0, 10.0), [np.eye(4)])]
    return scenes.assemble_raw(meshes, (0.115, 0.171, 0.787)), _camera((-1.0, 2.0, -3.0), (0.0, 0.75, 0.0), 60.0)


def _mid(rng, seed, boxes):
    srng = scenes.SceneRng(seed & 0x7FFFFFFF)
    kinds = [scenes.displaced_grid(64, srng), scenes.displaced_grid(64, srng), _sphere(4), _sphere(4),
             _mesh("box0", lambda: scenes.rounded_box(10, 0.15)), _mesh("box1", lambda: scenes.rounded_box(10, 0.3))]
    variants = [[(m, _material(rng), []) for _ in range(4)] for m in kinds]

    def put(kind, M):
        variants[kind][int(rng.integers(4))][2].append(M)

    for i in range(2):
        put(i, _at(10.0, (-10.0 + 20.0 * i, 0.0, 0.0)))
        s = rng.uniform(1.5, 3.0)
        put(2 + i, _at(s, (rng.uniform(-12, 12), s, rng.uniform(-4, 8))))
    for i, R in enumerate(_rotations(rng, boxes)):
        s = rng.uniform(0.3, 1.0)
        put(4 + i % 2, _at(s, (rng.uniform(-18, 18), s + rng.uniform(0.0, 1.5), rng.uniform(-8, 9)), R))
    meshes = [v for vs in variants for v in vs if v[2]]
    for _ in range(32):
        meshes.append(_emitter(rng, (rng.uniform(-16, 16), rng.uniform(6, 10), rng.uniform(-6, 10)), rng.uniform(0.6, 1.4)))
    return (scenes.assemble_raw(meshes, (0.033, 0.051, 0.133)),
            _camera((0.0, 5.0, -22.0), (0.0, 1.0, 0.0), 45.0, focus_dist=8.0, lens_radius=0.03))


def _heavy(rng, seed, instances):
    srng = scenes.SceneRng(seed & 0x7FFFFFFF)
    base = [scenes.displaced_grid(144, srng, amplitude=0.1) for _ in range(32)]
    p, n, uv, ix = _sphere(5)
    for _ in range(32):
        waves, ph = rng.uniform(1, 5, (3, 3)), rng.uniform(0, 6.283, 3)
        d = 1.0 + 0.06 * sum(np.sin(p @ waves[k] * 3.0 + ph[k]) for k in range(3))
        base.append(((p * d[:, None]).astype(np.float32), n, uv, ix))
    mats = [_material(rng, alpha=0.1 if rng.random() < 0.1 else 1.0) for _ in base]
    M = np.tile(np.eye(4), (instances, 1, 1))
    M[:, :3, :3] = _rotations(rng, instances) * rng.uniform(0.3, 2.5, instances)[:, None, None]
    M[:, :3, 3] = rng.uniform((-120, 0, -120), (120, 25, 120), (instances, 3))
    which = rng.integers(len(base), size=instances)
    meshes = [(m, mat, list(M[which == k])) for k, (m, mat) in enumerate(zip(base, mats)) if (which == k).any()]
    for _ in range(256):
        meshes.append(_emitter(rng, (rng.uniform(-110, 110), rng.uniform(30, 45), rng.uniform(-110, 110)), rng.uniform(1.0, 4.0)))
    return scenes.assemble_raw(meshes, (0.25, 0.3, 0.45)), _camera((0.0, 60.0, -170.0), (0.0, 5.0, 0.0), 50.0)


def _scene(case, seed):
    rng = np.random.default_rng([seed, 11])
    kind = case["scene"]
    if kind == "small":
        return _small(rng, case["detail"])
    if kind == "mid":
        return _mid(rng, seed, case["detail"])
    if kind == "heavy":
        return _heavy(rng, seed, case["detail"])
    if kind == "textured":
        return scenes.textured_raw(seed)
    raw, cam = scenes.glass_raw("glass")
    raw["materials"][:, :3] = np.where(raw["materials"][:, :3] > 0, rng.uniform(0.3, 1.0, raw["materials"][:, :3].shape), 0.0)
    return raw, cam


# ---------------------------------------------------------------- denoiser data

_LAYERS = [(16, 32), (32, 32), (32, 64), (64, 64), (64, 96), (96, 96), (96, 128), (128, 128), (224, 96), (96, 96), (160, 64),
           (64, 64), (96, 32), (32, 32), (32, 16)]
_LEVEL = [0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0, 0]


def _weights():
    return np.fromfile(WEIGHTS_DIR / "unet.bin", dtype="<f4")


def _frames(case, seed):
    """A batch of low-sample frames as the denoiser reads them: network input
    [n, h, w, 16] (BF16), residual base and linear target [n, h, w, 4] (FP32)."""
    n, h, w = case["batch"], case["height"], case["width"]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def blobs(c, size):
        lo = torch.rand((n, c, h // size + 2, w // size + 2), generator=g, device="cuda")
        return torch.nn.functional.interpolate(lo, size=(h, w), mode="bilinear").permute(0, 2, 3, 1)

    target = torch.zeros((n, h, w, 4), device="cuda")
    target[..., :3] = torch.exp(4.0 * blobs(3, 32) - 2.5)
    noise = torch.randn((n, h, w, 3), generator=g, device="cuda")
    noisy = target[..., :3] * torch.exp(0.6 * noise)
    other = target[..., :3] * torch.exp(0.6 * torch.randn((n, h, w, 3), generator=g, device="cuda"))
    x = torch.zeros((n, h, w, 16), device="cuda")
    x[..., 0:3] = torch.log1p(noisy)
    x[..., 3:6] = blobs(3, 16)
    x[..., 6:9] = torch.nn.functional.normalize(blobs(3, 24) - 0.5, dim=-1)
    x[..., 9] = torch.log1p(20.0 * blobs(1, 32)[..., 0]) * 0.25
    x[..., 10] = 0.25
    d = 0.5 * (other - noisy)
    x[..., 11:14] = torch.sign(d) * torch.log1p(d.abs())
    x[..., 14] = 1.0
    base = torch.zeros((n, h, w, 4), device="cuda")
    base[..., :3] = x[..., 0:3]
    return x.to(torch.bfloat16), base, target


# ---------------------------------------------------------------- prepare, run


def _pinned(h, w, fp64=False):
    return torch.empty((h, w, 4), dtype=torch.float64 if fp64 else torch.float32, pin_memory=True).numpy()


def _context(hs):
    ctx = P.Context(0)
    ctx.upload(hs.pack())
    ctx.build_accel()
    return ctx


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("unet_forward", "unet_gradients"):
        net = UNet(case["batch"], case["height"], case["width"])
        net.set_params(_weights())
        x, base, target = _frames(case, seed)
        net.input_tensor().copy_(x)
        net.base_tensor().copy_(base)
        torch.cuda.synchronize()
        s.update(net=net, target=target, output=torch.empty(x.shape, dtype=torch.float32, device="cuda"))
        return s
    if kind == "batch":
        # the queue (sizes, samples) belongs to the case, the scenes to the seed
        rng = np.random.default_rng([case["jobs"], case["side_hi"], case["spp_hi"]])

        def logu(lo, hi):
            return math.exp(rng.uniform(math.log(lo), math.log(hi)))

        jobs = []
        for j in range(case["jobs"]):
            raw, cam = scenes.batch_scene(seed * 100 + j, int(logu(case["tris_lo"], case["tris_hi"])))
            hs = P.HostScene.from_raw(raw, cam)
            side = int(logu(case["side_lo"], case["side_hi"]))
            jobs.append((_context(hs), hs.render_params(side, side, int(round(logu(case["spp_lo"], case["spp_hi"]))), case["bounces"])))
        s.update(ctx=P.Context(0), jobs=jobs)
        return s
    raw, cam = _scene(case, seed)
    hs = P.HostScene.from_raw(raw, cam)
    w, h = case["width"], case["height"]
    params = hs.render_params(w, h, case["spp"], case["bounces"], rr_start=case["rr_start"],
                              accum_mode=abi.PT_ACCUM_FP32_FP64 if case.get("fp64") else abi.PT_ACCUM_FP32)
    s.update(hs=hs, params=params, out=_pinned(h, w))
    if kind == "load":
        s.update(ctx=P.Context(0), view=hs.pack())
        return s
    s.update(ctx=_context(hs))
    if kind == "denoise":
        net = UNet(1, h, w)
        net.set_params(_weights())
        s.update(net=net)
    elif case["fp64"]:
        s.update(out64=_pinned(h, w, True))
    s["tonemap"] = bool(case.get("tonemap"))
    return s


def run(s):
    kind = s["kind"]
    if kind == "render":
        ctx = s["ctx"]
        ctx.render(s["params"], stats=False)
        got = {}
        if "out64" in s:
            got["fp64"] = ctx.read_image(fp64=True, out=s["out64"])
        if s["tonemap"]:
            ctx.tonemap()
        got["image"] = ctx.read_image(out=s["out"])
        return got
    if kind == "load":
        ctx = s["ctx"]
        ctx.upload(s["view"])
        info = ctx.build_accel()
        ctx.render(s["params"], stats=False)
        return {"triangles": int(info.triangles), "meshes": int(info.blas_count), "image": ctx.read_image(out=s["out"])}
    if kind == "denoise":
        s["ctx"].render_denoised(s["net"], s["params"])
        return s["ctx"].read_denoised(out=s["out"])
    if kind == "batch":
        st = s["ctx"].render_batch(s["jobs"])
        return {"segments": int(st.segments), "shadow_rays": int(st.shadow_rays),
                "images": [s["ctx"].read_batch_image(j) for j in range(len(s["jobs"]))]}
    if kind == "unet_forward":
        s["net"].forward(s["output"].data_ptr())  # into the program's own buffer, which outlives the network
        return s["output"]
    s["net"].forward()
    loss = s["net"].backward(s["target"].data_ptr())
    return {"loss": loss, "gradients": s["net"].grads()}


# ---------------------------------------------------------------- work, exact

# Per scene: path segments per path and, per ray, box-pair tests and triangle
# tests of a binned-SAH BVH2 and shadow rays per segment (the benchmark's
# roofline constants for the three configurations).
_SEGMENTS = {"small": 3.2, "mid": 1.6, "heavy": 2.9, "textured": 3.0, "glass": 3.0}
_RAYS = {"small": (13.8, 6.1, 0.52), "mid": (27.2, 9.0, 0.23), "heavy": (70.7, 24.7, 0.34), "textured": (13.8, 6.1, 0.5),
         "glass": (13.8, 6.1, 0.5)}
_TRIS = {"small": 1284, "mid": 36000, "heavy": 1983000, "textured": 372, "glass": 3844}


def _net_flops(case):
    px = case["batch"] * case["height"] * case["width"]
    return sum(2.0 * 9 * ci * co * px / 4 ** lv for (ci, co), lv in zip(_LAYERS, _LEVEL))


def work(case):
    kind = case["kind"]
    if kind in ("unet_forward", "unet_gradients"):
        px = case["batch"] * case["height"] * case["width"]
        params = 4.0 * sum(9 * ci * co + co for ci, co in _LAYERS)
        if kind == "unet_forward":
            return {"bytes": px * (32 + 16 + 64) + params, "flops": _net_flops(case)}
        return {"bytes": px * (32 + 16 + 16) + 2 * params, "flops": 3 * _net_flops(case)}
    if kind == "batch":
        side, spp = math.sqrt(case["side_lo"] * case["side_hi"]), math.sqrt(case["spp_lo"] * case["spp_hi"])
        tris, scene, jobs = math.sqrt(case["tris_lo"] * case["tris_hi"]), "mid", case["jobs"]
        pixels, paths = side * side, side * side * spp
    else:
        scene, tris, jobs = case["scene"], _TRIS[case["scene"]], 1
        pixels, paths = case["width"] * case["height"], case["width"] * case["height"] * case["spp"]
    nodes, leaves, nee = _RAYS[scene]
    segs = paths * _SEGMENTS[scene]
    # a pair of slab tests 44 operations, a watertight triangle test 50, shading one segment 400
    flops = segs * ((1 + nee) * (44 * nodes + 50 * leaves) + 400)
    # the scene is read once (36 B of vertices, 12 B of indices a triangle), the image written once
    nbytes = tris * 48 + pixels * 16
    if kind == "denoise":
        flops += _net_flops({"batch": 1, "height": case["height"], "width": case["width"]})
    return {"bytes": jobs * nbytes, "flops": jobs * flops}


def _exact_net(x, base, params):
    """The network in FP64 (torch); x [n, h, w, 16] -> [n, h, w, 16]."""
    F = torch.nn.functional
    layers, off = [], 0
    for ci, co in _LAYERS:
        w = params[off:off + 9 * ci * co].view(3, 3, ci, co).permute(3, 2, 0, 1)
        off += 9 * ci * co
        layers.append((w, params[off:off + co]))
        off += co

    def conv(i, t):
        t = F.conv2d(t, layers[i][0], layers[i][1], padding=1)
        return t if i == len(_LAYERS) - 1 else F.relu(t)

    def up(t):
        return F.interpolate(t, scale_factor=2, mode="nearest")

    e0 = conv(1, conv(0, x.permute(0, 3, 1, 2)))
    e1 = conv(3, conv(2, F.avg_pool2d(e0, 2)))
    e2 = conv(5, conv(4, F.avg_pool2d(e1, 2)))
    b3 = conv(7, conv(6, F.avg_pool2d(e2, 2)))
    d2 = conv(9, conv(8, torch.cat([up(b3), e2], 1)))
    d1 = conv(11, conv(10, torch.cat([up(d2), e1], 1)))
    d0 = conv(13, conv(12, torch.cat([up(d1), e0], 1)))
    out = conv(14, d0).permute(0, 2, 3, 1)
    return torch.cat([out[..., :4] + base, out[..., 4:]], -1)


def exact(case, seed):
    # rendered images have no closed form: they are compared as they are
    if case["kind"] not in ("unet_forward", "unet_gradients"):
        return None
    x, base, target = (t.double() for t in _frames(case, seed))
    params = torch.from_numpy(_weights().astype(np.float64)).cuda()
    if case["kind"] == "unet_forward":
        with torch.no_grad():
            return _exact_net(x, base, params)
    params.requires_grad_(True)
    # frame by frame: the activations of the whole batch in 64 bits would not fit beside other states
    n = case["batch"]
    loss = 0.0
    for k in range(n):
        out = _exact_net(x[k:k + 1], base[k:k + 1], params)
        t = target[k:k + 1, ..., :3].clamp(min=0)
        part = ((1 + t.clamp(max=16.0)) ** 2 * (out[..., :3] - torch.log1p(t)) ** 2).sum() / target[..., :3].numel()
        part.backward()
        loss += float(part.detach())
    return {"loss": loss, "gradients": params.grad}
