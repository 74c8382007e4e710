"""The work a user of this library has it do, as cases to be timed.

Each case is one pass through public entry points (the `lumina` package and
the C ABI it declares): building a BVH, loading a scene and rendering its
first frame, rendering frames of a resident scene, batches of camera poses,
denoising frames on the device or from host images, and the gradients of a
training step.  Scenes are the library's own seeded ones: the room of 20,500
triangles at 512x256 and the engine-scale scene of 1,050,972 triangles at
1728x864, 2 bounces.
"""
import ctypes as C
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "luminagi-cudaref_b200"))

import lumina  # noqa: E402
from lumina import _ffi  # noqa: E402
from lumina.scene import ENGINE_CENTER, Scene, box_scene, engine_scene, orbit_poses  # noqa: E402
from lumina.unet import flatten_state_dict, param_shapes  # noqa: E402

ENGINE_TRIS = 1050972
FULL = (1728, 864)


def listed():
    return [
        # A BVH over a small scene already on the device (BuildBVH of the box room), as an engine that
        # refits its scene every frame calls it: launches and the read of the node count are what it costs.
        {"name": "bvh-20k", "op": "bvh", "tris": 20500},
        # The same over the engine-scale scene: memory passes over 105 MB of triangles.
        {"name": "bvh-1M", "op": "bvh", "tris": ENGINE_TRIS},
        # Opening a scene and looking at it: upload, BVH, traversal records and one direct-light sample per
        # pixel (what the reference's RenderSceneCUDA does for each image).
        {"name": "open-scene-1M", "op": "open", "tris": ENGINE_TRIS, "w": 1728, "h": 864, "spp": 1, "bounces": 0},
        # The smallest frame: the box room at 1 sample, direct light, 8-bit image and radiance to the host.
        {"name": "frame-box-1spp", "op": "frame", "scene": "box", "w": 512, "h": 256, "spp": 1, "bounces": 0},
        # The reference's headline frame, 64 samples and 2 bounces, linear radiance to the host (--hdr).
        {"name": "frame-engine-64spp", "op": "frame", "scene": "engine", "w": 1728, "h": 864, "spp": 64,
         "bounces": 2},
        # 8 noisy samples and the denoiser, chained on the device: the fast path to a clean frame.
        {"name": "denoised-frame-8spp", "op": "chain", "scene": "engine", "w": 1728, "h": 864, "spp": 8, "bounces": 2},
        # A batch file of orbit poses, small previews (cuda_ref --batch; the training set's noisy renders).
        {"name": "batch-12-poses", "op": "batch", "scene": "engine", "w": 510, "h": 254, "spp": 8, "bounces": 2,
         "poses": 12},
        # The denoiser alone on one small G-buffer frame (12 input channels): the shortest network pass.
        {"name": "denoise-12ch-256x512", "op": "denoise", "variant": "ref", "in_ch": 12, "n": 1, "h": 256, "w": 512},
        # The denoiser alone on eight full frames (a sequence denoised after rendering).
        {"name": "denoise-8x864x1728", "op": "denoise", "variant": "ref", "in_ch": 3, "n": 8, "h": 864, "w": 1728},
        # The radiance variant (bilinear upsampling, log space) on one frame of an ordinary size.
        {"name": "denoise-hdr-720x1280", "op": "denoise", "variant": "hdr", "in_ch": 3, "n": 1, "h": 720, "w": 1280},
        # An image file denoised (python -m lumina.denoise): 8-bit host image in and out, a size that has to be
        # padded to multiples of 8.
        {"name": "denoise-image-1283x719", "op": "image", "w": 1283, "h": 719},
        # The gradients of a training step: the training recipe's batch of 16 crops of 128 x 128.
        {"name": "gradients-16x128x128", "op": "grad", "variant": "ref", "in_ch": 3, "n": 16, "h": 128, "w": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["bvh", "open", "frame", "frame", "chain", "batch", "denoise", "denoise", "image", "grad"])
    if op == "bvh":
        return {"op": op, "tris": _log(rng, 500, ENGINE_TRIS)}
    if op == "open":
        return {"op": op, "tris": _log(rng, 5000, ENGINE_TRIS), "w": rng.randint(256, 1728), "h": rng.randint(128, 864),
                "spp": rng.randint(1, 2), "bounces": rng.randint(0, 1)}
    if op == "frame":
        return {"op": op, "scene": rng.choice(["box", "engine"]), "w": _log(rng, 128, 1728), "h": _log(rng, 64, 864),
                "spp": rng.choice([1, 2, 4, 7, 8, 16, 24, 48, 64]), "bounces": rng.randint(0, 2)}
    if op == "chain":
        return {"op": op, "scene": rng.choice(["box", "engine"]), "w": 8 * _log(rng, 16, 216), "h": 8 * _log(rng, 12, 108),
                "spp": rng.choice([2, 4, 8]), "bounces": rng.randint(0, 2)}
    if op == "batch":
        return {"op": op, "scene": rng.choice(["box", "engine"]), "w": _log(rng, 128, 800), "h": _log(rng, 64, 400),
                "spp": rng.choice([1, 4, 8, 16]), "bounces": rng.randint(0, 2), "poses": rng.randint(2, 16)}
    if op == "image":
        return {"op": op, "w": _log(rng, 160, 1728), "h": _log(rng, 90, 864)}
    if op == "denoise":
        variant = rng.choice(["ref", "ref", "hdr"])
        n, h, w = rng.choice([1, 1, 2, 4]), 8 * _log(rng, 12, 108), 8 * _log(rng, 16, 216)
        return {"op": op, "variant": variant, "in_ch": 3 if variant == "hdr" else rng.choice([3, 12]), "n": n, "h": h,
                "w": w}
    variant = rng.choice(["ref", "hdr"])
    return {"op": op, "variant": variant, "in_ch": 3 if variant == "hdr" else rng.choice([3, 12]),
            "n": rng.choice([4, 8, 13, 16]), "h": 8 * rng.randint(8, 20), "w": 8 * rng.randint(8, 20)}


# ---- inputs ----
@functools.lru_cache(maxsize=None)
def _engine():
    return engine_scene(seed=7)


def _triangles(n, seed):
    """n triangles of the engine scene (a run of its meshes at a seeded place), turned about z and moved, as
    records on the GPU."""
    rng = np.random.default_rng(seed)
    base = _engine().tris
    at = int(rng.integers(0, len(base) - n + 1))
    t = torch.from_numpy(base[at:at + n].view(np.float32).reshape(n, 25).copy()).cuda()
    a = float(rng.uniform(0, 2 * math.pi))
    rot = torch.tensor([[math.cos(a), -math.sin(a), 0], [math.sin(a), math.cos(a), 0], [0, 0, 1]], dtype=torch.float32,
                       device="cuda")
    # by elementwise products: the same bits on every run
    p = t[:, :18].reshape(n, 6, 3)
    q = (p[..., None, :] * rot).sum(-1)
    q[:, :3] += torch.tensor(rng.uniform(-1, 1, 3), dtype=torch.float32, device="cuda")
    t[:, :18] = q.reshape(n, 18)
    return t


def _scene(name, w, h, seed):
    """The box room (a new one for each seed) or the engine scene (new materials), and a pose in or around it."""
    rng = np.random.default_rng(seed)
    if name == "box":
        sc = box_scene(seed, w, h)
        return sc, sc.camera
    e = _engine()
    cam = e.camera.copy()
    cam.width, cam.height = w, h
    sc = Scene(cam, e.sun, e.tris, rng.uniform(0.05, 0.95, e.mat_albedo.shape), e.mat_emissive, e.points)
    (pos, target), = orbit_poses(1, seed=seed, center=ENGINE_CENTER)
    return sc, cam.look_at(pos, target)


def _params(variant, in_ch, seed, trained):
    """The shipped denoiser weights, or a fresh network's (uniform in +-1/sqrt(fan-in))."""
    if trained:
        from lumina import surrogate
        path = os.path.join(os.path.dirname(os.path.abspath(surrogate.__file__)), "data", "unet_engine_long.npz")
        return np.load(path)["params"].astype(np.float32)
    rng = np.random.default_rng(seed)
    sd = {}
    for k, s in param_shapes(in_ch):
        fan = int(np.prod(s[1:])) if len(s) > 1 else fan
        sd[k] = rng.uniform(-1, 1, s) / math.sqrt(fan)
    return flatten_state_dict(sd, in_ch)


def _images(n, c, h, w, seed, hdr, noise=0.25):
    """Noisy renders: smooth shading, hard edges and per-pixel noise; radiance (hdr) has a long bright tail."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    low = torch.rand((n, c, max(2, h // 32), max(2, w // 32)), generator=g, device="cuda")
    x = torch.nn.functional.interpolate(low, size=(h, w), mode="nearest")
    x = 0.7 * x + 0.3 * torch.nn.functional.interpolate(low.flip(-1), size=(h, w), mode="bilinear")
    clean = x * x
    noisy = clean * (1 + noise * torch.randn(x.shape, generator=g, device="cuda")).clamp_min(0)
    if hdr:
        noisy = noisy * torch.empty_like(noisy).exponential_(1.0, generator=g)
        return noisy.contiguous(), clean[:, :3].contiguous()
    return noisy.sqrt().clamp(0, 1).contiguous(), clean[:, :3].sqrt().clamp(0, 1).contiguous()


def _net(case, seed, trained):
    net = lumina.UNet(in_ch=case.get("in_ch", 3), variant=case.get("variant", "ref"))
    p = _params(net.variant, net.in_ch, seed, trained and net.variant == "ref" and net.in_ch == 3)
    net.set_params(p)
    return net, p


def prepare(case, seed):
    op = case["op"]
    if op == "bvh":
        n = case["tris"]
        t = _triangles(n, seed)
        return {"op": op, "n": n, "tris": t, "out": torch.empty_like(t), "stream": torch.cuda.Stream(),
                "nodes": torch.zeros((2 * n - 1) * 40, dtype=torch.uint8, device="cuda"),
                "perm": torch.empty(n, dtype=torch.int32, device="cuda")}
    if op == "open":
        n = case["tris"]
        host = torch.empty((n, 25), dtype=torch.float32, pin_memory=True)
        host.copy_(_triangles(n, seed))
        e, cam = _scene("engine", case["w"], case["h"], seed)
        sc = Scene(cam, e.sun, host.numpy().view(_ffi.TRI_DTYPE).reshape(n), e.mat_albedo, e.mat_emissive, e.points)
        return {"op": op, "case": case, "r": lumina.Renderer(0), "scene": sc, "host": host}
    if op in ("frame", "chain", "batch"):
        sc, cam = _scene(case["scene"], case["w"], case["h"], seed)
        r = lumina.Renderer(0)
        r.set_scene(sc)
        st = {"op": op, "case": case, "r": r, "cam": cam}
        if op == "batch":
            if case["scene"] == "engine":
                st["cams"] = [cam.look_at(p, t) for p, t in orbit_poses(case["poses"], seed=seed, center=ENGINE_CENTER)]
            else:
                rng = np.random.default_rng(seed)
                st["cams"] = [cam.look_at(rng.uniform([-3.6, -3.5, 0.8], [-2.8, 0.5, 3.2]), [1.0, 0.2, 1.2])
                              for _ in range(case["poses"])]
        if op == "chain":
            st["net"], _ = _net({}, seed, True)
            st["x"] = torch.empty((1, 3, case["h"], case["w"]), device="cuda")
            st["y"] = torch.empty_like(st["x"])
            st["stream"] = torch.cuda.Stream()
        return st
    if op == "denoise":
        net, _ = _net(case, seed, True)
        x, _ = _images(case["n"], case["in_ch"], case["h"], case["w"], seed, case["variant"] == "hdr")
        y = torch.empty((case["n"], 3, case["h"], case["w"]), device="cuda")
        return {"op": op, "case": case, "net": net, "x": x, "y": y, "stream": torch.cuda.Stream()}
    if op == "image":
        net, _ = _net({}, seed, True)
        x, _ = _images(1, 3, case["h"], case["w"], seed, False)
        img = np.ascontiguousarray((x[0].permute(1, 2, 0) * 255).to(torch.uint8).cpu().numpy())
        return {"op": op, "net": net, "img": img}
    net, _ = _net(case, seed, False)
    x, t = _images(case["n"], case["in_ch"], case["h"], case["w"], seed, case["variant"] == "hdr")
    return {"op": op, "case": case, "net": net, "x": x, "t": t}


# ---- one pass ----
def run(state):
    op = state["op"]
    if op == "bvh":
        count = C.c_int32(0)
        _ffi.check(_ffi.lib().lg_build_bvh_device(
            C.c_void_p(state["tris"].data_ptr()), state["n"], C.c_void_p(state["nodes"].data_ptr()), C.byref(count),
            C.c_void_p(state["perm"].data_ptr()), C.c_void_p(state["out"].data_ptr()),
            C.c_void_p(state["stream"].cuda_stream)))
        return {"count": int(count.value), "nodes": state["nodes"], "perm": state["perm"], "tris": state["out"]}
    case = state.get("case")
    if op == "open":
        state["r"].set_scene(state["scene"])
        f = state["r"].render(spp=case["spp"], bounces=case["bounces"])
        return {"rgb": f["rgb"], "accum": f["accum"]}
    if op == "frame":
        # past 16 samples a pixel's chunks are summed in no fixed order, so an 8-bit value may round either way:
        # such frames come as linear radiance
        f = state["r"].render(camera=state["cam"], spp=case["spp"], bounces=case["bounces"], rgb=case["spp"] <= 16)
        return {"rgb": f["rgb"], "accum": f["accum"]}
    if op == "batch":
        n = case["poses"]
        rgb, _ = state["r"].render_batch(state["cams"], [case["spp"]] * n, [case["bounces"]] * n)
        return {"rgb": rgb}
    if op == "chain":
        c, o = state["cam"].to_c(), _ffi.LgRenderOpts(case["spp"], case["bounces"], 0, 0)
        st = state["stream"].cuda_stream
        rgb = C.c_void_p()
        _ffi.check(_ffi.lib().lg_render_device(state["r"]._h, C.byref(c), C.byref(o), C.c_void_p(st), C.byref(rgb), None,
                                               None))
        x, y = state["x"], state["y"]
        _ffi.check(_ffi.lib().lg_rgb8_to_f32(rgb, 1, case["h"], case["w"], C.c_void_p(x.data_ptr()), C.c_void_p(st)))
        state["net"].forward_device(x.data_ptr(), 1, case["h"], case["w"], y.data_ptr(), st)
        return {"noisy": x, "clean": y}
    if op == "denoise":
        x, y = state["x"], state["y"]
        state["net"].forward_device(x.data_ptr(), x.shape[0], x.shape[2], x.shape[3], y.data_ptr(),
                                    state["stream"].cuda_stream)
        return {"y": y}
    if op == "image":
        return {"rgb": state["net"].denoise_rgb8(state["img"])}
    x, t = state["x"], state["t"]
    loss, g = state["net"].loss_grad(x.data_ptr(), t.data_ptr(), x.shape[0], x.shape[2], x.shape[3])
    return {"loss": loss, "grad": g}


# ---- what a pass cannot do without ----
def _net_flops(n, h, w, in_ch=3):
    # multiply-adds per pixel of the network's convolutions, levels at 1, 1/4, 1/16, 1/64 of the pixels
    mac = 9 * (in_ch * 32 + 32 * 32 + 96 * 32 + 32 * 32) + 32 * 3
    mac += 9 * (32 * 64 + 64 * 64 + 192 * 64 + 64 * 64) / 4 + 9 * (64 * 128 + 128 * 128 + 384 * 128 + 128 * 128) / 16
    mac += 9 * (128 * 256 + 256 * 256) / 64
    return 2.0 * mac * n * h * w


def _trace(tris, pixels, spp, bounces, lights):
    """Bytes and operations of a frame: each triangle's vertices once, the radiance and 8-bit image out; per
    path segment a ray and a shadow ray per light, each going down a balanced binary tree once (two boxes a
    level, about 20 operations each) to one triangle test (about 40)."""
    rays = float(pixels) * spp * (1 + bounces) * (1 + lights)
    return {"bytes": 36.0 * tris + 15.0 * pixels, "flops": rays * (40.0 * math.log2(max(2, tris)) + 40.0)}


def work(case):
    op = case["op"]
    if op == "bvh":
        n = case["tris"]
        # triangles in and out, permutation, and a node (40 bytes) for each of about 0.7 per triangle
        return {"bytes": n * (100.0 + 100.0 + 4.0 + 28.0), "flops": 60.0 * n}
    if op in ("open", "frame", "chain", "batch"):
        pixels = case["w"] * case["h"] * case.get("poses", 1)
        box = case.get("scene") == "box"
        tris = case.get("tris", 20500 if box else ENGINE_TRIS)
        k = _trace(tris, pixels, case["spp"], case["bounces"], 2 if box else 3)
        if op == "open":
            k["bytes"] += tris * 300.0
        if op == "chain":
            k["bytes"] += pixels * 24.0
            k["flops"] += _net_flops(1, case["h"], case["w"])
        return k
    n, h, w, c = case.get("n", 1), case["h"], case["w"], case.get("in_ch", 3)
    n_params = sum(int(np.prod(s)) for _, s in param_shapes(c))
    if op == "image":
        return {"bytes": 6.0 * h * w + 4 * n_params, "flops": _net_flops(1, h, w)}
    if op == "denoise":
        return {"bytes": 4.0 * n * h * w * (c + 3) + 4 * n_params, "flops": _net_flops(n, h, w, c)}
    return {"bytes": 4.0 * n * h * w * (c + 3) + 8.0 * n_params, "flops": 3 * _net_flops(n, h, w, c)}


# ---- the network in 64 bits ----
def _forward64(sd, x, hdr):
    """The denoiser in float64: (output, network output before the last clamp or expm1)."""
    F = torch.nn.functional

    def act(v):
        return F.relu(v) if hdr else F.leaky_relu(v, 0.1)

    def block(name, v):
        v = act(F.conv2d(v, sd[name + ".net.0.weight"], sd[name + ".net.0.bias"], padding=1))
        return act(F.conv2d(v, sd[name + ".net.2.weight"], sd[name + ".net.2.bias"], padding=1))

    def up(v):
        if hdr:
            return F.interpolate(v, scale_factor=2, mode="bilinear", align_corners=False)
        return F.interpolate(v, scale_factor=2, mode="nearest")

    z = torch.log1p(x) if hdr else x
    d1 = block("d1", z)
    d2 = block("d2", F.max_pool2d(d1, 2))
    d3 = block("d3", F.max_pool2d(d2, 2))
    d4 = block("d4", F.max_pool2d(d3, 2))
    u = block("u3", torch.cat([up(d4), d3], 1))
    u = block("u2", torch.cat([up(u), d2], 1))
    u = block("u1", torch.cat([up(u), d1], 1))
    v = z[:, :3] + F.conv2d(u, sd["tail.weight"], sd["tail.bias"])
    return (torch.expm1(v.clamp_min(0)) if hdr else v.clamp(0, 1)), v


def _sd64(p, in_ch, grad=False):
    sd, at = {}, 0
    for k, s in param_shapes(in_ch):
        n = int(np.prod(s))
        sd[k] = torch.from_numpy(p[at:at + n].reshape(s)).to("cuda", torch.float64).requires_grad_(grad)
        at += n
    return sd


def exact(case, seed):
    """The network's outputs and gradients in float64.  Images, trees and path-traced frames have no such value:
    an image's bytes and a tree's records are exact or wrong, and a path's radiance is one sample of its RNG."""
    op = case["op"]
    if op not in ("denoise", "grad"):
        return None
    hdr = case["variant"] == "hdr"
    trained = op == "denoise" and not hdr and case["in_ch"] == 3
    p = _params(case["variant"], case["in_ch"], seed, trained)
    x, t = _images(case["n"], case["in_ch"], case["h"], case["w"], seed, hdr)
    if op == "denoise":
        sd = _sd64(p, case["in_ch"])
        with torch.no_grad():
            return {"y": torch.cat([_forward64(sd, x[i:i + 1].double(), hdr)[0] for i in range(x.shape[0])])}
    sd = _sd64(p, case["in_ch"], True)
    y, v = _forward64(sd, x.double(), hdr)
    loss = (v.clamp_min(0) - torch.log1p(t.double())).abs().mean() if hdr else (y - t.double()).abs().mean()
    loss.backward()
    return {"loss": loss.detach(), "grad": torch.cat([g.grad.reshape(-1) for g in sd.values()])}
