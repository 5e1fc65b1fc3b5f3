"""The work that users of this framework have it do, as cases that can be timed: whole frames
from the smallest to 4K, the traced and screen-space passes on device and host buffers, batched
views, the learned surrogate (a frame, a training step, one convolution), accelerator rebuilds
with closest-hit queries, and the path tracer. Every case goes through the package's public
entry points (raw-native_gb300/rn_ao.py).

A case is a dict of plain values; ``listed()`` names the fixed ones, ``draw(rng)`` makes one more
of the same ranges. ``prepare`` makes what a program holds before the call (scene, G-buffer,
accelerator, network), ``run`` is one pass and returns its outputs, ``work`` is the bytes and
operations of a pass that no implementation can do without, ``exact`` the same outputs in 64
bits by plain torch where the path computes rounded numbers of such a kind (a convolution,
gradients, GTAO). Traced and rasterized planes have no such value: the reference defines them by
its order of float32 operations.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.getcwd()
sys.path.insert(1, os.path.join(ROOT, "raw-native_gb300"))
import rn_ao as rn          # noqa: E402
import scene as scenes      # noqa: E402
import surrogate            # noqa: E402

DEV = "cuda"


def listed():
    return [
        # The smallest call: SSAO of one 512 x 512 G-buffer and its reconcile against a traced
        # AO image, what an editor or a test runs per change. Launches and latency.
        dict(name="judge_512", kind="judge", w=512, h=512, taps=24, radius=2.0),
        # The command line's default: the built-in scene rendered whole at 512 x 512, 64 spp
        # (rasterizer, accelerator build, traced AO with sky and sun, SSAO, reconcile, shading).
        dict(name="frame_512", kind="frame", boxes=0, spheres=0, w=512, h=512, spp=64, lighting=2, radius=2.0),
        # A whole frame of a 146k-triangle scene at an odd size and few samples: a preview, where
        # the rasterizer and the build weigh as much as the rays.
        dict(name="frame_scene_odd", kind="frame", boxes=200, spheres=50, w=1283, h=723, spp=16, lighting=2, radius=1.0),
        # The benchmark's frame: 4K, 256 spp with sky and sun, on a resident G-buffer.
        dict(name="ao_4k_256", kind="ao", boxes=0, spheres=0, w=3840, h=2160, spp=256, sky=True, radius=2.0),
        # The same passes from a C++ program's pinned host images, 1080p at the default 64 spp.
        dict(name="ao_host_1080", kind="host", boxes=0, spheres=0, w=1920, h=1080, spp=64, sky=True, radius=2.0),
        # Batched views of uneven size and spp over the 744k-triangle scene in one launch.
        dict(name="views_744k", kind="views", boxes=2000, spheres=500, radius=1.0,
             views="512x512x256,1280x720x64,1920x1080x16,2560x1440x16,1920x1080x64,1281x723x16"),
        # A 4K frame of the 7.88M-triangle scene by the learned surrogate: the 4-spp trace, the
        # U-Net with its trained weights, the fallback tiles.
        dict(name="surrogate_4k", kind="surrogate", boxes=10000, spheres=6000, w=3840, h=2160, spp=139, radius=1.0),
        # One training step of the surrogate at its recipe's batch: forward, backward, the
        # gradients handed out (as to an all-reduce), clip and Adam.
        dict(name="train_64x128", kind="train", batch=64, h=128, w=128),
        # One block of the network alone: the concatenated level-2 decoder convolution at 1080p.
        dict(name="conv_level2", kind="conv", batch=1, h=272, w=480, c0=128, c1=256, n=128),
        # A dynamic scene's frame: the accelerator rebuilt over 744k triangles, then a million
        # nearest-hit queries through it.
        dict(name="rebuild_744k", kind="rebuild", boxes=2000, spheres=500, rays=1 << 20),
        # The path tracer's lit room at 1080p, 4 samples a pixel, every output plane.
        dict(name="path_room", kind="path", scene="retro_room", w=1920, h=1080, spp=4),
        # The screen-space GTAO of a large odd-sized G-buffer, defaults (16 slices, 16 steps).
        dict(name="gtao_odd", kind="gtao", w=2561, h=1441, slices=16, steps=16, radius=0.5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, wlo, whi):
    w = _log(rng, wlo, whi)
    return w, max(16, int(w * rng.uniform(0.5, 0.8)))


def _scene_counts(rng, most):
    """0 (the built-in scene) a third of the time, else counts spread over their logarithms."""
    if rng.random() < 1 / 3:
        return 0, 0
    return _log(rng, 100, most), _log(rng, 20, max(40, most // 4))


def draw(rng):
    kind = rng.choice(["judge", "frame", "ao", "host", "views", "surrogate", "train", "conv", "rebuild", "path", "gtao"])
    if kind == "judge":
        w, h = _size(rng, 96, 4096)
        return dict(kind=kind, w=w, h=h, taps=rng.choice([8, 24, 24, 32]), radius=round(rng.uniform(0.5, 3.0), 3))
    if kind == "frame":
        b, s = _scene_counts(rng, 2000)
        w, h = _size(rng, 128, 1920)
        spp = _log(rng, 4, 64)
        while w * h * spp > 60_000_000 and spp > 4:
            spp //= 2
        return dict(kind=kind, boxes=b, spheres=s, w=w, h=h, spp=spp, lighting=rng.choice([2, 2, 1]),
                    radius=round(rng.uniform(0.5, 2.5), 3))
    if kind in ("ao", "host"):
        b, s = _scene_counts(rng, 2000) if kind == "ao" else (0, 0)
        w, h = _size(rng, 256, 3840 if kind == "ao" else 2560)
        spp, sky = _log(rng, 1, 256), rng.random() < 0.6
        most = 400_000_000 if not b else 60_000_000 if sky else 150_000_000
        while w * h * spp > most and spp > 1:
            spp //= 2
        return dict(kind=kind, boxes=b, spheres=s, w=w, h=h, spp=spp, sky=sky, radius=round(rng.uniform(0.5, 2.5), 3))
    if kind == "views":
        views = []
        for _ in range(rng.randint(2, 6)):
            w, h = _size(rng, 256, 2560)
            spp = rng.choice([4, 16, 64])
            while w * h * spp > 40_000_000:
                spp //= 2
            views.append("%dx%dx%d" % (w, h, max(1, spp)))
        return dict(kind=kind, boxes=_log(rng, 200, 2000), spheres=_log(rng, 50, 500), radius=1.0, views=",".join(views))
    if kind == "surrogate":
        w, h = _size(rng, 640, 3840)
        return dict(kind=kind, boxes=_log(rng, 200, 2000), spheres=_log(rng, 50, 500), w=w, h=h,
                    spp=rng.choice([64, 139, 256]), radius=1.0)
    if kind == "train":
        return dict(kind=kind, batch=8 * rng.randint(1, 8), h=rng.choice([64, 96, 128]), w=rng.choice([64, 128, 128]))
    if kind == "conv":
        lv = rng.randint(0, 3)
        c = 32 << lv
        c1 = rng.choice([0, 0, 2 * c]) if lv < 3 else 0
        return dict(kind=kind, batch=rng.randint(1, 4), h=8 * rng.randint(4, 160 >> lv), w=16 * rng.randint(2, 120 >> lv),
                    c0=c, c1=c1, n=c)
    if kind == "rebuild":
        return dict(kind=kind, boxes=_log(rng, 20, 2000), spheres=_log(rng, 5, 500), rays=_log(rng, 20_000, 2_000_000))
    if kind == "path":
        w, h = _size(rng, 160, 1920)
        spp = _log(rng, 1, 16)
        while w * h * spp > 8_000_000 and spp > 1:
            spp //= 2
        return dict(kind=kind, scene=rng.choice(["retro_room", "iso_street"]), w=w, h=h, spp=spp)
    w, h = _size(rng, 256, 2560)
    return dict(kind="gtao", w=w, h=h, slices=rng.choice([4, 8, 16]), steps=rng.choice([8, 16]),
                radius=round(rng.uniform(0.25, 1.0), 3))


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=4)
def _scene(boxes, spheres):
    """(triangles, normals, to-light) on the host: the built-in scene, or a seeded synthetic one
    (the scene is part of the case; the seed moves the camera)."""
    sc = scenes.build_test_scene() if not boxes and not spheres else scenes.build_synthetic_scene(5, boxes, spheres)
    return sc.tris, sc.normals, tuple(float(v) for v in sc.to_light)


def _camera(boxes, seed, k=0):
    r = np.random.Generator(np.random.PCG64([seed, k]))
    if not boxes:       # around the command line's default view
        e = np.array([4.0, 4.0, 6.0]) + r.uniform(-0.3, 0.3, 3)
        return (*map(float, e), 0.0, 1.0, 0.0, 0.0, 1.0, 0.0, 0.9)
    a, y = r.uniform(0, 2 * math.pi), r.uniform(3.0, 20.0)
    return (40.0 * math.cos(a), float(y), 40.0 * math.sin(a), 0.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.9)


def _analytic_gbuffer(w, h, seed):
    """A G-buffer by plain torch: a ground plane and 24 seeded spheres seen by a seeded camera
    (positions and normals of the nearest surface; the sky uncovered). Returns
    (rn.GBuffer, camera)."""
    cam = _camera(0, seed)
    r = np.random.Generator(np.random.PCG64([seed, 77]))
    eye = torch.tensor(cam[0:3], device=DEV, dtype=torch.float64)
    f = torch.tensor(cam[3:6], device=DEV, dtype=torch.float64) - eye
    f = f / f.norm()
    side = torch.linalg.cross(f, torch.tensor(cam[6:9], device=DEV, dtype=torch.float64))
    side = side / side.norm()
    up = torch.linalg.cross(side, f)
    t = math.tan(0.5 * cam[9])
    px = ((torch.arange(w, device=DEV, dtype=torch.float64) + 0.5) / w * 2 - 1) * t * w / h
    py = (1 - (torch.arange(h, device=DEV, dtype=torch.float64) + 0.5) / h * 2) * t
    d = (f + px[None, :, None] * side + py[:, None, None] * up).float()
    d = d / d.norm(dim=-1, keepdim=True)
    o = eye.float()
    best = torch.full((h, w), float("inf"), device=DEV)
    nrm = torch.zeros(h, w, 3, device=DEV)
    tp = torch.where(d[..., 1] < -1e-3, -o[1] / d[..., 1], torch.inf)
    hit = tp < 40
    best[hit] = tp[hit]
    nrm[hit] = torch.tensor([0.0, 1.0, 0.0], device=DEV)
    for c in r.uniform([-4, 0.2, -4, 0.3], [4, 1.2, 4, 1.0], (24, 4)):
        oc = o - torch.tensor(c[:3], device=DEV, dtype=torch.float32)
        b = (d * oc).sum(-1)
        disc = b * b - (oc.dot(oc) - float(c[3]) ** 2)
        ts = -b - disc.clamp_min(0).sqrt()
        hit = (disc > 0) & (ts > 0.05) & (ts < best)
        best[hit] = ts[hit]
        n = (oc + ts[hit][:, None] * d[hit]) / float(c[3])
        nrm[hit] = n / n.norm(dim=-1, keepdim=True)
    mask = torch.isfinite(best)
    pos = torch.where(mask[..., None], o + best.nan_to_num(posinf=0.0)[..., None] * d, 0.0)
    return rn.GBuffer(pos.contiguous(), nrm, mask.to(torch.uint8)), cam


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _pt_scene(key):
    z = np.load(os.path.join(ROOT, "tests", "golden", "pt_scenes.npz"))
    sc = {k.split("/", 1)[1]: z[k] for k in z.files if k.startswith(key + "/")}
    return sc, sc.pop("camera")


def _unet_weights(seed):
    """He-initialized parameters in rn.UNet.set_params' order: per convolution w[cout][9 cin]
    (tap-major) and b, then the head; BF16-representable weights. numpy, from the seed."""
    r = np.random.Generator(np.random.PCG64([seed, 3]))
    parts = []
    for cin, cout in rn.UNET_CONVS:
        parts.append(r.standard_normal((cout, 9 * cin), np.float32) * np.float32(math.sqrt(2.0 / (9 * cin))))
        parts.append(r.standard_normal(cout, np.float32) * np.float32(0.02))
    parts += [r.standard_normal(32, np.float32) * np.float32(0.05), np.array([0.8], np.float32)]
    return np.concatenate([p.ravel() for p in parts])


def _train_batch(c, seed):
    """Surrogate features as the recipe makes them (depth in [-4, 4], unit normals, AO in
    quarters) and a smooth target."""
    g = _gen(seed)
    B, H, W = c["batch"], c["h"], c["w"]
    low = torch.rand(B, 8, H // 16, W // 16, device=DEV, generator=g) * 2 - 1
    s = torch.nn.functional.interpolate(low, size=(H, W), mode="bilinear").permute(0, 2, 3, 1)
    n = s[..., 1:4] + torch.tensor([0.0, 1.0, 0.0], device=DEV)
    ao = (0.75 + 0.35 * s[..., 4]).clamp(0, 1)
    ao4 = (torch.rand(B, H, W, 4, device=DEV, generator=g) < ao[..., None]).float().mean(-1)
    x = torch.cat([0.5 * s[..., :1], n / n.norm(dim=-1, keepdim=True).clamp_min(1e-3), ao4[..., None]], -1)
    return x.contiguous(), ao.contiguous()


def _conv_inputs(c, seed):
    g = _gen(seed)
    half = lambda *s: torch.randn(*s, device=DEV, generator=g)   # noqa: E731
    x0 = half(c["batch"], c["h"], c["w"], c["c0"]).relu_().bfloat16()
    x1 = half(c["batch"], c["h"], c["w"], c["c1"]).relu_().bfloat16() if c["c1"] else None
    cin = c["c0"] + c["c1"]
    w = (half(c["n"], 9 * cin) * math.sqrt(2.0 / (9 * cin))).bfloat16()
    return x0, x1, w, half(c["n"]) * 0.1


def _to_device(c):
    tris, nrm, tl = _scene(c["boxes"], c["spheres"])
    return torch.from_numpy(tris).to(DEV), torch.from_numpy(nrm).to(DEV), tl


def prepare(case, seed):
    rn.init()
    c, kind = dict(case), case["kind"]
    s = {"c": c, "kind": kind}
    if kind in ("judge", "gtao"):
        s["g"], s["cam"] = _analytic_gbuffer(c["w"], c["h"], seed)
        if kind == "judge":
            s["truth"] = torch.randint(0, 65, (c["h"], c["w"]), device=DEV, generator=_gen(seed)).float() / 64
    elif kind == "frame":
        s["tris"], s["nrm"], tl = _to_device(c)
        s["light"] = (tuple(-v for v in tl), 1.0)
        s["cam"] = _camera(c["boxes"], seed)
        s["albedo"] = torch.rand(len(s["tris"]), 3, device=DEV, generator=_gen(seed))
    elif kind in ("ao", "host", "surrogate"):
        tris, nrm, s["tl"] = _to_device(c)
        s["acc"] = rn.LinearAccel(tris)
        s["g"], s["depth"] = rn.rasterize(tris, nrm, _camera(c["boxes"], seed), c["w"], c["h"], want_depth=True)
        if kind == "host":
            pin = lambda t: t.cpu().pin_memory()      # noqa: E731
            s["keep"] = [pin(s["g"].position), pin(s["g"].normal), pin(s["g"].mask)]
            s["g"] = rn.GBuffer(*[t.numpy() for t in s["keep"]])
            names = ["ao", "ss", "err"] + (["sky", "sun"] if c["sky"] else [])
            s["outs"] = {k: torch.zeros(c["h"], c["w"], pin_memory=True) for k in names}
        if kind == "surrogate":
            s["net"] = rn.UNet(1, *surrogate.padded_shape(c["h"], c["w"]), inference=True)
            surrogate.load_weights(s["net"], os.path.join(ROOT, "raw-native_gb300", "weights", "surrogate_mixed_bf16.npz"))
    elif kind == "views":
        tris, nrm, _ = _to_device(c)
        s["acc"] = rn.LinearAccel(tris)
        views = []
        for k, v in enumerate(c["views"].split(",")):
            w, h, spp = map(int, v.split("x"))
            views.append(dict(g=rn.rasterize(tris, nrm, _camera(c["boxes"], seed, k), w, h), spp=spp, radius=c["radius"]))
        s["batch"] = rn.Batch(s["acc"], views)
    elif kind == "train":
        s["net"] = rn.UNet(c["batch"], c["h"], c["w"])
        s["net"].set_params(_unet_weights(seed))
        s["x"], s["y"] = _train_batch(c, seed)
        s["flat"] = torch.empty(s["net"].grad_count, device=DEV)
    elif kind == "conv":
        s["x0"], s["x1"], s["w"], s["b"] = _conv_inputs(c, seed)
    elif kind == "rebuild":
        s["tris"], _, _ = _to_device(c)
        # moving geometry: every vertex displaced a little
        s["tris"] = s["tris"] + 1e-3 * torch.randn(s["tris"].shape, device=DEV, generator=_gen(seed))
        g = _gen(seed + 1)
        o = torch.rand(c["rays"], 3, device=DEV, generator=g) * torch.tensor([100.0, 6.0, 100.0], device=DEV) - \
            torch.tensor([50.0, -0.5, 50.0], device=DEV)
        d = torch.randn(c["rays"], 3, device=DEV, generator=g)
        s["rays"] = torch.cat([o, d / d.norm(dim=-1, keepdim=True)], 1).contiguous()
        s["tmax"] = torch.full((c["rays"],), 1e30, device=DEV)
    elif kind == "path":
        sc, cam = _pt_scene(c["scene"])
        s["scene"] = rn.PtScene(sc)
        s["desc"] = dict(seed=int(seed), spp=c["spp"], width=c["w"], height=c["h"], camera=[float(v) for v in cam])
    return s


def _numbers(r):
    return [float(r.rmse), float(r.max_error), int(r.pixels), bool(r.within_tolerance)]


def run(s):
    c, kind = s["c"], s["kind"]
    if kind == "judge":
        ss = rn.compute_ssao(s["g"], c["taps"], c["radius"])
        r = rn.reconcile(ss, s["truth"], s["g"].mask)
        return {"ss": ss, "err": r.error_map, "rec": _numbers(r)}
    if kind == "gtao":
        return rn.gtao(s["g"], s["cam"], c["radius"], c["slices"], c["steps"])
    if kind == "frame":
        o = rn.render_frame(s["tris"], s["nrm"], s["albedo"], s["cam"], c["w"], c["h"], light=s["light"], spp=c["spp"],
                            radius=c["radius"], lighting=c["lighting"])
        if c["lighting"] != 2:
            del o["sky"], o["sun"]
        o["rec"] = _numbers(o["rec"])
        return o
    if kind in ("ao", "host"):
        o = rn.ao_frame(s["g"], s["acc"], c["spp"], c["radius"], to_light=s["tl"] if c["sky"] else None,
                        outputs={k: t.numpy() for k, t in s["outs"].items()} if kind == "host" else None)
        o["rec"] = _numbers(o["rec"])
        return o
    if kind == "views":
        r = s["batch"].run()
        return {"views": s["batch"].outputs, "rec": [_numbers(x) for x in r]}
    if kind == "surrogate":
        ao, st, parts = rn.surrogate_ao(s["net"], s["g"], s["depth"], s["acc"], c["spp"], c["radius"], want_parts=True)
        return {"ao": ao, "tiles": st["tiles_covered"], **parts}
    if kind == "train":
        # the first step of the recipe's warm-up: lr 1e-3 / 100
        loss = s["net"].backward(s["x"], s["y"])
        s["net"].grads_to(s["flat"])
        s["net"].apply(1e-5)
        return {"loss": loss, "grads": s["flat"]}
    if kind == "conv":
        return rn.tc_conv3x3(s["x0"], s["w"], s["x1"], bias=s["b"], relu=True, out_dtype=torch.bfloat16)
    if kind == "rebuild":
        tri, t = rn.closest(rn.LinearAccel(s["tris"]), s["rays"], s["tmax"])
        return {"tri": tri, "t": t}
    return rn.path_trace(s["scene"], s["desc"], device=True)


# ------------------------------------------------------------------ what a pass cannot do without
def _rays_flops(rays):
    """At least the root's four boxes (24 multiply-adds), one triangle (about 60 operations) and
    the sample's direction (about 60) for every ray."""
    return rays * (48 + 60 + 60)


def work(case):
    c, kind = case, case["kind"]
    px = c.get("w", 0) * c.get("h", 0)
    tri = lambda: len(_scene(c["boxes"], c["spheres"])[0])      # noqa: E731
    if kind == "judge":     # position, normal, mask, truth in; ss, err out; a tap about 40 operations
        return {"bytes": px * (25 + 4 + 8), "flops": px * c["taps"] * 40}
    if kind == "gtao":      # position, normal, mask in, AO out; a sample about 30 operations
        return {"bytes": px * 29, "flops": px * c["slices"] * 2 * c["steps"] * 30}
    if kind == "frame":     # the scene in, every plane out
        return {"bytes": tri() * 84 + px * 85, "flops": _rays_flops(px * c["spp"]) + px * 24 * 40}
    if kind in ("ao", "host"):
        return {"bytes": px * (25 + 12 + (8 if c["sky"] else 0)) + min(tri() * 48, px * c["spp"] * 48),
                "flops": _rays_flops(px * c["spp"]) + px * 24 * 40}
    if kind == "views":
        v = [tuple(map(int, x.split("x"))) for x in c["views"].split(",")]
        return {"bytes": sum(w * h * 37 for w, h, _ in v) + tri() * 48,
                "flops": sum(_rays_flops(w * h * s) + w * h * 24 * 40 for w, h, s in v)}
    if kind == "surrogate":     # G-buffer and depth in, the frame and its parts out
        return {"bytes": px * (29 + 12), "flops": _rays_flops(px * 4) + px * _unet_flops()}
    if kind == "train":
        m = c["batch"] * px
        return {"bytes": m * 24 + 1948321 * 4 * 7, "flops": 3 * m * _unet_flops()}
    if kind == "conv":
        m, cin = c["batch"] * px, c["c0"] + c["c1"]
        return {"bytes": m * (cin + c["n"]) * 2 + c["n"] * 9 * cin * 2, "flops": 2 * m * 9 * cin * c["n"]}
    if kind == "rebuild":
        return {"bytes": tri() * 36 + c["rays"] * 36, "flops": tri() * 60 + c["rays"] * 108}
    return {"bytes": px * 104, "flops": px * c["spp"] * 1000}


def _unet_flops():
    """Multiply-adds x 2 of the 3x3 convolutions per level-0 pixel."""
    level = [0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0]
    return sum(18 * a * b / 4 ** lv for (a, b), lv in zip(rn.UNET_CONVS, level))


# ------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    c, kind = dict(case), case["kind"]
    if kind == "conv":
        x0, x1, w, b = _conv_inputs(c, seed)
        x = torch.cat([x0, x1], -1) if x1 is not None else x0
        return _conv64(x, w, b)
    if kind == "gtao" and c["w"] * c["h"] * c["slices"] * c["steps"] <= 1_000_000_000:
        g, cam = _analytic_gbuffer(c["w"], c["h"], seed)
        return _gtao64(g, cam, c)
    if kind == "train" and c["batch"] * c["w"] * c["h"] <= 64 * 128 * 128:
        return _train64(c, seed)
    return None


def _conv64(x, w, b):
    B, H, W, C = x.shape
    p = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1))
    out = torch.zeros(B * H * W, w.shape[0], device=DEV, dtype=torch.float64)
    for t in range(9):
        out += p[:, t // 3:t // 3 + H, t % 3:t % 3 + W].reshape(-1, C) @ w[:, t * C:(t + 1) * C].double().t()
    return (out + b.double()).relu_().reshape(B, H, W, -1)


def _train64(c, seed):
    """Loss and gradients of the network in float64 autograd, laid out as grads_to lays them:
    per convolution [kpad][cout] (kpad = 9 cin rounded up to 128), the bias, then the head."""
    flat = torch.from_numpy(_unet_weights(seed)).to(DEV).double()
    x, y = _train_batch(c, seed)
    ws, o = [], 0
    for cin, cout in rn.UNET_CONVS:
        w = flat[o:o + cout * 9 * cin].reshape(cout, 9 * cin)
        o += cout * 9 * cin
        ws.append((w.clone().requires_grad_(), flat[o:o + cout].clone().requires_grad_()))
        o += cout
    wh, bh = flat[o:o + 32].clone().requires_grad_(), flat[o + 32:].clone().requires_grad_()

    n = c["batch"] * c["h"] * c["w"]
    total = 0.0
    for k in range(0, c["batch"], 8):        # eight images at a time bound the memory
        it = iter(ws)

        def conv(t):
            w, b = next(it)
            C = t.shape[-1]
            p = torch.nn.functional.pad(t, (0, 0, 1, 1, 1, 1))
            H, W = t.shape[1:3]
            acc = b
            for q in range(9):
                acc = acc + p[:, q // 3:q // 3 + H, q % 3:q % 3 + W] @ w[:, q * C:(q + 1) * C].t()
            return acc.relu()

        pool = lambda t: 0.25 * (t[:, ::2, ::2] + t[:, ::2, 1::2] + t[:, 1::2, ::2] + t[:, 1::2, 1::2])   # noqa: E731
        up = lambda t: t.repeat_interleave(2, 1).repeat_interleave(2, 2)   # noqa: E731
        x8 = torch.nn.functional.pad(x[k:k + 8].double(), (0, 3))
        e0 = conv(conv(x8))
        e1 = conv(conv(pool(e0)))
        e2 = conv(conv(pool(e1)))
        b3 = conv(conv(pool(e2)))
        d2 = conv(conv(torch.cat([e2, up(b3)], -1)))
        d1 = conv(conv(torch.cat([e1, up(d2)], -1)))
        d0 = conv(conv(torch.cat([e0, up(d1)], -1)))
        loss = ((torch.sigmoid(d0 @ wh + bh) - y[k:k + 8].double()) ** 2).sum() / n
        loss.backward()
        total += float(loss.detach())
    parts = []
    for (cin, cout), (w, b) in zip(rn.UNET_CONVS, ws):
        gw = torch.zeros(-(-9 * cin // 128) * 128, cout, device=DEV, dtype=torch.float64)
        gw[:9 * cin] = w.grad.t()
        parts += [gw.reshape(-1), b.grad]
    return {"loss": total, "grads": torch.cat(parts + [wh.grad, bh.grad])}


def _gtao64(g, cam, c):
    """GTAO (Jimenez et al. 2016) as raw::post defines it, in float64: per pixel `slices` screen
    directions, `steps` depth samples to each side, the horizon angles' closed-form integral.
    The view-space G-buffer is formed from the float32 one."""
    f64 = dict(device=DEV, dtype=torch.float64)
    h, w = g.shape
    eye, ctr, upv = (torch.tensor(cam[k:k + 3], **f64) for k in (0, 3, 6))
    f = (ctr - eye) / (ctr - eye).norm()
    sd = torch.linalg.cross(f, upv)
    sd = sd / sd.norm()
    R = torch.stack([sd, torch.linalg.cross(sd, f), -f])
    mask = g.mask.bool()
    ys, xs = torch.nonzero(mask, as_tuple=True)
    P = ((g.position.double()[mask] - eye) @ R.t()).float().double()
    N = g.normal.double()[mask] @ R.t()
    N = (N / N.norm(dim=-1, keepdim=True)).float().double()
    depth = -P[:, 2]
    D = torch.full((h, w), -1.0, **f64)
    D[mask] = depth
    th, asp = math.tan(0.5 * float(np.float32(cam[9]))), float(np.float32(w) / np.float32(h))
    V = -P / P.norm(dim=-1, keepdim=True)
    rpx = c["radius"] * h / (2 * th * depth)
    T = torch.tensor([1.0, 0.0, 0.0], **f64) - V[:, :1] * V
    T = T / T.norm(dim=-1, keepdim=True)
    Bt = torch.linalg.cross(V, T)
    dot = lambda a, b: (a * b).sum(-1)      # noqa: E731

    def at(qx, qy):
        ok = (qx >= 0) & (qy >= 0) & (qx < w) & (qy < h)
        d = D[qy.clamp(0, h - 1), qx.clamp(0, w - 1)]
        return torch.where(ok, d, -1.0)

    def project(p):
        z = -p[:, 2]
        return torch.stack([(p[:, 0] / (z * th * asp) * 0.5 + 0.5) * w, (1 - (p[:, 1] / (z * th) * 0.5 + 0.5)) * h], -1)

    p0, total = project(P), torch.zeros(len(P), **f64)
    for s in range(c["slices"]):
        a = math.pi * (s + 0.5) / c["slices"]
        dr = math.cos(a) * T + math.sin(a) * Bt
        dd = project(P + dr * (1e-3 * depth)[:, None]) - p0
        dd = dd / dd.norm(dim=-1, keepdim=True).clamp_min(1e-12)
        od = dr - dot(dr, V)[:, None] * V
        ax = torch.linalg.cross(od, V)
        ax = ax / ax.norm(dim=-1, keepdim=True)
        pn = N - ax * dot(N, ax)[:, None]
        pnl = pn.norm(dim=-1)
        cn = (dot(pn, V) / pnl.clamp_min(1e-30)).clamp(0, 1)
        ang = torch.where(dot(od, pn) >= 0, 1.0, -1.0) * cn.acos()
        hc = [(ang + math.pi / 2).cos(), (ang - math.pi / 2).cos()]
        for side in (0, 1):
            for k in range(1, c["steps"] + 1):
                off = (1 - 2 * side) * rpx * k / c["steps"]
                fx, fy = xs + 0.5 + off * dd[:, 0], ys + 0.5 + off * dd[:, 1]
                sx, sy = fx.floor().long(), fy.floor().long()
                near = at(sx, sy)
                ok = (near >= 0) & ((sx != xs) | (sy != ys))
                gx, gy = fx - 0.5, fy - 0.5
                x0, y0 = gx.floor().long(), gy.floor().long()
                bx, by = gx - x0, gy - y0
                q = torch.stack([at(x0, y0), at(x0 + 1, y0), at(x0, y0 + 1), at(x0 + 1, y0 + 1)])
                flat = (q < 0).any(0) | (q.amax(0) > 1.1 * q.amin(0))
                i = 1 / torch.where(q > 0, q, 1.0)
                lin = 1 / ((i[0] * (1 - bx) + i[1] * bx) * (1 - by) + (i[2] * (1 - bx) + i[3] * bx) * by)
                d = torch.where(flat, near, lin)
                S = torch.stack([(fx / w * 2 - 1) * d * th * asp, (1 - fy / h * 2) * d * th, -d], -1) - P
                dl = S.norm(dim=-1)
                ok &= (dl >= 1e-9) & (dl <= c["radius"])
                hc[side] = torch.where(ok, torch.maximum(hc[side], dot(S, V) / dl.clamp_min(1e-9)), hc[side])
        h1 = ang + torch.clamp_max(hc[0].clamp(-1, 1).acos() - ang, math.pi / 2)
        h0 = ang + torch.clamp_min(-hc[1].clamp(-1, 1).acos() - ang, -math.pi / 2)
        arc = lambda t: (cn + 2 * t * ang.sin() - (2 * t - ang).cos()) * 0.25      # noqa: E731
        total += torch.where(pnl < 1e-9, 0.0, pnl * (arc(h0) + arc(h1)))
    out = torch.ones(h, w, **f64)
    out[mask] = total / c["slices"]
    return out
