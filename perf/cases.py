"""The work that programs give this library, as cases that can be timed.

A case is a dict of plain values. ``listed()`` gives the fixed ones, ``draw``
further ones of the same ranges; ``prepare`` makes what a program holds before
the call (scene handle, buffers, weights), ``run`` is one pass through the
public entry points of ``nostrum_pray_gb300.native``, ``work`` the bytes and
operations a pass cannot do without, ``exact`` the outputs in 64 bits where
they have such a value.

Kinds of work:

* ``frame``   a ray-traced frame (primary rays, one occlusion ray per light)
* ``closest`` / ``occluded``  caller-given rays: closest hits, any-hit answers
* ``paths``   a path-traced frame: the reference's Kajiya estimator, or next-event
  estimation with Russian roulette, optionally with the first-hit features
  that the denoiser reads
* ``batch``   many scenes, one path-traced frame each, in one launch
* ``denoise`` U-Net inference on rendered radiance and features
* ``train``   loss and all gradients of one training batch of the U-Net
"""
from __future__ import annotations

import functools
import math
import random
from typing import Dict, List, Optional

import numpy as np
import torch

from nostrum_pray_gb300 import denoise, native, scenes

DEVICE = "cuda:0"


# -- the cases ---------------------------------------------------------------


def listed() -> List[Dict]:
    return [
        # a thumbnail or test frame through the host call, as the command line
        # makes it: launch, copy-out and latency are all there is
        {"name": "frame_thumbnail_host", "kind": "frame", "scene": "soup", "size": 2_000, "tree": "median",
         "width": 96, "height": 64, "lights": 1, "host": True, "hits": False},
        # the benchmark's default workload: the 1.31M-triangle displaced
        # sphere at 1080p with two lights
        {"name": "frame_sphere_1080p", "kind": "frame", "scene": "sphere", "size": 8, "tree": "sah",
         "width": 1920, "height": 1080, "lights": 2, "host": False, "hits": False},
        # incoherent rays inside the 101k-triangle room: what a renderer of
        # its own asks of the library as a ray engine; an odd count
        {"name": "closest_room_300k", "kind": "closest", "scene": "room", "size": 53, "tree": "sah",
         "rays": 300_007},
        # visibility queries in a 10k-triangle soup on the reference's default
        # median tree
        {"name": "occluded_soup_100k", "kind": "occluded", "scene": "soup", "size": 10_000, "tree": "median",
         "rays": 100_003},
        # the reference's own path tracer (Kajiya recursion) on a small frame
        # of odd size
        {"name": "paths_kajiya_401x299", "kind": "paths", "mode": "kajiya", "size": 16, "width": 401,
         "height": 299, "spp": 8, "depth": 6, "features": False},
        # the denoiser's input: one sample per pixel and the first-hit features
        {"name": "paths_1spp_512", "kind": "paths", "mode": "nee", "size": 16, "width": 512, "height": 512,
         "spp": 1, "depth": 8, "features": True},
        # the path-traced room of the benchmark (1024 x 1024, depth 8) at an
        # interactive sample count
        {"name": "paths_room_1024_16spp", "kind": "paths", "mode": "nee", "size": 53, "width": 1024,
         "height": 1024, "spp": 16, "depth": 8, "features": False},
        # many views of many scenes (data generation): uneven scenes and
        # resolutions in one launch
        {"name": "batch_12_scenes", "kind": "batch", "scenes": 12, "spp": 4, "depth": 6},
        # a preview-sized image of ragged tile counts through the denoiser
        {"name": "denoise_208x144", "kind": "denoise", "n": 1, "h": 144, "w": 208},
        # one frame of the evaluation size
        {"name": "denoise_512", "kind": "denoise", "n": 1, "h": 512, "w": 512},
        # eight frames per call (an animation)
        {"name": "denoise_8x512", "kind": "denoise", "n": 8, "h": 512, "w": 512},
        # one training batch: eight 128 x 128 crops
        {"name": "train_8x128", "kind": "train", "n": 8, "h": 128, "w": 128},
    ]


def _log(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> Dict:
    kind = rng.choice(["frame", "frame", "closest", "occluded", "paths", "paths", "batch", "denoise", "denoise",
                       "train"])
    if kind == "frame":
        scene = rng.choice(["soup", "sphere", "room"])
        return {"kind": kind, "scene": scene, "size": _size(rng, scene), "tree": rng.choice(["median", "sah"]),
                "width": _log(rng, 64, 1920), "height": _log(rng, 48, 1080), "lights": rng.randint(1, 3),
                "host": rng.random() < 0.3, "hits": rng.random() < 0.3}
    if kind in ("closest", "occluded"):
        scene = rng.choice(["soup", "sphere", "room"])
        return {"kind": kind, "scene": scene, "size": _size(rng, scene), "tree": rng.choice(["median", "sah"]),
                "rays": _log(rng, 1_000, 1_000_000)}
    if kind == "paths":
        mode = rng.choice(["kajiya", "nee"])
        w, h = _log(rng, 64, 1024), _log(rng, 48, 1024)
        most = (4 if mode == "kajiya" else 16) * (1 << 20)
        return {"kind": kind, "mode": mode, "size": _log(rng, 4, 53), "width": w, "height": h,
                "spp": _log(rng, 1, max(1, min(64, most // (w * h)))), "depth": rng.randint(1, 8),
                "features": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 12), "spp": rng.randint(1, 4), "depth": rng.randint(1, 6)}
    if kind == "denoise":
        h, w = 16 * _log(rng, 1, 32), 16 * _log(rng, 1, 32)
        return {"kind": kind, "n": _log(rng, 1, 8), "h": h, "w": w}
    h, w = 16 * _log(rng, 1, 12), 16 * _log(rng, 1, 12)
    return {"kind": "train", "n": _log(rng, 1, max(1, min(16, 8 * 128 * 128 // (h * w)))), "h": h, "w": w}


def _size(rng: random.Random, scene: str) -> int:
    return {"soup": _log(rng, 500, 50_000), "sphere": rng.randint(3, 7), "room": _log(rng, 4, 53)}[scene]


# -- scenes ------------------------------------------------------------------


@functools.lru_cache(maxsize=8)
def _mesh(scene: str, size: int) -> scenes.Mesh:
    if scene == "soup":
        return scenes.soup(size, 1)
    if scene == "sphere":
        return scenes.icosphere(size)
    return scenes.room(grid=size)


@functools.lru_cache(maxsize=4)
def _batch_meshes(n: int):
    # the benchmark's batch of spheres and soups, with the lighter half of its
    # range of triangle counts and resolutions
    return scenes.batch_workload(n, seed=3, median=20_000, hi=100_000, resolutions=(256, 384, 512))


def _triangles(scene: str, size: int) -> int:
    if scene == "soup":
        return size
    return 20 * 4 ** size if scene == "sphere" else 36 * size * size + 32


def _setup(case: Dict, rng: np.random.Generator) -> scenes.RenderSetup:
    """The camera and the lights of a view: near the benchmark's, moved by the seed."""
    w, h = case.get("width", 16), case.get("height", 16)
    scene = case.get("scene", "room")
    if scene == "soup":
        st = scenes.soup_setup(w, h)
    elif scene == "sphere":
        st = scenes.icosphere_setup(w, h)
    else:
        st = scenes.room_setup(w, h)
    d = rng.uniform(-0.05, 0.05, 6)
    st.cam_pos = tuple(float(p + q) for p, q in zip(st.cam_pos, d[:3] * (0.2 if scene == "room" else 1.0)))
    st.cam_look = tuple(float(p + q) for p, q in zip(st.cam_look, d[3:]))
    if "tree" in case:
        st.tree = case["tree"]
    if "lights" in case:
        at = rng.uniform(-1, 1, (case["lights"], 3))
        if scene == "room":
            at = at * np.array([0.8, 0.4, 0.8]) + np.array([0, 1.3, 0])
        else:
            at = at + np.array([0.5, 2.5, -2.0])
        st.lights = [tuple(float(x) for x in p) + (4.0, 4.0, 3.5) for p in at]
    return st


def _rays(case: Dict, gen: torch.Generator) -> torch.Tensor:
    """Rays (origin, unit direction, 1 / direction) from points spread through
    the scene: uniform directions in the room and the soup, towards the
    sphere from around it."""
    n = case["rays"]
    u = torch.rand((n, 3), generator=gen, device=DEVICE)
    d = torch.randn((n, 3), generator=gen, device=DEVICE)
    if case["scene"] == "room":
        o = u * torch.tensor([1.9, 1.9, 1.9], device=DEVICE) + torch.tensor([-0.95, 0.04, -0.95], device=DEVICE)
    elif case["scene"] == "soup":
        o = u
    else:
        p = torch.randn((n, 3), generator=gen, device=DEVICE)
        o = 2.5 * p / p.norm(dim=1, keepdim=True)
        d = 0.4 * d - o
    d = d / d.norm(dim=1, keepdim=True)
    return torch.cat([o, d, 1.0 / d], 1).contiguous()


# -- the network's weights and data -------------------------------------------


def _params(gen: torch.Generator) -> torch.Tensor:
    """Weights [cout][3][3][cin] then biases of the 19 convolutions, He-normal
    (the output convolution a tenth of it, as training starts)."""
    parts = []
    for i, (ci, co, _) in enumerate(denoise.CONVS):
        scale = (0.1 if i == len(denoise.CONVS) - 1 else 1.0) * math.sqrt(2.0 / (9 * ci))
        parts.append(scale * torch.randn(co * 9 * ci, generator=gen, device=DEVICE))
        parts.append(0.01 * torch.randn(co, generator=gen, device=DEVICE))
    return torch.cat(parts)


def _images(case: Dict, gen: torch.Generator):
    """Rendered-looking data: piecewise smooth albedo, normals and depth, a
    smooth target and a few-sample estimate of it with heavy-tailed noise."""
    n, h, w = case["n"], case["h"], case["w"]

    def smooth(c):
        g = torch.rand((n, c, h // 16 + 2, w // 16 + 2), generator=gen, device=DEVICE)
        return torch.nn.functional.interpolate(g, size=(h, w), mode="bilinear").permute(0, 2, 3, 1)

    albedo = torch.round(smooth(3) * 4) / 4 * 0.8 + 0.1
    normal = smooth(3) * 2 - 1
    normal = normal / normal.norm(dim=3, keepdim=True).clamp_min(1e-3)
    feat = torch.cat([albedo, normal, 1 + 2 * smooth(1)], 3).to(torch.float16).contiguous()
    target = (albedo * (0.2 + 2 * smooth(3))).contiguous()
    e = torch.rand((n, h, w, 3), generator=gen, device=DEVICE).clamp_min(1e-6)
    rad = (target * -torch.log(e)).contiguous()
    return rad, feat, target


# -- one pass ------------------------------------------------------------------


def prepare(case: Dict, seed: int) -> Dict:
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    new = lambda *shape, dtype: torch.zeros(shape, dtype=dtype, device=DEVICE)  # noqa: E731
    if kind == "frame":
        st = _setup(case, rng)
        w, h = st.width, st.height
        s = {"case": case, "setup": st, "scene": native.Scene.from_setup(_mesh(case["scene"], case["size"]), st)}
        if case["host"]:
            s["out"] = torch.zeros((h, w, 3), dtype=torch.uint8, pin_memory=True).numpy()
        else:
            s["rgb"] = new(h, w, 3, dtype=torch.uint8)
            s["ids"] = new(h, w, dtype=torch.int32) if case["hits"] else None
            s["ts"] = new(h, w, dtype=torch.float32) if case["hits"] else None
        return s
    if kind in ("closest", "occluded"):
        st = _setup(case, rng)
        rays = _rays(case, gen)
        n = case["rays"]
        s = {"case": case, "eps": st.det_eps, "rays": rays,
             "scene": native.Scene.from_setup(_mesh(case["scene"], case["size"]), st)}
        if kind == "closest":
            s["ids"], s["ts"] = new(n, dtype=torch.int32), new(n, dtype=torch.float32)
        else:
            s["dist2"] = (0.05 + torch.rand(n, generator=gen, device=DEVICE)) ** 2
            s["occluded"] = new(n, dtype=torch.uint8)
        return s
    if kind == "paths":
        st = _setup(case, rng)
        w, h = st.width, st.height
        mode = native.PT_NEE if case["mode"] == "nee" else native.PT_KAJIYA
        p = native.pt_params(st, spp=case["spp"], max_depth=case["depth"], seed=seed, mode=mode,
                             scheduler=native.SCHED_AUTO)
        return {"case": case, "params": p, "scene": native.Scene.from_setup(_mesh("room", case["size"]), st),
                "rgb": new(h, w, 3, dtype=torch.uint8), "radiance": new(h, w, 3, dtype=torch.float32),
                "features": new(h, w, 7, dtype=torch.float16) if case["features"] else None}
    if kind == "batch":
        items = _batch_meshes(case["scenes"])
        scs = [native.Scene.from_setup(m, st) for m, st in items]
        ps = [native.pt_params(st, spp=case["spp"], max_depth=case["depth"], seed=seed * 64 + i)
              for i, (_, st) in enumerate(items)]
        outs = [(new(st.height, st.width, 3, dtype=torch.uint8), new(st.height, st.width, 3, dtype=torch.float32))
                for _, st in items]
        b = native.Batch(scs, ps, outs)
        # the launch shape that the library's own tuner settles on for such batches
        b.set_config(native.BatchConfig(4, 8, 256, 0, 32))
        return {"case": case, "batch": b, "outs": outs}
    rad, feat, target = _images(case, gen)
    net = native.Denoiser()
    net.set_params(_params(gen).cpu().numpy())
    return {"case": case, "net": net, "rad": rad, "feat": feat, "target": target,
            "out": new(*rad.shape, dtype=torch.float32)}


def run(s: Dict):
    case = s["case"]
    kind = case["kind"]
    if kind == "frame":
        if case["host"]:
            img, rays = s["scene"].render_rt_host(s["setup"], out=s["out"])
            return {"rgb": img, "rays": rays.astype(np.int64)}
        s["scene"].render_rt(s["setup"], s["rgb"], s["ids"], s["ts"])
        return {"rgb": s["rgb"], "ids": s["ids"], "ts": s["ts"]}
    if kind == "closest":
        s["scene"].trace_closest(s["rays"], s["eps"], s["ids"], s["ts"])
        return {"ids": s["ids"], "ts": s["ts"]}
    if kind == "occluded":
        s["scene"].trace_occluded(s["rays"], s["dist2"], s["eps"], s["occluded"])
        return {"occluded": s["occluded"]}
    if kind == "paths":
        s["scene"].render_pt(s["params"], s["rgb"], s["radiance"])
        if s["features"] is not None:
            s["scene"].render_features(s["params"], s["features"])
        return {"rgb": s["rgb"], "radiance": s["radiance"], "features": s["features"]}
    if kind == "batch":
        s["batch"].render()
        return [list(o) for o in s["outs"]]
    if kind == "denoise":
        s["net"].denoise(s["rad"], s["feat"], s["out"])
        return {"out": s["out"]}
    loss, grads = s["net"].gradients(s["rad"], s["feat"], s["target"])
    return {"loss": loss, "grads": grads}


# -- what a pass cannot do without ----------------------------------------------


def _ray_flops(triangles: int) -> float:
    """One walk down a binary tree to a leaf of a few triangles: two box tests
    (18 operations each) per level and two triangle tests (about 45 each)."""
    return 36.0 * max(1.0, math.log2(max(2, triangles) / 4)) + 90.0


def work(case: Dict) -> Dict:
    kind = case["kind"]
    if kind == "frame":
        px, tris = case["width"] * case["height"], _triangles(case["scene"], case["size"])
        # the primary rays, and the occlusion rays of the half of the pixels
        # that see a lit surface; triangles (48 bytes) can be read at most
        # once per pixel
        return {"bytes": px * (3 + (8 if case["hits"] else 0)) + 48 * min(px, tris),
                "flops": px * (1 + 0.5 * case["lights"]) * _ray_flops(tris)}
    if kind in ("closest", "occluded"):
        n, tris = case["rays"], _triangles(case["scene"], case["size"])
        return {"bytes": n * (36 + (8 if kind == "closest" else 5)) + 48 * min(n, tris),
                "flops": n * _ray_flops(tris)}
    if kind == "paths":
        px, tris = case["width"] * case["height"], _triangles("room", case["size"])
        # segments per path in the closed room: every bounce and, with
        # next-event estimation, its occlusion ray (Russian roulette ends
        # about half of the paths after the third bounce)
        seg = case["depth"] + 1 if case["mode"] == "kajiya" else 2 * min(case["depth"], 4) + 1
        return {"bytes": px * (15 + (14 if case["features"] else 0)) + 48 * min(px, tris),
                "flops": px * case["spp"] * seg * _ray_flops(tris)}
    if kind == "batch":
        b = f = 0.0
        for m, st in _batch_meshes(case["scenes"]):
            px = st.width * st.height
            b += px * 15 + 48 * min(px, m.n)
            # about two segments per path: half of the pixels see the sky
            f += px * case["spp"] * 2 * _ray_flops(m.n)
        return {"bytes": b, "flops": f}
    n, h, w = case["n"], case["h"], case["w"]
    weights = 4 * denoise.num_params()
    if kind == "denoise":
        return {"bytes": n * h * w * (12 + 14 + 12) + weights, "flops": denoise.forward_flops(h, w, n)}
    # training: the weight gradients and (but for the first convolution) the
    # input gradients each cost a forward pass
    return {"bytes": n * h * w * (12 + 14 + 12) + 2 * weights, "flops": 3 * denoise.forward_flops(h, w, n)}


# -- 64-bit values -----------------------------------------------------------------


def _hits32(rays, a, e1, e2, eps):
    """Which triangles each ray hits: the one-sided test in single precision,
    every operation rounded by itself (n rays x m triangles)."""
    f = lambda x, k: x[:, k][None, :]  # noqa: E731
    r = lambda k: rays[:, k][:, None]  # noqa: E731
    ox, oy, oz, dx, dy, dz = (r(k) for k in range(6))
    px, py, pz = (dy * f(e2, 2) - dz * f(e2, 1), dz * f(e2, 0) - dx * f(e2, 2), dx * f(e2, 1) - dy * f(e2, 0))
    det = f(e1, 0) * px + f(e1, 1) * py + f(e1, 2) * pz
    inv = 1.0 / det
    tx, ty, tz = ox - f(a, 0), oy - f(a, 1), oz - f(a, 2)
    u = (tx * px + ty * py + tz * pz) * inv
    qx, qy, qz = (ty * f(e1, 2) - tz * f(e1, 1), tz * f(e1, 0) - tx * f(e1, 2), tx * f(e1, 1) - ty * f(e1, 0))
    v = (dx * qx + dy * qy + dz * qz) * inv
    t = (f(e2, 0) * qx + f(e2, 1) * qy + f(e2, 2) * qz) * inv
    return (det >= eps) & (det > 0) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > 0)


def _exact_distances(case: Dict, seed: int) -> Optional[torch.Tensor]:
    """Closest one-sided hits of every ray over every triangle, as matrix
    products: with n = e1 x e2 and m = o x d, det = -d.n, u det = e2.m - d.(e2 x a),
    v det = d.(e1 x a) - e1.m, t det = (o - a).n. Whether a ray that passes
    within rounding of an edge hits the triangle is the single-precision
    test's answer (_hits32), its distance is then taken in 64 bits all the same."""
    mesh = _mesh(case["scene"], case["size"])
    n = case["rays"]
    if n * mesh.n > 4e10:
        return None
    rng = np.random.default_rng(seed)
    eps = float(np.float32(_setup(case, rng).det_eps))
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    rays32 = _rays(case, gen)
    rays = rays32.double()
    v = torch.from_numpy(mesh.verts).to(DEVICE)
    a32, e1_32, e2_32 = v[:, 0:3], v[:, 3:6] - v[:, 0:3], v[:, 6:9] - v[:, 0:3]
    a, e1, e2 = a32.double(), e1_32.double(), e2_32.double()
    cross = lambda x, y: torch.cross(x, y, dim=1)  # noqa: E731
    nrm = cross(e1, e2)
    m_u = torch.cat([-cross(e2, a), e2], 1).T.contiguous()
    m_v = torch.cat([cross(e1, a), -e1], 1).T.contiguous()
    m_t = torch.cat([nrm, -(a * nrm).sum(1, keepdim=True)], 1).T.contiguous()
    far = float(np.finfo(np.float32).max)
    ts = torch.empty(n, dtype=torch.float64, device=DEVICE)

    def some(at):
        o, d = rays[at, 0:3], rays[at, 3:6]
        dm = torch.cat([d, cross(o, d)], 1)
        det = -(d @ nrm.T)
        t = (torch.cat([o, torch.ones_like(o[:, :1])], 1) @ m_t) / det
        return det, dm @ m_u, dm @ m_v, t

    step = max(1, int(2e8 // mesh.n))
    near = []
    for i in range(0, n, step):
        at = torch.arange(i, min(n, i + step), device=DEVICE)
        det, u, w, t = some(at)
        low = torch.minimum(torch.minimum(u, w), det - u - w) / det
        del u, w
        ok = (det >= eps) & (det > 0) & (low >= 0) & (t > 0)
        best = torch.where(ok, t, far).min(1).values
        ts[at] = best
        # candidates that rounding may decide, at or before that distance
        unsure = (det > 0) & (t < 1.001 * best[:, None]) & (low > -1e-4) & (t > -1e-4) & (det > 0.999 * eps) & (
            (low < 1e-4) | (t < 1e-4) | (det < 1.001 * eps))
        near.append(at[unsure.any(1)])
        del det, t, low, ok, unsure
    near = torch.cat(near)
    step = max(1, int(5e7 // mesh.n))
    for i in range(0, near.numel(), step):
        at = near[i:i + step]
        t = some(at)[3]
        ts[at] = torch.where(_hits32(rays32[at], a32, e1_32, e2_32, eps), t, far).min(1).values
    return ts


def _network(p: torch.Tensor, rad: torch.Tensor, feat: torch.Tensor) -> torch.Tensor:
    """The U-Net in the parameters' type: log(1 + demodulated radiance) of the
    estimate, NCHW (csrc/denoise_net.cpp's layers)."""
    f = torch.nn.functional
    demod = feat[..., 0:3].double().clamp_min(0) + np.float32(0.05).astype(np.float64)
    x0 = torch.cat([torch.log1p(rad.double().clamp_min(0) / demod), feat.double()], 3).permute(0, 3, 1, 2)
    at = 0
    k = 0

    def conv(x):
        nonlocal at, k
        ci, co, _ = denoise.CONVS[k]
        wt = p[at:at + co * 9 * ci].view(co, 3, 3, ci).permute(0, 3, 1, 2)
        b = p[at + co * 9 * ci:at + co * 9 * ci + co]
        at += co * 9 * ci + co
        k += 1
        # as one matrix product per image (64-bit convolutions by the library
        # are slow)
        n, _, h, w = x.shape
        out = []
        for i in range(n):
            cols = f.unfold(x[i:i + 1], 3, padding=1)[0]
            out.append((wt.reshape(co, -1) @ cols + b[:, None]).view(1, co, h, w))
        y = torch.cat(out)
        return torch.relu(y) if k < len(denoise.CONVS) else y

    x, skips = x0, []
    for level in range(5):
        x = conv(conv(x))
        if level < 4:
            skips.append(x)
            x = f.avg_pool2d(x, 2)
    for level in range(3, -1, -1):
        x = torch.cat([f.interpolate(x, scale_factor=2, mode="nearest"), skips[level]], 1)
        x = conv(conv(x))
    return conv(x) + x0[:, 0:3], demod


def exact(case: Dict, seed: int):
    kind = case["kind"]
    if kind == "closest":
        return {"ids": None, "ts": _exact_distances(case, seed)}
    if kind not in ("denoise", "train"):
        # bytes and whole numbers; a path-traced frame's radiance is the
        # estimate of one 32-bit random stream, whose hits and branches
        # another precision would not repeat
        return None
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    rad, feat, target = _images(case, gen)
    p = _params(gen).double()
    if kind == "denoise":
        with torch.no_grad():
            outs = []
            for i in range(case["n"]):
                y, demod = _network(p, rad[i:i + 1], feat[i:i + 1])
                outs.append(torch.expm1(y).permute(0, 2, 3, 1) * demod)
            return {"out": torch.cat(outs)}
    p.requires_grad_(True)
    total = 0.0
    for i in range(case["n"]):
        y, demod = _network(p, rad[i:i + 1], feat[i:i + 1])
        want = torch.log1p(target[i:i + 1].double().clamp_min(0) / demod)
        loss = (y.permute(0, 2, 3, 1) - want).abs().sum() / target.numel()
        loss.backward()
        total += float(loss)
    return {"loss": total, "grads": p.grad.detach()}
