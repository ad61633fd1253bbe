"""Measured workloads of the frame path, through the entry points that a program calls.

A case is one pass of one of these:

  frame  Renderer.render: the next frame of a camera orbit into caller-owned buffers
  loop   FrameLoop.step: the same plus the post-process (progressive or TAA) and the u8 frame
  batch  Batch.render: many views of one scene, each with its own size and samples per pixel
  scan   gps_workload_scan_noalloc: one pass's point offsets for a host that owns every buffer
  taa    gps_post_taa: the temporal post-process alone, on a program's own colour and depth

Scenes are the two kinds that synth.py describes (a cube of random Gaussians, a town of flat ones
on a ground plane and boxes), generated here on the GPU from the seed.  A renderer draws random
samples whose number depends on single-precision roundings, so its images have no 64-bit value to
compare with (one count that rounds the other way gives all later samples other random numbers):
exact() covers the arithmetic paths.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "gaussian-point-splatting_b200"))

import gpsplat  # noqa: E402
import synth  # noqa: E402

DEV = "cuda"
FORMATS = {"fp32": gpsplat.GPS_SCENE_FP32, "compressed": gpsplat.GPS_SCENE_COMPRESSED, "half": gpsplat.GPS_SCENE_HALF}
GEOMETRY_BYTES = {"fp32": 48, "compressed": 17, "half": 32}
SH_BYTES = {"fp32": 192, "compressed": 64, "half": 48}

# Every key that a frame or loop case may carry, with the library's own default where it has one.
FRAME = dict(kind="frame", scene="town", n=60000, tiles=1, format="fp32", width=1920, height=1080, ss=2, spp=1,
             reduce=True, unbiased=True, culling=True, occlusion=True, cull_small=False, post="progressive")


def _frame(name, **kw):
    return dict(FRAME, name=name, **kw)


def listed():
    return [
        # a thumbnail of a small scene: the smallest call, all launches and latency
        _frame("cube20k_160x90", scene="cube", n=20_000, width=160, height=90, ss=1, culling=False, occlusion=False),
        # a preview pane of a small scene with everything on: two passes, culling, Hi-Z
        _frame("town60k_320x180_spp4", n=60_000, width=320, height=180, spp=4),
        # the first benchmark configuration: a million Gaussians, 640 x 360, no culling
        _frame("cube1m_640x360", scene="cube", n=1_000_000, width=640, height=360, ss=1, culling=False, occlusion=False),
        # the viewer's defaults (compressed scene, ss 2, 1 sample, progressive) in a 720p window, odd scene size
        _frame("town500k_720p_progressive", kind="loop", n=500_123, format="compressed", width=1280, height=720),
        # the headline view: 1080p, ss 2, 4 samples, culling, TAA, one keyframe of the orbit per frame
        _frame("town4m_1080p_taa", kind="loop", n=4_000_000, spp=4, post="taa"),
        # a large scene in the half format, tiled from a smaller one, crossing the scan's big-scene size
        _frame("town33m_half_1080p_taa", kind="loop", n=2_100_000, tiles=16, format="half", spp=4, post="taa"),
        # a 4K frame (531 MB splat buffer)
        _frame("town1m_4k_spp2", n=1_000_000, width=3840, height=2160, spp=2),
        # an odd window with one point per thread and a sample count that is no power of two
        _frame("town700k_odd_onepoint", n=700_001, width=1237, height=689, spp=3, reduce=False),
        # the biased splat with small Gaussians culled, no supersampling
        _frame("town300k_biased", n=300_000, width=999, height=571, ss=1, spp=4, unbiased=False, cull_small=True),
        # an offline batch: 16 views of mixed sizes and samples of one scene
        dict(name="batch16_town1m", kind="batch", n=1_000_000, views=16, workers=4, max_spp=8),
        # one pass's point offsets at the size of a large scene
        dict(name="scan_20m", kind="scan", n=20_000_000, density=0.1),
        # the temporal post-process at 4K
        dict(name="taa_4k", kind="taa", width=3840, height=2160),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["frame", "loop", "batch", "scan", "taa"], [5, 4, 1, 1, 1])[0]
    if kind == "scan":
        return dict(kind=kind, n=_log(rng, 10_000, 36_000_000), density=rng.choice([0.01, 0.1, 0.5]))
    if kind == "taa":
        h = _log(rng, 90, 2160)
        return dict(kind=kind, width=int(h * rng.uniform(1.2, 1.78)), height=h)
    if kind == "batch":
        return dict(kind=kind, n=_log(rng, 50_000, 1_500_000), views=rng.randint(2, 16), workers=rng.choice([1, 2, 4]),
                    max_spp=rng.choice([1, 4, 8]))
    c = dict(FRAME, kind=kind, scene=rng.choice(["town", "town", "town", "cube"]), n=_log(rng, 8_000, 2_500_000),
             format=rng.choice(["fp32", "fp32", "compressed", "half"]), height=_log(rng, 90, 1440),
             ss=rng.choice([1, 2, 2, 2, 3]), spp=rng.choice([1, 1, 2, 3, 4, 8]), reduce=rng.random() < 0.8,
             unbiased=rng.random() < 0.85, culling=rng.random() < 0.75, occlusion=rng.random() < 0.75,
             cull_small=rng.random() < 0.15, post=rng.choice(["progressive", "taa", "none"]))
    c["width"] = int(c["height"] * rng.uniform(1.3, 1.85))
    if c["format"] == "half" and rng.random() < 0.5:
        c["n"] -= c["n"] % 16
        c["tiles"] = rng.choice([4, 9])
        c["scene"] = "town"
    while c["width"] * c["height"] * c["ss"] ** 2 * c["spp"] > 30_000_000 and c["spp"] > 1:
        c["spp"] -= 1
    return c


# ---------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _activated(pos, dc, rest, logit, log_scale, quat):
    """The CPUGaussian layout: mean 3, sh 48, opacity, scale 3, rotation 4."""
    n = pos.shape[0]
    out = torch.zeros((n, gpsplat.GAUSSIAN_FLOATS), device=DEV)
    out[:, 0:3] = pos
    out[:, 3:6] = dc
    if rest is not None:
        out[:, 6:51] = rest
    out[:, 51] = torch.sigmoid(logit)
    out[:, 52:55] = torch.exp(log_scale)
    out[:, 55:59] = quat / quat.norm(dim=1, keepdim=True)
    return out


def _cube(n, gen):
    u = lambda *s: torch.rand(s, generator=gen, device=DEV)  # noqa: E731
    g = lambda *s: torch.randn(s, generator=gen, device=DEV)  # noqa: E731
    return _activated(u(n, 3) * 20.0 - 10.0, u(n, 3), None, 1.5 * g(n), 0.5 * g(n, 3) - 3.0, g(n, 4))


def _town(n, gen, seed):
    """synth.town's distribution: surfaces by area, flat Gaussians, random in-plane rotation, Morton order."""
    foot, height, centre = synth.town_boxes(int(seed))
    half = synth.TOWN_EXTENT / 2
    # every surface as origin + a * e0 + b * e1, normal along e0 x e1; ground first
    org, e0, e1 = [(-half, 0.0, -half)], [(2 * half, 0.0, 0.0)], [(0.0, 0.0, 2 * half)]
    for (w, d), h, (cx, cz) in zip(foot, height, centre):
        x0, x1, z0, z1 = cx - w / 2, cx + w / 2, cz - d / 2, cz + d / 2
        for o, a, b in (((x1, 0, z0), (0, 0, d), (0, h, 0)), ((x0, 0, z0), (0, 0, d), (0, h, 0)),
                        ((x0, 0, z1), (w, 0, 0), (0, h, 0)), ((x0, 0, z0), (w, 0, 0), (0, h, 0)),
                        ((x0, h, z0), (w, 0, 0), (0, 0, d))):
            org.append(o), e0.append(a), e1.append(b)
    org, e0, e1 = (torch.tensor(np.array(v, np.float64), dtype=torch.float32, device=DEV) for v in (org, e0, e1))
    area = torch.linalg.cross(e0, e1).norm(dim=1).double()
    cdf = torch.cumsum(area / area.sum(), 0)
    u = lambda *s: torch.rand(s, generator=gen, device=DEV)  # noqa: E731
    g = lambda *s: torch.randn(s, generator=gen, device=DEV)  # noqa: E731
    f = torch.searchsorted(cdf, u(n).double()).clamp_(max=len(area) - 1)
    pos = org[f] + u(n, 1) * e0[f] + u(n, 1) * e1[f]
    cell = ((pos - pos.amin(0)) / (pos.amax(0) - pos.amin(0)) * 1023.0).long()
    code = torch.zeros(n, dtype=torch.long, device=DEV)
    for b in range(10):
        for axis in range(3):
            code |= ((cell[:, axis] >> b) & 1) << (3 * b + axis)
    order = torch.argsort(code, stable=True)
    pos, f = pos[order], f[order]
    t, nrm = e0 / e0.norm(dim=1, keepdim=True), torch.linalg.cross(e0, e1)
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    # the quaternion (w, x, y, z) of each surface's frame, then a random turn about its normal
    base = torch.tensor(np.stack([_quaternion(m) for m in torch.stack([t, torch.linalg.cross(nrm, t), nrm], 2).cpu().numpy()]),
                        dtype=torch.float32, device=DEV)[f]
    half_turn = math.pi * u(n)
    c, s = torch.cos(half_turn), torch.sin(half_turn)
    w, x, y, z = base.unbind(1)
    quat = torch.stack([w * c - z * s, x * c + y * s, y * c - x * s, z * c + w * s], 1)
    scale = torch.cat([0.5 * g(n, 2) - 3.0, 0.3 * g(n, 1) - 6.0], 1)
    return _activated(pos, u(n, 3), 0.2 * g(n, 45), 2.0 + g(n), scale, quat)


def _quaternion(m):
    """(w, x, y, z) of a rotation matrix, from the eigenvector of its symmetric 4 x 4 form."""
    k = np.array([[m[0, 0] + m[1, 1] + m[2, 2], m[2, 1] - m[1, 2], m[0, 2] - m[2, 0], m[1, 0] - m[0, 1]],
                  [0, m[0, 0] - m[1, 1] - m[2, 2], m[0, 1] + m[1, 0], m[0, 2] + m[2, 0]],
                  [0, 0, m[1, 1] - m[0, 0] - m[2, 2], m[1, 2] + m[2, 1]],
                  [0, 0, 0, m[2, 2] - m[0, 0] - m[1, 1]]], np.float64)
    return np.linalg.eigh(np.triu(k) + np.triu(k, 1).T)[1][:, -1]


def _scene(case, seed):
    gen = _generator(seed)
    g = _cube(case["n"], gen) if case.get("scene") == "cube" else _town(case["n"], gen, seed)
    scene = gpsplat.Scene.from_host(g.cpu().numpy(), FORMATS[case.get("format", "fp32")], presorted=True)
    side = int(math.isqrt(case.get("tiles", 1)))
    if side > 1:
        step = synth.TOWN_EXTENT
        scene = scene.tile([((i - (side - 1) / 2) * step, (j - (side - 1) / 2) * step) for i in range(side) for j in range(side)])
    return scene


def _cameras(case, settings, seed, count=24):
    """Consecutive keyframes of a 120-frame orbit (of the cube: around its outside), from a phase of the seed."""
    rng = np.random.default_rng(seed)
    if case.get("scene") == "cube":
        poses = synth.orbit(120, 30.0, 4.0)
    else:
        poses = synth.orbit(120, 30.0, 10.0)
    phase = int(rng.integers(120))
    cams = []
    for i in range(count):
        p, r = poses[(phase + i) % 120]
        cam = gpsplat.camera_from_pose(p, np.asarray(r, np.float32).T, settings, i + 1)
        cam.camera_moved = 1
        cams.append(cam)
    return cams


class _Device:
    """A device buffer of the library's as an array that torch reads in place; keeps its owner alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _prepare_frame(case, seed):
    s = gpsplat.default_settings(
        width=case["width"], height=case["height"], supersampling_factor=case["ss"], samples_per_pixel=case["spp"],
        reduce_point_count=int(case["reduce"]), use_unbiased_2d_splatting=int(case["unbiased"]),
        cull_small_gaussians=int(case["cull_small"]), enable_occlusion_culling=int(case["occlusion"]),
        enable_hierarchical_culling=int(case["culling"]), fully_disable_hierarchical_culling=int(not case["culling"]),
        accumulation_mode={"progressive": gpsplat.GPS_ACCUM_PROGRESSIVE, "taa": gpsplat.GPS_ACCUM_TAA,
                           "none": gpsplat.GPS_ACCUM_NONE}[case["post"]])
    scene = _scene(case, seed)
    renderer = gpsplat.Renderer(scene, s)
    st = dict(kind=case["kind"], renderer=renderer, cams=_cameras(case, s, seed), next=0, shape=(s.height, s.width))
    if case["kind"] == "loop":
        st["loop"] = gpsplat.FrameLoop(renderer)
    else:
        st["image"] = torch.zeros((s.height, s.width, 3), device=DEV)
        st["depth"] = torch.zeros((s.height, s.width), device=DEV)
    return st


def _prepare_batch(case, seed):
    rng = np.random.default_rng(seed)
    sizes = [(320, 180), (640, 360), (961, 541), (1280, 720), (1920, 1080)]
    scene = _scene(case, seed)
    s = gpsplat.default_settings(width=1920, height=1080, samples_per_pixel=case["max_spp"])
    batch = gpsplat.Batch(scene, s, 1920, 1080, case["max_spp"], workers=case["workers"])
    entries, outs = [], []
    poses = synth.random_poses(case["views"], seed=int(rng.integers(1 << 30)))
    for i, (p, r) in enumerate(poses):  # the sizes and sample counts in turn: equal work for every seed
        w, h = sizes[i % len(sizes)]
        spp = min(case["max_spp"], (1, 4, 2, 8)[i % 4])
        vs = gpsplat.default_settings(width=w, height=h)
        cam = gpsplat.camera_from_pose(p, np.asarray(r, np.float32).T, vs, i + 1)
        image, depth = torch.zeros((h, w, 3), device=DEV), torch.zeros((h, w), device=DEV)
        outs.append((image, depth))
        entries.append((cam, w, h, spp, image.data_ptr(), depth.data_ptr()))
    return dict(kind="batch", batch=batch, scene=scene, views=gpsplat.Batch.views(entries), outs=outs)


def _prepare_scan(case, seed):
    n, gen = case["n"], _generator(seed)
    pad = (n + 31) // 32 * 32
    on = torch.rand(pad, generator=gen, device=DEV) < case["density"]
    on[n:] = False
    counts = torch.where(on, torch.randint(1, 40, (pad,), generator=gen, device=DEV), 0).to(torch.int32)
    bits = on.view(-1, 32).to(torch.int64) << torch.arange(32, device=DEV)
    mask = bits.sum(1)
    mask = torch.where(mask >= 1 << 31, mask - (1 << 32), mask).to(torch.int32)
    cap = 250_000_000
    # entries past the survivors (and past the last tile) are not written: zeroed once here
    st = dict(kind="scan", n=n, cap=cap, counts=counts, mask=mask)
    for key, size in (("gid", n), ("start", n), ("tile", cap // 256 + 2), ("counters", 8)):
        st[key] = torch.zeros(size, dtype=torch.int32, device=DEV)
    return st


def _prepare_taa(case, seed):
    w, h, gen = case["width"], case["height"], _generator(seed)
    u = lambda *s: torch.rand(s, generator=gen, device=DEV)  # noqa: E731
    s = gpsplat.default_settings(width=w, height=h)
    # history and current frame of one slowly turning view: similar colours, depths near the far end
    prev = u(h, w, 3)
    cur = (prev + 0.1 * (u(h, w, 3) - 0.5)).clamp(0.0, 1.2)
    depth, prev_depth = 0.95 + 0.05 * u(h, w), 0.95 + 0.05 * u(h, w)
    k = int(torch.randint(120, (1,), generator=gen, device=DEV))
    vp = []
    for i in (k, k + 1):
        p, r = synth.orbit(720, 30.0, 10.0)[i]
        c = gpsplat.camera_to_numpy(gpsplat.camera_from_pose(p, np.asarray(r, np.float32).T, s, 1))
        vp.append(c["proj"].reshape(4, 4).T.astype(np.float64) @ c["view"].reshape(4, 4).T.astype(np.float64))
    reproj = (vp[0] @ np.linalg.inv(vp[1])).T.astype(np.float32).reshape(-1)  # column-major
    return dict(kind="taa", w=w, h=h, cur=cur, prev=prev, depth=depth, prev_depth=prev_depth, reproj=reproj,
                reproj_arg=(ctypes.c_float * 16)(*reproj.tolist()), image=torch.zeros((h, w, 3), dtype=torch.uint8, device=DEV),
                out=torch.zeros((h, w, 3), device=DEV))


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("frame", "loop"):
        return _prepare_frame(case, seed)
    return {"batch": _prepare_batch, "scan": _prepare_scan, "taa": _prepare_taa}[kind](case, seed)


# ---------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------
def run(st):
    kind = st["kind"]
    if kind == "frame":
        cam = st["cams"][st["next"] % len(st["cams"])]
        st["next"] += 1
        st["renderer"].render(cam, st["image"].data_ptr(), st["depth"].data_ptr(), _stream())
        return st["image"], st["depth"]
    if kind == "loop":
        cam = st["cams"][st["next"] % len(st["cams"])]
        st["next"] += 1
        loop, (h, w) = st["loop"], st["shape"]
        loop.step(cam, _stream())
        u8, color, _ = loop.buffers(cam.frame % 2)
        depth = loop.buffers(1 - cam.frame % 2)[2]
        return tuple(torch.as_tensor(_Device(loop, *a), device=DEV) for a in
                     ((u8, (h, w, 3), "|u1"), (color, (h, w, 3), "<f4"), (depth, (h, w), "<f4")))
    if kind == "batch":
        st["batch"].render(st["views"], _stream())
        return st["outs"]
    if kind == "scan":
        status = gpsplat.load_library().gps_workload_scan_noalloc(
            st["counts"].data_ptr(), st["mask"].data_ptr(), st["n"], st["cap"], st["gid"].data_ptr(),
            st["start"].data_ptr(), st["tile"].data_ptr(), st["counters"].data_ptr(), _stream())
        assert status == 0
        return st["gid"], st["start"], st["tile"], st["counters"]
    status = gpsplat.load_library().gps_post_taa(
        st["image"].data_ptr(), st["out"].data_ptr(), st["cur"].data_ptr(), st["prev"].data_ptr(), st["depth"].data_ptr(),
        st["prev_depth"].data_ptr(), st["reproj_arg"], 0.9, st["w"], st["h"], 1, _stream())
    assert status == 0
    return st["image"], st["out"]


# ---------------------------------------------------------------------------------
# what a pass cannot do without, and its value in 64 bits
# ---------------------------------------------------------------------------------
def _frame_work(n, fmt, w, h, ss, spp, culling, passes):
    """Bytes: the Gaussians in view once (all of them without culling; with it the block boxes and about a
    tenth of a town, as its orbit sees it), SH for half of those, one 8-byte key per sample slot, colour and
    depth out.  Operations: about five draws of 100 per slot."""
    share = 0.1 if culling else 1.0
    scene = n * share * (GEOMETRY_BYTES[fmt] + 0.5 * SH_BYTES[fmt]) + (n / 4.0 * 32 if culling else 0)
    slots = w * h * ss * ss * spp
    return scene + 8.0 * slots + 16.0 * w * h, 500.0 * slots


def work(case):
    kind = case["kind"]
    if kind in ("frame", "loop"):
        b, f = _frame_work(case["n"] * case["tiles"], case["format"], case["width"], case["height"], case["ss"],
                           case["spp"], case["culling"], 2 if case["occlusion"] else 1)
        if kind == "loop":  # colour in and out, history in, u8 out
            b += (12 + 12 + 3) * case["width"] * case["height"]
        return {"bytes": b, "flops": f}
    if kind == "batch":
        b = f = 0.0
        for i in range(case["views"]):
            w, h = [(320, 180), (640, 360), (961, 541), (1280, 720), (1920, 1080)][i % 5]
            x, y = _frame_work(case["n"], "fp32", w, h, 2, min(case["max_spp"], (1, 4, 2, 8)[i % 4]), True, 2)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    if kind == "scan":  # the mask, the counts of the survivors, their ids and first points
        n, live = case["n"], case["n"] * case["density"]
        return {"bytes": n / 8 + live * 12 + live * 20 / 256 * 4, "flops": 2.0 * live}
    px = case["width"] * case["height"]
    return {"bytes": px * (12 + 12 + 4 + 12 + 3), "flops": px * 120.0}


def _exact_taa(case, seed):
    st = _prepare_taa(case, seed)
    w, h = case["width"], case["height"]
    cur, prev, depth = st["cur"].double(), st["prev"].double(), st["depth"].double()
    m = torch.tensor(st["reproj"], device=DEV).double().view(4, 4).T
    y, x = torch.meshgrid(torch.arange(h, device=DEV).double(), torch.arange(w, device=DEV).double(), indexing="ij")
    clip = torch.stack([(x + 0.5) / w * 2 - 1, (y + 0.5) / h * 2 - 1, depth, torch.ones_like(depth)], -1)
    p = clip @ m.T
    px, py = ((p[..., 0] / p[..., 3]) * 0.5 + 0.5) * w - 0.5, ((p[..., 1] / p[..., 3]) * 0.5 + 0.5) * h - 0.5
    inside = (px >= 0) & (px < w) & (py >= 0) & (py < h)
    fx, fy = px.floor(), py.floor()
    x0, x1 = fx.clamp(0, w - 1).long(), (fx + 1).clamp(0, w - 1).long()
    y0, y1 = fy.clamp(0, h - 1).long(), (fy + 1).clamp(0, h - 1).long()
    tx, ty = (px - fx).unsqueeze(-1), (py - fy).unsqueeze(-1)
    top, bottom = prev[y0, x0] * (1 - tx) + prev[y0, x1] * tx, prev[y1, x0] * (1 - tx) + prev[y1, x1] * tx
    hist = top * (1 - ty) + bottom * ty
    c = cur.permute(2, 0, 1).unsqueeze(0)
    hi = torch.nn.functional.max_pool2d(c, 3, 1, 1)[0].permute(1, 2, 0)
    lo = -torch.nn.functional.max_pool2d(-c, 3, 1, 1)[0].permute(1, 2, 0)
    hist = torch.minimum(torch.maximum(hist, lo - 0.05), hi + 0.05)
    return None, torch.where(inside.unsqueeze(-1), cur * (1 - 0.9) + hist * 0.9, cur)


def exact(case, seed):
    return _exact_taa(case, seed) if case["kind"] == "taa" else None
