"""The block cull bit for bit, both passes: numpy in single precision with the sums of both tests in the
rounding that the kernels spell out (fused steps through round-to-odd in 64 bits), and the division
and the logarithm of the Hi-Z level, which are approximate, from the device."""
import ctypes
import os

import numpy as np
import pytest

import gpsplat
import gpsutil
import synth
from test_gpu_resolve import _chain

pytestmark = pytest.mark.gpu

F = np.float32


def _library():
    gpsplat.load_library()
    return ctypes.CDLL(os.path.join(gpsutil.PKG, "libgps_check.so"))


def _fma(a, b, c):
    """float32 a * b + c rounded once: the 64-bit sum is forced to an odd last bit where it is inexact."""
    p, c = a.astype(np.float64) * b, np.broadcast_to(c, np.broadcast(a, b, c).shape).astype(np.float64)
    s = p + c
    t = s - p
    err = (p - (s - t)) + (c - t)
    even = (s.view(np.int64) & 1) == 0
    return np.where((err != 0) & even, np.nextafter(s, np.where(err > 0, np.inf, -np.inf)), s).astype(F)


def _divide(a, b):
    a, b = np.ascontiguousarray(a, F), np.ascontiguousarray(np.broadcast_to(b, a.shape), F)
    out = np.empty_like(a)
    ptr = [v.ctypes.data_as(ctypes.c_void_p) for v in (a, b, out)]
    assert _library().gps_check_divide(ptr[0], ptr[1], ctypes.c_uint32(a.size), ptr[2]) == 0
    return out


def _hiz_level(extent):
    table = np.empty(int(extent.max()) + 1, np.int32)
    assert _library().gps_check_hiz_levels(ctypes.c_uint32(table.size), table.ctypes.data_as(ctypes.c_void_p)) == 0
    return table[extent]


def _outside(nodes, planes):
    out = np.zeros(len(nodes), bool)
    for n in planes.reshape(6, 4).astype(F):
        v = np.where(n[:3] >= 0, nodes[:, 4:7], nodes[:, 0:3])
        s = _fma(n[2], v[:, 2], _fma(n[0], v[:, 0], n[1] * v[:, 1])) + n[3]
        out |= s < 0
    return out


def _row(m, r, v, fused=True):
    """Row r of view-projection * (v, 1)."""
    a, b, c, d = (F(m[4 * k + r]) for k in range(4))
    x, y, z = v[:, 0], v[:, 1], v[:, 2]
    if not fused:  # the compiler's other choice: the left product rounded, the right one fused
        return _fma(b, y, a * x) + _fma(c, z, np.full_like(x, d))
    return _fma(a, x, b * y) + _fma(c, z, np.full_like(x, d))


def _pixel(ndc, size):
    v = (ndc * F(0.5) + F(0.5)) * F(size)
    with np.errstate(invalid="ignore"):
        return np.clip(np.trunc(v.astype(np.float64)), -(2**31), 2**31 - 1).astype(np.int64)


def _occluded(nodes, vp, levels, w, h, fused=True):
    """levels: finest first."""
    lo = np.full((len(nodes), 2), 0)
    lo[:, 0], lo[:, 1] = w - 1, h - 1
    hi = np.zeros((len(nodes), 2), np.int64)
    front, any_front = np.full(len(nodes), F(1e30)), np.zeros(len(nodes), bool)
    for i in range(8):
        v = np.stack([nodes[:, (4 if (i >> k) & 1 else 0) + k] for k in range(3)], 1)
        cx, cy, cz, cw = (_row(vp, r, v, fused) for r in range(4))
        ok = cw > 0
        safe = np.where(ok, cw, F(1))
        px, py, z = _pixel(_divide(cx, safe), w), _pixel(_divide(cy, safe), h), _divide(cz, safe)
        any_front |= ok
        lo[:, 0], lo[:, 1] = np.where(ok, np.minimum(lo[:, 0], px), lo[:, 0]), np.where(ok, np.minimum(lo[:, 1], py), lo[:, 1])
        hi[:, 0], hi[:, 1] = np.where(ok, np.maximum(hi[:, 0], px), hi[:, 0]), np.where(ok, np.maximum(hi[:, 1], py), hi[:, 1])
        front = np.where(ok, np.minimum(front, z), front)
    lo, hi = np.maximum(lo, 0), np.minimum(hi, [w - 1, h - 1])
    seen = any_front & (lo <= hi).all(1)
    lo, hi = np.where(seen[:, None], lo, 0), np.where(seen[:, None], hi, 0)
    lod = np.clip(_hiz_level((hi - lo + 1).max(1)), 0, len(levels) - 1)
    out = np.zeros(len(nodes), bool)
    for j, level in enumerate(levels):
        at = seen & (lod == j)
        tw, th = max(1, min(w, 1 << j)), max(1, min(h, 1 << j))
        x0, x1 = (np.clip(c[at, 0] // tw, 0, level.shape[1] - 1) for c in (lo, hi))
        y0, y1 = (np.clip(c[at, 1] // th, 0, level.shape[0] - 1) for c in (lo, hi))
        zmax = np.maximum(np.maximum(level[y0, x0], level[y0, x1]), np.maximum(level[y1, x0], level[y1, x1]))
        out[at] = zmax < front[at]
    return out


def _camera(seed):
    s = gpsplat.default_settings(width=640, height=360)
    p, r = synth.random_poses(1, seed=seed)[0]
    cam = gpsplat.camera_from_pose(p, np.asarray(r, F).T, s, 1)
    c = gpsplat.camera_to_numpy(cam)
    view, proj = (c[k].reshape(4, 4).T.astype(np.float64) for k in ("view", "proj"))
    return np.array(list(cam.frustum_planes), F), (proj @ view).T.astype(F).ravel(), np.asarray(p, np.float64)


def _nodes(count, planes, vp, eye, rng, depth):
    """Boxes of many sizes around points of three kinds: anywhere, on a plane of the frustum, and at
    the NDC depth `depth` within a few of its last places."""
    inv = np.linalg.inv(vp.astype(np.float64).reshape(4, 4).T)
    third = count // 3
    any_ = eye + rng.normal(0, 60, (third, 3))
    ndc = np.concatenate([rng.uniform(-1.2, 1.2, (count - third, 2)), rng.uniform(0.9, 0.9999, (count - third, 1)), np.ones((count - third, 1))], 1)
    ndc[third:, 2] = depth * (1 + rng.normal(0, 3e-7, count - 2 * third))
    p = ndc @ inv.T
    p = p[:, :3] / p[:, 3:]
    on = p[:third]
    k = rng.integers(0, 6, third)
    n = planes.reshape(6, 4).astype(np.float64)[k]
    on = on - (((on * n[:, :3]).sum(1) + n[:, 3]) / (n[:, :3] ** 2).sum(1))[:, None] * n[:, :3]
    c = np.concatenate([any_, on, p[third:]])
    size = np.exp(rng.uniform(-9, 1, (count, 3)))
    nodes = np.zeros((count, 8), F)
    nodes[:, 0:3], nodes[:, 4:7] = c - size, c + size
    exact = rng.random(count) < 0.5  # boxes with their corner at the point itself
    grow = (rng.random((count, 3)) < 0.5) * size
    nodes[exact, 0:3], nodes[exact, 4:7] = (c - grow)[exact], (c - grow + size)[exact]
    return nodes[rng.permutation(count)] if count > 100 else nodes


@pytest.mark.parametrize("count,per_block,short", [(1, 4, 3), (31, 4, 0), (33, 5, 2), (65, 33, 1), (1000, 7, 6), (200_000, 4, 1),
                                                   (120_000, 5, 3), (30_001, 33, 32)])
def test_both_passes(count, per_block, short):
    rng = np.random.default_rng(count)
    planes, vp, eye = _camera(count % 7)
    w, h, n = 640, 360, count * per_block - short
    flat = F(0.97)
    nodes = _nodes(count, planes, vp, eye, rng, float(flat))
    if count >= 1000:
        nodes[rng.integers(0, count, 5), rng.integers(0, 3, 5)] = np.nan  # no box of 32 may hide what is in it
        nodes[rng.integers(0, count, 5), 4 + rng.integers(0, 3, 5)] = np.inf
    first = [np.full_like(d, flat) for d in _chain(np.zeros((h, w), F), 0)]
    second = _chain(rng.uniform(0.9, 1.0, (h, w)).astype(F) ** 3, 0)
    chunks, words = (n + 31) // 32, (count + 31) // 32
    mips = [np.concatenate([d.ravel() for d in chain[::-1]]) for chain in (first, second)]
    out = {k: [np.zeros(size, np.uint32) for _ in range(2)] for k, size in (("culled", words), ("list", chunks), ("mask", chunks))}
    lengths = np.zeros(2, np.uint32)
    pair = lambda arrays: (ctypes.c_void_p * 2)(*(v.ctypes.data for v in arrays))  # noqa: E731
    ptr = lambda v: v.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    assert _library().gps_check_cull(ptr(nodes), ctypes.c_uint32(count), ctypes.c_uint32(per_block), ctypes.c_uint32(n), ptr(planes), ptr(vp),
                                     pair(mips), w, h, pair(out["culled"]), pair(out["list"]), pair(out["mask"]), ptr(lengths)) == 0
    with np.errstate(invalid="ignore", over="ignore"):
        outside = _outside(nodes, planes)
        finite = np.isfinite(nodes).all(1)
        for k, levels in enumerate((first, second)):
            want = outside | (~outside & _occluded(nodes, vp, levels, w, h))
            bits = np.unpackbits(out["culled"][k].view(np.uint8), bitorder="little")
            assert not bits[count:].any()
            got = bits[:count].astype(bool)
            assert np.array_equal(got[finite], want[finite])
            of = np.arange(n) // per_block
            visible = np.zeros(chunks, bool)
            np.logical_or.at(visible, np.arange(n) // 32, ~got[of])
            assert np.array_equal(np.sort(out["list"][k][: lengths[k]]), np.flatnonzero(visible))
            assert np.array_equal(out["mask"][k], np.where(visible, 0xFFFFFFFF, 0).astype(np.uint32))
        if count > 100_000:  # the boxes tell the rounding: fused the other way, some are culled otherwise
            other = outside | (~outside & _occluded(nodes, vp, first, w, h, fused=False))
            this = outside | (~outside & _occluded(nodes, vp, first, w, h))
            assert (other != this)[finite].sum() >= 10
            assert 0.1 < outside.mean() < 0.9 and 0.1 < this[~outside].mean() < 0.9


@pytest.mark.parametrize("n,immediate", [(20_001, 0), (20_001, 1)])
def test_cull_of_a_frame(n, immediate):
    """The same inside the preprocess (and, for comparison, as a launch), on a frame's own Hi-Z: large opaque
    Gaussians, so that pass 1 splats all that is in view and pass 2's Hi-Z is the one left behind."""
    import torch

    g = synth.activate(synth.cube(n, seed=12))
    g[:, 52:55] = 0.3
    g[:, 51] = 0.99
    scene = gpsplat.Scene.from_host(g[gpsplat.morton_order(g)])
    s = gpsplat.default_settings(width=320, height=180, samples_per_pixel=2, immediate_splat_threshold=immediate)
    cam = gpsutil.cameras_for(s, [(np.array([3.0, 2.0, -14.0]), synth.look_at_c2w([3.0, 2.0, -14.0], [4.0, 0.0, 0.0]))])[0]
    image, depth = torch.zeros((180, 320, 3), device="cuda"), torch.zeros((180, 320), device="cuda")
    r = gpsplat.Renderer(scene, s)
    r.render(cam, image.data_ptr(), depth.data_ptr(), 0)
    torch.cuda.synchronize()
    st, v = r.stats(), r.debug_view()
    assert st.num_points_one > 100_000 and st.num_points_two == 0
    nodes = gpsutil.d2h(v.block_nodes, v.block_count * 8, F).reshape(-1, 8)
    bits = np.unpackbits(gpsutil.d2h(v.block_culled, v.block_words, np.uint32).view(np.uint8), bitorder="little")
    vp = r.derived(cam)[:16].astype(F)
    outside = _outside(nodes, np.array(list(cam.frustum_planes), F))
    levels = _chain(depth.cpu().numpy(), 0)
    r.close()
    scene.close()
    want = outside | (~outside & _occluded(nodes, vp, levels, 320, 180))
    assert 0.05 < want.mean() < 0.99 and outside.any() and (want & ~outside).any()
    assert np.array_equal(bits[: v.block_count].astype(bool), want)
