"""Resolve and Hi-Z chain at the edges of their tiles, against numpy on the frame's own splat buffer.

The chain is minima and maxima of the depth image, so it has to be equal bit for bit.  Depth and
colour are compared with 64-bit values: an NDC depth a + b / z has |a|, |b / z| <= 1 + 2^-11 and 2
here, a handful of roundings and one approximate division of at most 2 ulp (4e-7 each at most:
2e-6 in all); a channel is a sum of n terms of at most 4095/255, each addition rounding once, so
its mean is off by at most (n + 2) 2^-24 times 4095/255."""
import numpy as np
import pytest

import gpsplat
import gpsutil
import synth

pytestmark = pytest.mark.gpu


def _spread(a):
    a = a.astype(np.int64)
    out = np.zeros_like(a)
    for b in range(6):
        out |= ((a >> b) & 1) << (2 * b)
    return out


def _pixels(buf, w, h, ss, spp):
    """The buffer as (h, w, ss * ss * spp) words."""
    x, y = np.meshgrid(np.arange(w * ss), np.arange(h * ss))
    tiles_x = (w * ss + 63) // 64
    at = (((y >> 6) * tiles_x + (x >> 6)) * 4096 + (_spread(x & 63) | (_spread(y & 63) << 1))) * spp
    v = buf[at[..., None] + np.arange(spp)]
    return v.reshape(h, ss, w, ss, spp).transpose(0, 2, 1, 3, 4).reshape(h, w, -1)


def _chain(depth, min_levels):
    """Finest level first."""
    levels, j = [depth], 1
    while max(levels[-1].shape) > 1:
        d = levels[-1]
        op, pad = (np.minimum, np.inf) if j <= min_levels else (np.maximum, -np.inf)
        d = np.pad(d, ((0, d.shape[0] & 1), (0, d.shape[1] & 1)), constant_values=pad)
        levels.append(op(op(d[::2, ::2], d[::2, 1::2]), op(d[1::2, ::2], d[1::2, 1::2])))
        j += 1
    return levels


@pytest.mark.parametrize("width,height,ss,spp,min_levels", [
    (1, 1, 2, 1, 0), (4, 3, 2, 2, 0), (5, 8, 1, 2, 1),           # chains around the four fine levels
    (8, 8, 2, 4, 0), (9, 7, 2, 4, 2), (65, 33, 2, 4, 5),         # one group of 64 pixels and its edges
    (129, 127, 1, 4, 0), (131, 70, 1, 1, 3), (257, 19, 2, 3, 0),  # 16 x 16-texel blocks; unstaged runs
    (67, 35, 4, 4, 0), (67, 35, 4, 8, 1), (40, 23, 8, 1, 0),     # 64- and 32-pixel blocks, one group a tile
    (97, 61, 3, 2, 0), (37, 50, 3, 1, 2), (33, 31, 5, 1, 0),     # factors that are no power of two
    (70, 41, 2, 5, 0), (90, 33, 4, 3, 0), (41, 90, 1, 7, 0), (21, 17, 2, 9, 0),  # runs that are none
    (1030, 517, 2, 2, 0),                                        # levels past shared memory
])
def test_resolve_and_hiz_against_numpy(width, height, ss, spp, min_levels):
    raw = synth.cube(4000, seed=9)
    scene = gpsplat.Scene.from_host(synth.activate(raw))
    s = gpsplat.default_settings(width=width, height=height, supersampling_factor=ss, samples_per_pixel=spp,
                                 occlusion_culling_min_reduce_count=min_levels, background=(0.25, 0.5, 1.5),
                                 max_number_of_points=4_000_000)
    cam = gpsutil.cameras_for(s, [(np.array([0.0, 0.0, -24.0]), synth.look_at_c2w([0.0, 0.0, -24.0], [0.0, 0.0, 0.0]))])[0]
    import torch

    image = torch.zeros((height, width, 3), device="cuda")
    depth = torch.zeros((height, width), device="cuda")
    r = gpsplat.Renderer(scene, s)
    for _ in range(2):
        r.render(cam, image.data_ptr(), depth.data_ptr(), 0)
    torch.cuda.synchronize()
    ptr, entries = r.splat_buffer()
    px = _pixels(gpsutil.d2h(ptr, entries, np.uint64), width, height, ss, spp)
    v = r.debug_view()
    hiz = gpsutil.d2h(v.hiz, v.hiz_size, np.float32)
    r.close()
    scene.close()
    got = depth.cpu().numpy()
    near, far = float(s.near_view_plane), float(s.far_view_plane)
    z = (px.min(axis=2) >> np.uint64(36)).astype(np.float64) / (2**28 - 1) * (far - near) + near
    want = (far + near) / (far - near) - 2.0 * far * near / (far - near) / z
    assert np.abs(got - want).max() <= 2e-6
    n = ss * ss * spp
    for c, shift in enumerate((24, 12, 0)):
        mean = ((px >> np.uint64(shift)) & np.uint64(0xFFF)).astype(np.float64).mean(axis=2) / 255.0
        assert np.abs(image.cpu().numpy()[..., c] - mean).max() <= (n + 2) * 2.0**-24 * 4095 / 255
    levels = _chain(got, min_levels)[::-1]  # coarsest first, as stored
    flat = np.concatenate([d.ravel() for d in levels])
    assert flat.size == hiz.size
    assert np.array_equal(flat.view(np.uint32), hiz.view(np.uint32))
