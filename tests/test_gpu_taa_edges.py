"""gps_post_taa at the edges of its tiles against a 64-bit restatement: images smaller than a tile, one
pixel over, widths whose rows of bytes are on words and not, unaligned byte images.

The blended colour may differ by the reprojected position's rounding: a position p has an error of
a few 2^-24 p and meets neighbouring history pixels that differ by up to 0.2 here, weighted 0.9, so
1e-6 max(w, h) covers it; a position that rounds across a pixel's edge has weights of that size too."""
import ctypes

import numpy as np
import pytest

import gpsplat

pytestmark = pytest.mark.gpu


def _taa64(cur, prev, depth, m, blend):
    h, w, _ = cur.shape
    y, x = np.meshgrid(np.arange(h, dtype=np.float64), np.arange(w, dtype=np.float64), indexing="ij")
    clip = np.stack([(x + 0.5) / w * 2 - 1, (y + 0.5) / h * 2 - 1, depth, np.ones_like(x)], -1)
    p = clip @ m.T
    px, py = (p[..., 0] / p[..., 3] * 0.5 + 0.5) * w - 0.5, (p[..., 1] / p[..., 3] * 0.5 + 0.5) * h - 0.5
    inside = (px >= 0) & (px < w) & (py >= 0) & (py < h)
    fx, fy = np.floor(px), np.floor(py)
    x0, x1 = (np.clip(fx + d, 0, w - 1).astype(int) for d in (0, 1))
    y0, y1 = (np.clip(fy + d, 0, h - 1).astype(int) for d in (0, 1))
    tx, ty = (px - fx)[..., None], (py - fy)[..., None]
    hist = ((prev[y0, x0] * (1 - tx) + prev[y0, x1] * tx) * (1 - ty) + (prev[y1, x0] * (1 - tx) + prev[y1, x1] * tx) * ty)
    pad = np.pad(cur, ((1, 1), (1, 1), (0, 0)), mode="edge")
    win = np.stack([pad[dy:dy + h, dx:dx + w] for dy in range(3) for dx in range(3)])
    hist = np.clip(hist, win.min(0) - 0.05, win.max(0) + 0.05)
    return np.where(inside[..., None], cur * (1 - blend) + hist * blend, cur), inside


@pytest.mark.parametrize("width,height,offset", [(1, 1, 0), (5, 3, 0), (31, 16, 1), (32, 16, 0), (33, 17, 0), (64, 33, 2),
                                                 (66, 15, 0), (100, 50, 3), (128, 48, 0), (97, 100, 1)])
@pytest.mark.parametrize("frame", [0, 3])
def test_taa_edges(width, height, offset, frame):
    import torch

    rng = np.random.default_rng(width * 1000 + height)
    prev = rng.random((height, width, 3), np.float32) * 0.2 + 0.4
    cur = (prev + (rng.random((height, width, 3), np.float32) - 0.5) * 0.3).astype(np.float32)
    depth = (0.9 + 0.1 * rng.random((height, width), np.float32)).astype(np.float32)
    m = np.eye(4)
    m[0, 3], m[1, 3], m[0, 1], m[3, 2] = 0.03, -0.02, 0.01, 0.002  # a small turn, some of it off the image
    d = {k: torch.from_numpy(v).cuda() for k, v in (("cur", cur), ("prev", prev), ("depth", depth))}
    out = torch.full((height, width, 3), -1.0, device="cuda")
    raw = torch.full((height * width * 3 + 8,), 7, dtype=torch.uint8, device="cuda")
    st = gpsplat.load_library().gps_post_taa(
        ctypes.c_void_p(raw.data_ptr() + offset), out.data_ptr(), d["cur"].data_ptr(), d["prev"].data_ptr(),
        d["depth"].data_ptr(), d["depth"].data_ptr(), (ctypes.c_float * 16)(*m.T.astype(np.float32).ravel().tolist()),
        0.9, width, height, frame, None)
    assert st == 0
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    bytes_ = raw.cpu().numpy()
    if frame == 0:
        assert np.array_equal(got, cur)
    else:
        want, _ = _taa64(cur.astype(np.float64), prev.astype(np.float64), depth.astype(np.float64),
                         m.astype(np.float32).astype(np.float64), float(np.float32(0.9)))
        # (a position at the image's very edge may be inside for one and outside for the other)
        assert (np.abs(got - want).max(axis=2) > 1e-6 * max(width, height)).sum() <= 0.001 * width * height
    image = bytes_[offset:offset + height * width * 3].reshape(height, width, 3)
    v = np.clip(got.astype(np.float64), 0, 1).astype(np.float32) * np.float32(255.0)
    assert np.array_equal(image, np.floor(v.astype(np.float64) + 0.5).astype(np.uint8))
    assert (bytes_[:offset] == 7).all() and (bytes_[offset + height * width * 3:] == 7).all()
