"""The screen-binned splat, whose first pass tests its samples in shared memory, against the walk in
Gaussian order: the minimum of the same samples, so the buffers are equal bit for bit."""
import os

import numpy as np
import pytest

import gpsplat
import gpsutil
import synth

pytestmark = pytest.mark.gpu

def _min_points(spp):
    """Of a pass that surely takes the shared-memory test: two groups per block, 4 or 1 blocks on 148 SMs."""
    return 2 * (592 if spp <= 6 else 148) * 1024


def _frames(scene, s, cams, crowded):
    import torch

    if crowded is not None:
        os.environ["GPS_BIN_CROWDED"] = crowded
    try:
        r = gpsplat.Renderer(scene, s)
    finally:
        os.environ.pop("GPS_BIN_CROWDED", None)
    image = torch.zeros((s.height, s.width, 3), device="cuda")
    depth = torch.zeros((s.height, s.width), device="cuda")
    out = []
    for cam in cams:
        r.render(cam, image.data_ptr(), depth.data_ptr(), 0)
        torch.cuda.synchronize()
        ptr, entries = r.splat_buffer()
        st = r.stats()
        out.append((gpsutil.d2h(ptr, entries, np.uint64), st.num_points_one, st.screen_order_one, st.truncated))
    r.close()
    return out


@pytest.mark.parametrize("width,height,spp,k,max_points,fmt", [
    (1920, 1080, 4, 4, 250_000_000, gpsplat.GPS_SCENE_FP32),        # three blocks per SM
    (2500, 1300, 1, 1, 250_000_000, gpsplat.GPS_SCENE_FP32),        # one plane, K = 1, edge tiles on both axes
    (1237, 689, 3, 1, 250_000_000, gpsplat.GPS_SCENE_COMPRESSED),   # planes no power of two
    (1300, 1000, 2, 2, 250_000_000, gpsplat.GPS_SCENE_FP32),
    (1100, 900, 6, 1, 250_000_000, gpsplat.GPS_SCENE_HALF),         # the most planes, two blocks per SM
    (1100, 900, 7, 1, 250_000_000, gpsplat.GPS_SCENE_FP32),         # one more: a block of 1024 threads per SM
    (1100, 900, 13, 4, 250_000_000, gpsplat.GPS_SCENE_FP32),        # its most planes
    (1100, 900, 14, 1, 250_000_000, gpsplat.GPS_SCENE_FP32),        # one more: the test in L1
    (1920, 1080, 4, 1, 1_300_000, gpsplat.GPS_SCENE_FP32),          # truncated: Gaussian order
])
def test_binned_equals_gaussian_order(width, height, spp, k, max_points, fmt):
    scene = gpsplat.Scene.from_host(synth.activate(synth.town(400_000, seed=21)), fmt)
    s = gpsplat.default_settings(width=width, height=height, samples_per_pixel=spp, points_per_thread=k,
                                 max_number_of_points=max_points)
    cams = gpsutil.cameras_for(s, synth.orbit(60, 30.0, 10.0)[:2])
    binned = _frames(scene, s, cams, None)
    plain = _frames(scene, s, cams, "0")
    scene.close()
    for (a, points, order, truncated), (b, _, other, _) in zip(binned, plain):
        assert other == 0 and order == (0 if truncated else 1)
        assert truncated == (1 if max_points < 2_000_000 else 0)
        assert truncated or points >= _min_points(spp), points
        assert np.array_equal(a, b)
