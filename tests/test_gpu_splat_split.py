"""The two kernels of a screen-binned first pass: which takes it is decided by its points (two groups
of 1024 per block of 256 threads, one per block of 1024 threads) and by its order, on the device."""
import os

import numpy as np
import pytest

import gpsplat
import gpsutil
import synth

pytestmark = pytest.mark.gpu

SMS = 148
# blocks per SM that the planes of 16 KB per sample leave room for, and groups of 1024 points per block
SPLIT = {4: SMS * 3 * 2 * 1024, 2: SMS * 4 * 2 * 1024, 8: SMS * 1024}


def _renderer(scene, s, crowded):
    if crowded:
        os.environ["GPS_BIN_CROWDED"] = "0"
    try:
        return gpsplat.Renderer(scene, s)
    finally:
        os.environ.pop("GPS_BIN_CROWDED", None)


def _frames(r, s, cams):
    import torch

    image, depth = torch.zeros((s.height, s.width, 3), device="cuda"), torch.zeros((s.height, s.width), device="cuda")
    out = []
    for cam in cams:
        r.render(cam, image.data_ptr(), depth.data_ptr(), 0)
        torch.cuda.synchronize()
        ptr, entries = r.splat_buffer()
        st = r.stats()
        out.append((gpsutil.d2h(ptr, entries, np.uint64), st.num_points_one, st.screen_order_one))
    return out


# points of the first pass against the split: (lowest, highest) as a share of it
@pytest.mark.parametrize("n,spp,lowest,highest", [
    (2_000, 4, 0.0, 0.1), (60_000, 4, 0.05, 0.49),   # less than one group per block
    (180_000, 4, 0.5, 1.0), (220_000, 4, 0.5, 1.5),  # between one and two, and around two
    (500_000, 4, 1.0, 9.0), (500_000, 2, 1.0, 9.0),  # more
    (20_000, 8, 0.1, 1.0), (90_000, 8, 1.0, 3.0),
])
def test_both_sides_of_the_split(n, spp, lowest, highest):
    scene = gpsplat.Scene.from_host(synth.activate(synth.town(n, seed=5)))
    s = gpsplat.default_settings(width=1920, height=1080, samples_per_pixel=spp)
    cams = gpsutil.cameras_for(s, synth.orbit(60, 30.0, 10.0)[:3])
    got = []
    for crowded in (False, True):
        r = _renderer(scene, s, crowded)
        got.append(_frames(r, s, cams))
        r.close()
    scene.close()
    for (a, points, order), (b, _, other) in zip(*got):
        assert order == 1 and other == 0
        assert lowest * SPLIT[spp] <= points < highest * SPLIT[spp], points
        assert np.array_equal(a, b)


def test_a_crowded_pass_has_the_whole_l1():
    """A pass that is walked in Gaussian order takes 1.2 times as long as in screen-bin order (1M town,
    1080p, 4 spp), and 2.2 times beside the shared memory that the other kernel reserves."""
    import torch

    scene = gpsplat.Scene.from_host(synth.activate(synth.town(1_000_000, seed=5)))
    s = gpsplat.default_settings(width=1920, height=1080, samples_per_pixel=4, enable_occlusion_culling=0)
    cams = gpsutil.cameras_for(s, synth.orbit(120, 30.0, 10.0)[:12])
    image, depth = torch.zeros((1080, 1920, 3), device="cuda"), torch.zeros((1080, 1920), device="cuda")
    took = []
    for crowded in (False, True):
        r = _renderer(scene, s, crowded)
        for _ in range(3):  # the last of three rounds is timed
            r.enable_timing(True)
            r.stage_times(reset=True)
            for cam in cams:
                r.render(cam, image.data_ptr(), depth.data_ptr(), 0)
            torch.cuda.synchronize()
            ms = r.stage_times(reset=True)["splat"][0]
        took.append(ms)
        r.close()
    scene.close()
    assert took[1] < 1.7 * took[0], took
