"""The splat against a plain one of the same records: one thread per point, one sample after the other in
the reference's form, no pre-test.  A minimum (or, biased, the sum of the colours at the smallest depth)
does not depend on the order, so the buffers are equal.  Small passes, whose points' samples are split
among two or four threads, and large ones in screen-bin order."""
import ctypes
import os

import numpy as np
import pytest

import gpsplat
import gpsutil
import synth

pytestmark = pytest.mark.gpu

THREADS = 148 * 4 * 256  # of the splat's grid at its fewest: a pass of at most half as many points is split


def _frame_and_plain(g, s, cam):
    """The frame's statistics, its buffer, the plain splat's and the background."""
    import torch

    lib = ctypes.CDLL(os.path.join(gpsutil.PKG, "libgps_check.so"))
    image, depth = torch.zeros((s.height, s.width, 3), device="cuda"), torch.zeros((s.height, s.width), device="cuda")
    scene = gpsplat.Scene.from_host(g)
    r = gpsplat.Renderer(scene, s)
    r.render(cam, image.data_ptr(), depth.data_ptr(), 0)
    torch.cuda.synchronize()
    st, v = r.stats(), r.debug_view()
    ptr, entries = r.splat_buffer()
    got, want = gpsutil.d2h(ptr, entries, np.uint64), np.empty(entries, np.uint64)
    ss = s.supersampling_factor
    k = 1 if not s.reduce_point_count else s.points_per_thread or ss**2
    initial = int(got.max())  # (the farthest depth)
    rc = lib.gps_check_splat(ctypes.c_void_p(v.records), ctypes.c_void_p(v.surv_gid), ctypes.c_void_p(v.surv_start),
                             ctypes.c_uint32(v.survivors), ctypes.c_uint32(st.num_points_one), 4 * cam.frame + 1, s.width * ss,
                             s.height * ss, s.samples_per_pixel, k, int(s.use_unbiased_2d_splatting), ctypes.c_uint64(initial),
                             ctypes.c_uint64(entries), want.ctypes.data_as(ctypes.c_void_p))
    assert rc == 0
    r.close()
    scene.close()
    return st, got, want, initial


@pytest.mark.parametrize("n,ss,spp,reduce,unbiased", [
    (6000, 2, 4, True, True), (6000, 2, 2, True, True), (25_000, 2, 1, True, True),    # 16, 8 and 4 samples in fours
    (9000, 1, 5, True, True), (9000, 1, 7, True, True), (9000, 2, 5, False, True),     # odd counts, one draw per pass
    (6000, 3, 1, True, True), (4000, 3, 3, True, True),                                # 9 and 27: any K
    (6000, 2, 4, True, False), (6000, 2, 1, True, False), (9000, 1, 5, False, False),  # biased
])
def test_split_samples(n, ss, spp, reduce, unbiased):
    s = gpsplat.default_settings(width=160, height=90, supersampling_factor=ss, samples_per_pixel=spp, reduce_point_count=int(reduce),
                                 use_unbiased_2d_splatting=int(unbiased), enable_occlusion_culling=0,
                                 fully_disable_hierarchical_culling=1, background=(0.1, 0.2, 0.3))
    pose = np.array([0.0, 0.0, -26.0])
    cam = gpsutil.cameras_for(s, [(pose, synth.look_at_c2w(pose, [0.0, 0.0, 0.0]))])[0]
    st, got, want, initial = _frame_and_plain(synth.activate(synth.cube(n, seed=n + ss)), s, cam)
    assert 2000 < st.num_points_one <= THREADS // 2
    assert (want != initial).mean() > 0.05
    assert np.array_equal(got, want)


@pytest.mark.parametrize("width,height,ss,spp,k,unbiased", [
    (1920, 1080, 2, 4, 4, True), (2500, 1300, 2, 1, 1, True), (1300, 1000, 2, 2, 2, True),  # the test in shared memory
    (1100, 900, 2, 8, 4, True), (1100, 900, 2, 14, 4, True), (1920, 1080, 2, 4, 8, True),  # 1024 threads; in L1
    (1237, 689, 3, 2, 9, True), (1920, 1080, 2, 1, 4, False), (1237, 689, 3, 3, 1, False),
])
def test_large_passes(width, height, ss, spp, k, unbiased):
    s = gpsplat.default_settings(width=width, height=height, supersampling_factor=ss, samples_per_pixel=spp, points_per_thread=k,
                                 use_unbiased_2d_splatting=int(unbiased), enable_occlusion_culling=0)
    cam = gpsutil.cameras_for(s, synth.orbit(60, 30.0, 10.0)[:1])[0]
    st, got, want, _ = _frame_and_plain(synth.activate(synth.town(500_000, seed=2)), s, cam)
    assert st.num_points_one > 400_000
    assert np.array_equal(got, want)


def test_biased_against_unbiased_time():
    """The biased splat of a large pass takes twice the unbiased one's time (700k town, 1280x720, 4 spp: 232 and
    117 us), and 2.9 times with its samples in batches of four."""
    import torch

    scene = gpsplat.Scene.from_host(synth.activate(synth.town(700_000, seed=5)))
    image, depth = torch.zeros((720, 1280, 3), device="cuda"), torch.zeros((720, 1280), device="cuda")
    took = []
    for unbiased in (0, 1):
        s = gpsplat.default_settings(width=1280, height=720, samples_per_pixel=4, use_unbiased_2d_splatting=unbiased, enable_occlusion_culling=0)
        cams = gpsutil.cameras_for(s, synth.orbit(120, 30.0, 10.0)[:12])
        r = gpsplat.Renderer(scene, s)
        for _ in range(3):  # the last of three rounds counts
            r.enable_timing(True)
            r.stage_times(reset=True)
            for cam in cams:
                r.render(cam, image.data_ptr(), depth.data_ptr(), 0)
            torch.cuda.synchronize()
            ms = r.stage_times(reset=True)["splat"][0]
        took.append(ms)
        r.close()
    scene.close()
    assert took[0] < 2.4 * took[1], took


@pytest.mark.parametrize("fmt", [gpsplat.GPS_SCENE_FP32, gpsplat.GPS_SCENE_COMPRESSED, gpsplat.GPS_SCENE_HALF])
def test_immediate_against_listed_time(fmt):
    """Splatting Gaussians of up to 20 points in the preprocess takes 5.5 times the two kernels' time without
    (a Gaussian's points one after the other), and 9.3 times with three blocks per SM."""
    import torch

    scene = gpsplat.Scene.from_host(synth.activate(synth.town(150_000, seed=5)), fmt)
    image, depth = torch.zeros((191, 411, 3), device="cuda"), torch.zeros((191, 411), device="cuda")
    took = []
    for threshold in (20, 0):
        s = gpsplat.default_settings(width=411, height=191, samples_per_pixel=8, immediate_splat_threshold=threshold,
                                     enable_occlusion_culling=0, fully_disable_hierarchical_culling=1)
        cams = gpsutil.cameras_for(s, synth.orbit(120, 30.0, 10.0)[:12])
        r = gpsplat.Renderer(scene, s)
        for _ in range(3):  # the last of three rounds counts
            r.enable_timing(True)
            r.stage_times(reset=True)
            for cam in cams:
                r.render(cam, image.data_ptr(), depth.data_ptr(), 0)
            torch.cuda.synchronize()
            t = r.stage_times(reset=True)
        took.append(t["preprocess"][0] + t["splat"][0])
        r.close()
    scene.close()
    assert took[0] < 7.2 * took[1], took
