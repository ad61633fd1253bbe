"""The nearest depth of a pixel, bit for bit, for planes on both sides of the resolve's rule: where a
key's NDC depth falls nowhere as the key grows it is the smallest key's, else the smallest of all samples'."""
import ctypes
import os

import numpy as np
import pytest

import gpsplat
import gpsutil
import synth
from test_gpu_resolve import _pixels

pytestmark = pytest.mark.gpu


def _check_library():
    gpsplat.load_library()
    lib = ctypes.CDLL(os.path.join(gpsutil.PKG, "libgps_check.so"))
    lib.gps_check_depth_falls.argtypes = [ctypes.c_float, ctypes.c_float]
    lib.gps_check_depths.argtypes = [ctypes.c_void_p, ctypes.c_uint32, ctypes.c_float, ctypes.c_float, ctypes.c_void_p]
    return lib


def _planes(count, seed):
    rng = np.random.default_rng(seed)
    near = np.exp(rng.uniform(np.log(1e-6), np.log(1e3), count))
    return [(float(n), float(n * (1.0 + f))) for n, f in zip(near, np.exp(rng.uniform(np.log(1e-4), np.log(1e9), count)))]


def test_sweep_over_all_keys():
    """Every plane pair in use is monotone, the view depth through zero is not."""
    lib = _check_library()
    for near, far in [(0.2, 10000.0), (0.01, 100.0), (0.1, 1000.0), (1e-6, 1e9), (1e-7, 100.0), (0.01, 2e9)] + _planes(24, 3):
        assert lib.gps_check_depth_falls(near, far) == 0, (near, far)
    for near, far in [(0.0, 100.0), (-5.0, 100.0)]:
        assert lib.gps_check_depth_falls(near, far) == 1, (near, far)


@pytest.mark.parametrize("near,far", [(0.2, 10000.0), (1e-7, 100.0), (0.01, 2e9), (3.0, 60.0), (-5.0, 100.0)])
@pytest.mark.parametrize("ss,spp", [(1, 1), (1, 3), (2, 1), (2, 4), (4, 2), (4, 5), (4, 8), (8, 1), (3, 2), (5, 1), (2, 9)])
def test_nearest_depth(near, far, ss, spp):
    import torch

    w, h = 131, 70
    scene = gpsplat.Scene.from_host(synth.activate(synth.cube(4000, seed=9)))
    s = gpsplat.default_settings(width=w, height=h, supersampling_factor=ss, samples_per_pixel=spp, near_view_plane=near,
                                 far_view_plane=far, max_number_of_points=4_000_000)
    cam = gpsutil.cameras_for(s, [(np.array([0.0, 0.0, -24.0]), synth.look_at_c2w([0.0, 0.0, -24.0], [0.0, 0.0, 0.0]))])[0]
    image, depth = torch.zeros((h, w, 3), device="cuda"), torch.zeros((h, w), device="cuda")
    r = gpsplat.Renderer(scene, s)
    r.render(cam, image.data_ptr(), depth.data_ptr(), 0)
    torch.cuda.synchronize()
    ptr, entries = r.splat_buffer()
    px = _pixels(gpsutil.d2h(ptr, entries, np.uint64), w, h, ss, spp)
    r.close()
    scene.close()
    keys = np.ascontiguousarray((px >> np.uint64(36)).astype(np.uint32))
    assert near < 0 or far > 1e6 or len(np.unique(keys)) > 100
    each = np.empty(keys.shape, np.float32)
    assert _check_library().gps_check_depths(keys.ctypes.data, keys.size, near, far, each.ctypes.data) == 0
    want = each.min(axis=2)
    assert np.array_equal(depth.cpu().numpy().view(np.uint32), want.view(np.uint32))
