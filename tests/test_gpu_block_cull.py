"""The block cull's bits against the frustum test in 64 bits, inside the preprocess (up to 303,104
Gaussians), as a launch with its list of chunks, and at the edges of its words and chunks.  A node whose
nearest plane distance is within 1e-5 of the terms' magnitude may round either way; all others agree."""
import numpy as np
import pytest

import gpsplat
import gpsutil
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,immediate", [(1, 0), (31, 0), (33, 0), (127, 0), (129, 0), (4097, 0), (303_104, 0), (303_105, 0),
                                         (1, 1), (129, 1), (8191, 1), (8193, 1), (303_104, 1)])
def test_block_cull_bits(n, immediate):
    import torch

    scene = gpsplat.Scene.from_host(synth.activate(synth.town(n, seed=n)))
    s = gpsplat.default_settings(width=320, height=180, enable_occlusion_culling=0, immediate_splat_threshold=immediate)
    image, depth = torch.zeros((180, 320, 3), device="cuda"), torch.zeros((180, 320), device="cuda")
    r = gpsplat.Renderer(scene, s)
    for cam in gpsutil.cameras_for(s, synth.orbit(7, 30.0, 10.0)[:3]):
        r.render(cam, image.data_ptr(), depth.data_ptr(), 0)
        torch.cuda.synchronize()
        v = r.debug_view()
        nodes = gpsutil.d2h(v.block_nodes, v.block_count * 8, np.float32).reshape(-1, 8).astype(np.float64)
        bits = np.unpackbits(gpsutil.d2h(v.block_culled, v.block_words, np.uint32).view(np.uint8), bitorder="little")
        assert not bits[v.block_count:].any()
        culled = bits[: v.block_count].astype(bool)
        planes = np.array(list(cam.frustum_planes), np.float64).reshape(6, 4)
        lo, hi = nodes[:, None, 0:3], nodes[:, None, 4:7]
        terms = planes[None, :, :3] * np.where(planes[None, :, :3] >= 0, hi, lo)
        dist = terms.sum(2) + planes[:, 3]
        margin = 1e-5 * (np.abs(terms).sum(2) + np.abs(planes[:, 3]))
        assert culled[(dist < -margin).any(1)].all()
        assert not culled[(dist > margin).all(1)].any()
        gid = gpsutil.d2h(v.surv_gid, v.survivors, np.uint32)
        assert not culled[gid // v.per_block].any()
        mask = np.unpackbits(gpsutil.d2h(v.mask_last, (n + 31) // 32, np.uint32).view(np.uint8), bitorder="little")[:n]
        assert np.array_equal(np.flatnonzero(mask), gid)
    r.close()
    scene.close()
