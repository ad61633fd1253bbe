"""What a renderer's kernels leave for the next pass, when something went wrong between them."""
import ctypes
import os

import numpy as np
import pytest

import gpsplat
import gpsutil
import synth

pytestmark = pytest.mark.gpu


def _check_library():
    gpsplat.load_library()
    return ctypes.CDLL(os.path.join(gpsutil.PKG, "libgps_check.so"))


@pytest.mark.parametrize("n,stale", [(1, 0), (1, 1), (8193, 0), (8193, 100), (303_105, 0), (303_105, 9000), (303_105, 1 << 30)])
def test_chunk_list_ends_at_its_capacity(n, stale):
    """A list whose count did not start at zero takes no entry past the scene's chunks."""
    chunks = (n + 31) // 32
    got, count = np.zeros(2 * chunks, np.uint32), ctypes.c_uint32(0)
    rc = _check_library().gps_check_cull_list(ctypes.c_uint32(n), ctypes.c_uint32(stale), got.ctypes.data_as(ctypes.c_void_p),
                                              ctypes.byref(count))
    assert rc == 0
    assert count.value == stale + chunks  # every chunk is visible
    assert (got[chunks:] == 0xFFFFFFFF).all()
    assert (got[: min(stale, chunks)] == 0xFFFFFFFF).all()
    listed = got[min(stale, chunks) : chunks]
    assert len(np.unique(listed)) == len(listed) and (listed < chunks).all()


@pytest.mark.parametrize("n", [60_000, 400_000])
def test_frames_after_a_failed_one(n):
    """A frame whose launches fail is reported, and the frames after it are a new renderer's."""
    import torch

    scene = gpsplat.Scene.from_host(synth.activate(synth.town(n, seed=4)))
    s = gpsplat.default_settings(width=320, height=180, samples_per_pixel=2)
    cams = gpsutil.cameras_for(s, synth.orbit(30, 30.0, 10.0)[:3])
    image, depth = torch.zeros((180, 320, 3), device="cuda"), torch.zeros((180, 320), device="cuda")
    cudart = gpsutil.cudart()
    stream = torch.cuda.Stream()
    handle = ctypes.c_void_p(stream.cuda_stream)

    def frames(r):
        out = []
        for cam in cams:
            r.render(cam, image.data_ptr(), depth.data_ptr(), stream.cuda_stream)
            stream.synchronize()
            ptr, entries = r.splat_buffer()
            out.append((gpsutil.d2h(ptr, entries, np.uint64), image.cpu().numpy(), depth.cpu().numpy()))
        return out

    r = gpsplat.Renderer(scene, s)
    want = frames(r)
    r.close()
    r = gpsplat.Renderer(scene, s)
    assert cudart.cudaStreamBeginCapture(handle, 1) == 0  # thread-local
    cudart.cudaStreamSynchronize(handle)  # not allowed while capturing: the capture is invalid from here on
    with pytest.raises(gpsplat.GpsError):
        r.render(cams[0], image.data_ptr(), depth.data_ptr(), stream.cuda_stream)
    graph = ctypes.c_void_p(0)
    cudart.cudaStreamEndCapture(handle, ctypes.byref(graph))
    cudart.cudaGetLastError()
    for got, expected in zip(frames(r), want):
        for a, b in zip(got, expected):
            assert np.array_equal(a, b)
    r.close()
    scene.close()


@pytest.mark.parametrize("earlier", [0, 1])
def test_refused_shared_memory_keeps_an_earlier_error(earlier):
    refused, pending = ctypes.c_int(0), ctypes.c_int(0)
    _check_library().gps_check_smem_refusal(earlier, ctypes.byref(refused), ctypes.byref(pending))
    assert refused.value == 1
    assert pending.value == earlier
