"""The scan's survivors that own many tiles (their warp writes four at a time from 129 on)."""
import ctypes

import numpy as np
import pytest

import gpsplat
from test_gpu_scan_edges import _scan_numpy

pytestmark = pytest.mark.gpu

BIG = 32 << 20  # Gaussians from which the tiles are 16384


def _run(counts, bits, n, max_points):
    import torch

    gid, start, total, points, owner = _scan_numpy(counts, bits, max_points)
    mask = np.packbits(bits, bitorder="little").view(np.uint32)
    d = {"counts": counts, "mask": mask, "gid": np.zeros(n, np.uint32), "start": np.zeros(n, np.uint32),
         "tile": np.zeros(max_points // 256 + 2, np.uint32), "ctr": np.full(8, 7, np.uint32)}
    d = {k: torch.from_numpy(v.view(np.int32)).cuda() for k, v in d.items()}
    st = gpsplat.load_library().gps_workload_scan_noalloc(
        *(ctypes.c_void_p(d[k].data_ptr()) for k in ("counts", "mask")), n, max_points,
        *(ctypes.c_void_p(d[k].data_ptr()) for k in ("gid", "start", "tile", "ctr")), None)
    assert st == 0, gpsplat.load_library().gps_last_error().decode()
    torch.cuda.synchronize()
    got = {k: v.cpu().numpy().view(np.uint32) for k, v in d.items()}
    assert list(got["ctr"]) == [gid.size, total, points, int(total > max_points), 0, 0, 0, 0]
    assert np.array_equal(got["gid"][: gid.size], gid) and np.array_equal(got["start"][: gid.size], start)
    assert np.array_equal(got["tile"][: owner.size], owner)


@pytest.mark.parametrize("points,owners,max_points", [
    (128 * 256 - 1, 9, 1 << 24), (128 * 256, 9, 1 << 24), (129 * 256, 9, 1 << 24), (132 * 256 + 1, 9, 1 << 24),
    (600_000, 20, 1 << 24), (600_000, 20, 4_000_000),  # cut off inside one
    (100_000_000, 1, 250_000_000),
])
@pytest.mark.parametrize("n", [70_001, BIG + 7])
def test_owners_of_many_tiles(n, points, owners, max_points):
    rng = np.random.default_rng(points)
    pad = (n + 31) // 32 * 32
    bits = np.zeros(pad, bool)
    bits[: min(n, 200_000)] = rng.random(min(n, 200_000)) < 0.1
    counts = rng.integers(0, 9, pad).astype(np.uint32)
    at = 9000 + 7 * np.arange(owners)
    bits[at] = True
    counts[at] = points
    _run(counts, bits, n, max_points)
