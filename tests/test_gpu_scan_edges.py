"""The allocation-free scan against numpy at the edges of its dispatch: around a 4096-Gaussian tile,
where the tile totals get a launch of their own (more than 4096 tiles), where tiles grow to 16384
Gaussians; counts of zero, and one Gaussian that owns most of the 256-point tiles.  Integers: exact."""
import ctypes

import numpy as np
import pytest

import gpsplat

pytestmark = pytest.mark.gpu


def _scan_numpy(counts, bits, max_points):
    gid = np.flatnonzero(bits)
    cnt = counts[gid].astype(np.uint64)
    start = np.cumsum(cnt) - cnt
    total = int(cnt.sum())
    points = min(total, max_points)
    first = np.arange(0, points, 256, dtype=np.uint64)
    owner = np.searchsorted(start, first, side="right") - 1 if gid.size else np.zeros(0)
    return gid, start, total, points, owner


@pytest.mark.parametrize("n,density,big,max_points", [
    (1, 1.0, 0, 1 << 20), (31, 0.5, 0, 1 << 20), (4095, 0.3, 0, 1 << 20), (4096, 1.0, 0, 1 << 20), (4097, 0.9, 0, 5000),
    (70_001, 0.0, 0, 1 << 20), (70_001, 0.02, 300_000, 1 << 20), (70_001, 0.6, 1_000_000, 900_000),
    (4096 * 4096, 0.01, 0, 1 << 23), (4096 * 4096 + 1, 0.01, 70_000, 1 << 23), ((32 << 20) + 5, 0.01, 0, 1 << 23),
])
def test_scan_edges(n, density, big, max_points):
    import torch

    rng = np.random.default_rng(n)
    pad = (n + 31) // 32 * 32
    bits = np.zeros(pad, bool)
    bits[:n] = rng.random(n) < density
    counts = rng.integers(0, 30, pad).astype(np.uint32)  # zeros among the marked ones too
    if big and bits.any():
        counts[np.flatnonzero(bits)[bits.sum() // 2]] = big
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
