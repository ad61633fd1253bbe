"""The scan's 16384-Gaussian tiles, taken in four rounds or, with few survivors, at once (from bit to bit
or from word to word of the mask, up to 12 steps and 2560 survivors), and survivors that own many tiles (their warp writes four at a time from 129 on)."""
import ctypes

import numpy as np
import pytest

import gpsplat
from test_gpu_scan_edges import _scan_numpy

pytestmark = pytest.mark.gpu

BIG = 32 << 20  # Gaussians from which the tiles are 16384
GROUP = 4096 * 16384  # Gaussians up to which a block adds up the tile totals itself


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


@pytest.mark.parametrize("n,density", [
    (BIG + 5, 0.06), (BIG + 5, 0.156),  # about 12 steps, about 2560 survivors a tile: both ways
    (BIG + 16383, 0.4), (BIG + 1, 0.001), (GROUP + 1, 0.004), (GROUP + 20_000, 0.0),
])
def test_big_tiles(n, density):
    rng = np.random.default_rng(n)
    pad = (n + 31) // 32 * 32
    bits = np.zeros(pad, bool)
    bits[:n] = rng.random(n, np.float32) < density
    bits[5 * 16384 : 7 * 16384] = False
    bits[5 * 16384 : 5 * 16384 + 2560] = True  # exactly 2560 in one tile, one more in the next
    bits[7 * 16384 - 2561 : 7 * 16384] = True
    bits[n - 1] = True
    counts = rng.integers(0, 5, pad).astype(np.uint32)
    _run(counts, bits, n, 1 << 26)


@pytest.mark.parametrize("run,every", [(1, 700), (31, 600), (64, 640), (130, 2048), (385, 2048), (400, 16384), (2560, 16384)])
def test_neighbours_in_big_tiles(run, every):
    """Runs of survivors that start anywhere in a word: from word to word, a few of them in all words."""
    n = BIG + 129
    pad = (n + 31) // 32 * 32
    bits = (np.arange(pad) + 13) % every < run
    bits[n:] = False
    counts = np.random.default_rng(run).integers(0, 700, pad).astype(np.uint32)
    _run(counts, bits, n, 1 << 28)


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
