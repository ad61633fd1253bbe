"""The sample draw's own steps against CUDA's functions over all floats that they are used for, and its
paired and single forms against the one in the reference's form, sample by sample."""
import ctypes
import os

import pytest

import gpsplat
import gpsutil

pytestmark = pytest.mark.gpu


def _library():
    gpsplat.load_library()
    return ctypes.CDLL(os.path.join(gpsutil.PKG, "libgps_check.so"))


def test_steps_over_all_floats():
    differ = (ctypes.c_ulonglong * 6)()
    assert _library().gps_check_draw_steps(differ) == 0
    assert list(differ) == [0, 0, 0, 0, 0, 0]


@pytest.mark.parametrize("salt", [1, 77, 123456])
def test_samples(salt):
    out = (ctypes.c_ulonglong * 2)()
    assert _library().gps_check_draws(ctypes.c_uint32(1_000_000), ctypes.c_uint32(64), ctypes.c_uint32(salt), out) == 0
    assert out[1] > 20_000_000
    assert out[0] == 0
