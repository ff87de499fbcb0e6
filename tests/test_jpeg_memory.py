"""The entropy decoder's memory: by what the picture can have, not by the
buffer's length or the number of scans."""
import ctypes as C
from pathlib import Path

import numpy as np
import pytest

from zig_ornament_gb300 import _lib, textures

GOLDEN = Path(__file__).resolve().parent / "golden"
FIX = np.load(GOLDEN / "jpeg_fixtures.npz")


def _data(name):
    return (GOLDEN / "jpeg" / f"{name}.jpg").read_bytes()


def test_a_buffer_beyond_two_gigabytes(tmp_path):
    """A picture at the start of a buffer of more than 2^31 bytes (a sparse file here)."""
    data = np.frombuffer(_data("rgb444_128x96"), np.uint8)
    path = tmp_path / "long.jpg"
    with open(path, "wb") as f:
        f.truncate((1 << 31) + (1 << 20))
    buf = np.memmap(path, np.uint8, "r+")
    buf[:len(data)] = data
    want = FIX["rgb444_128x96/coef0"]
    got = np.zeros(want.shape, np.int16)
    w, h = C.c_uint32(), C.c_uint32()
    lib = _lib.load()
    assert lib.orn_jpeg_coefficients(C.c_void_p(buf.ctypes.data), buf.size, 0, C.c_void_p(got.ctypes.data), got.size,
                                     C.byref(w), C.byref(h), None) == _lib.ORN_OK
    assert np.array_equal(got, want)


@pytest.mark.parametrize("name", ["rgb422_multiscan", "rgb444_q1", "rgb420_restart"])
@pytest.mark.parametrize("times", [1, 2, 40])
def test_scans_repeated(name, times):
    """Each scan of a component replaces the one before."""
    data = _data(name)
    first = data.index(b"\xff\xda")
    again = data[:-2] + (times - 1) * data[first:-2] + data[-2:]
    for c in range(3):
        coef, _ = textures.jpeg_coefficients(again, c)
        assert np.array_equal(coef, FIX[f"{name}/coef{c}"])
