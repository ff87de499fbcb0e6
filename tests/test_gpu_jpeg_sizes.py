"""The JPEG pixel stage at sizes where its grids wrap and end: one pixel, one
row or column of blocks, odd edges, more blocks than one pass of the transform
grid takes, and blocks without any coefficient — against the float64 oracle
within one level, as the fixtures."""
import importlib.util
from pathlib import Path

import numpy as np
import pytest

from oracle import jpeg as oj
from zig_ornament_gb300 import textures

pytestmark = pytest.mark.gpu

_spec = importlib.util.spec_from_file_location("make_jpeg", Path(__file__).resolve().parent / "golden" / "make_jpeg.py")
make_jpeg = importlib.util.module_from_spec(_spec)
_spec.loader.exec_module(make_jpeg)


@pytest.mark.parametrize("flip", [True, False], ids=["flip", "noflip"])
@pytest.mark.parametrize("w,h,sampling", [(1, 1, ((1, 1),) * 3), (9, 257, ((2, 2), (1, 1), (1, 1))),
                                          (515, 7, ((2, 1), (1, 1), (1, 1))), (601, 457, ((1, 1),) * 3)])
def test_pixels_match_the_oracle(w, h, sampling, flip):
    img = make_jpeg.synthetic_rgb(w, h, 3)
    img[h // 3:2 * h // 3] = 128   # grey: blocks whose coefficients are all zero
    out = make_jpeg.encode(img, [tuple(s) for s in sampling], [(3.0,), (4.0,)])
    data = out[0]
    planes = [textures.jpeg_coefficients(data, c) for c in range(3)]
    want = oj.to_rgba([oj.idct_plane(*p) for p in planes], sampling, w, h, True, flip)
    got = textures.read_jpeg(data, flip_y=flip, device=0)
    diff = np.abs(got.astype(int) - want.astype(int))
    assert diff.max() <= 1
