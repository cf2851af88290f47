"""The single post passes' taps without clamps (post_taps.h), compiled for the host: no pixel takes them with a
position outside the image, wherever the sun is."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "project-marshmallow_gb300", "csrc")
F = np.float32


@pytest.fixture(scope="module")
def taps(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("taps") / "taps.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC,
                    os.path.join(HERE, "c_host", "post_taps.cpp"), "-o", out], check=True)
    return C.CDLL(out)


def _scan(fn, w, h, sx, sy):
    inside, bad = C.c_longlong(), C.c_longlong()
    fn(w, h, C.c_float(sx), C.c_float(sy), C.byref(inside), C.byref(bad))
    return inside.value, bad.value


def _suns(w, h):
    """The sun on fragments, beside them, in the middle, at the edges, outside, at infinity."""
    def at(i, n):
        return F(F(F(F(i) + F(0.5)) / F(n)) * F(2.0) - F(1.0))
    suns = [(0.0, 0.0), (1e-30, 0.0), (0.0, -1e-25), (1e-12, 1e-13), (3.0, -0.2), (1e20, 0.0), (np.inf, 0.0),
            (np.nan, 0.3), (-1.0, 1.0)]
    for i, j in ((0, 0), (w // 2, h // 2), (w - 1, h // 3), (w // 3, h - 1), (1, 1)):
        x, y = at(i, w), at(j, h)
        suns += [(x, y), (np.nextafter(x, F(2)), y), (x, np.nextafter(y, F(-2))), (x, 0.1)]
    return suns


@pytest.mark.parametrize("which", ["scan_radial", "scan_god_rays"])
@pytest.mark.parametrize("w,h", [(1, 1), (2, 3), (3, 3), (33, 9), (257, 129), (641, 361), (640, 360), (1367, 7),
                                 (32768, 5)])
def test_taps_are_inside(taps, which, w, h):
    most = 0
    for sx, sy in _suns(w, h):
        inside, bad = _scan(getattr(taps, which), w, h, sx, sy)
        assert bad == 0, (sx, sy, inside, bad)
        most = max(most, inside)
    if min(w, h) > 100:
        assert most > 0.4 * w * h  # the fast path is what most pixels take
