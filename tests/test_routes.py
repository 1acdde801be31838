"""The routes that calls take by image size and window (no GPU needed): narrow
images and small windows, which the tap-parallel kernels serve badly, go to a
thread per pixel."""
import ctypes

import pytest

from cvt_gb300 import params as P

TAPS, SWEEPS, COST, ADJOINT = 1, 2, 4, 8


def routes(w, h, patch, exact=False):
    from cvt_gb300 import _lib
    p = P.default_params(P.PRESET_REFERENCE if exact else P.PRESET_BASELINE, patchsize=patch)
    r = _lib.lib().cvtpm_tool_routes(ctypes.byref(p), w, h)
    return r if r < 0 else r & (TAPS | SWEEPS | COST | ADJOINT)


@pytest.mark.parametrize("w,h,patch", [(1, 8000, 17), (2, 4000, 5), (4, 4000, 17), (8, 4500, 17), (8, 4500, 5),
                                       (16, 8000, 17), (1, 2000, 9), (640, 480, 17), (240, 160, 1)])
@pytest.mark.parametrize("exact", [False, True])
def test_thread_per_pixel(w, h, patch, exact):
    assert routes(w, h, patch, exact) == 0


@pytest.mark.parametrize("w,h,patch", [(64, 48, 17), (64, 48, 3), (96, 72, 9), (31, 300, 17), (1, 1, 1)])
@pytest.mark.parametrize("exact", [False, True])
def test_small_images_by_taps(w, h, patch, exact):
    assert routes(w, h, patch, exact) & (TAPS | COST) == TAPS | COST


def test_lines_between():
    assert routes(160, 120, 17) == SWEEPS | COST | ADJOINT
    assert routes(320, 192, 17) & COST and not routes(320, 192, 17) & (TAPS | SWEEPS | ADJOINT)
    assert not routes(320, 192, 3) & COST


def test_bad_arguments():
    from cvt_gb300 import _lib
    assert _lib.lib().cvtpm_tool_routes(None, 8, 8) == -1
    assert routes(0, 8, 3) == -1 and routes(8, 8, 0) == -1
