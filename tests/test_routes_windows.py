"""Where a pass shares plane windows (no GPU needed): not for windows of a few
taps, nor where the image holds less than about half of a window's columns."""
import ctypes

import pytest

from cvt_gb300 import params as P

WINDOWS = 16


@pytest.mark.parametrize("w,h,patch,want", [(1242, 375, 17, True), (321, 243, 3, True), (640, 480, 2, False),
                                            (640, 480, 1, False), (16, 8000, 17, True), (8, 8000, 17, False),
                                            (8, 8000, 9, False), (8, 8000, 5, True), (4, 20000, 5, False),
                                            (1, 8000, 3, False), (30, 4000, 31, True)])
@pytest.mark.parametrize("preset", [P.PRESET_REFERENCE, P.PRESET_BASELINE])
def test_windows(w, h, patch, want, preset):
    from cvt_gb300 import _lib
    p = P.default_params(preset, patchsize=patch)
    assert bool(_lib.lib().cvtpm_tool_routes(ctypes.byref(p), w, h) & WINDOWS) == want
