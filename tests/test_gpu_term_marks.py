"""The shared terms of the windows and of the tap-parallel blocks mark a tap
outside the images; a valid term that is itself a NaN still counts.  Large
pixel values and truncations that let the combined cost overflow (EXACT: 0 or
an overflow times an infinite sum), and truncations that are not finite,
against the oracle by route, bit for bit."""
import numpy as np
import pytest
import torch

from bitcmp import bit_diff
from cvt_gb300 import params as P
from cvt_gb300 import scenes

pytestmark = pytest.mark.gpu
PER_PIXEL = {"taps": 576, "windows": 32, "pixel": 0}


def _case(what, exact):
    sc = scenes.make_scene(60, 24, 2, 9.0, seed=5)
    left, right = sc.left.copy(), sc.right.copy()
    p = P.default_params(P.PRESET_REFERENCE if exact else P.PRESET_BASELINE, patchsize=3, depthmax=9.0, iterations=3,
                         pd_iterations=2)
    if what == "overflow":                   # alpha 1: the gradients' share is 0 times their sum
        left[6:18, 12:40, :3] *= np.float32(3e38)
        p.color_alpha, p.grad_maxdiff, p.color_maxdiff = 1.0, 3e38, 0.05
    elif what == "alpha":
        left[6:18, 12:40, :3] *= np.float32(1e10)
        p.color_alpha, p.grad_maxdiff, p.color_maxdiff = 1e30, 1e10, 1e10
    else:
        left[4, 7, 1], left[9, 30, 0], right[9, 20, 2] = np.nan, np.inf, np.nan
        v = {"inf": np.inf, "minus_inf": -np.inf, "nan": np.nan}[what]
        p.color_maxdiff = p.grad_maxdiff = float(v)
    return p, left, right


@pytest.mark.parametrize("route", list(PER_PIXEL))
@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("what", ["overflow", "alpha", "inf", "minus_inf", "nan"])
def test_terms(cuda, oracle, what, exact, route):
    from cvt_gb300.stereo import PMHuberStereo
    p, left, right = _case(what, exact)
    H, W = left.shape[:2]
    st = PMHuberStereo(0, p)
    st.set_memory_budget(PER_PIXEL[route] * W * H)
    tr = {}
    L, R = torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda()
    dm = st.depthMap(None, L, R, 3, 9.0, 3, 4, trace=tr)
    want, wex = oracle.depthmap(p, left, right, trace=True)
    assert not bit_diff(tr["states"].cpu().numpy(), wex["states"]).any()
    assert np.array_equal(tr["winners"].cpu().numpy(), wex["winners"])
    assert not bit_diff(dm.cpu().numpy(), want).any()
    s = wex["states"][0]
    got = st.cost(L, R, torch.from_numpy(s).cuda())
    assert not bit_diff(got.cpu().numpy(), oracle.cost_field(p, left, right, s)).any()
