"""The routes a propagation pass can take — tap-parallel blocks (small images),
shared plane windows, every candidate per pixel — against the oracle, bit for
bit, at sizes around their tiles (32 columns, 16 rows) and windows from 3x3 to
larger than the image.  The memory budget selects the route."""
import numpy as np
import pytest
import torch

from bitcmp import bit_diff
from cvt_gb300 import params as P
from cvt_gb300 import scenes

pytestmark = pytest.mark.gpu

# budget, bytes per pixel: with both views' scratch apart, or one view at a time
PER_PIXEL = {"taps": 576, "taps_one": 320, "windows": 32, "windows_one": 24, "pixel": 0}


def _run(route, p, left, right):
    from cvt_gb300.stereo import PMHuberStereo
    H, W = left.shape[:2]
    st = PMHuberStereo(0, p)
    st.set_memory_budget(PER_PIXEL[route] * W * H)
    tr = {}
    dm = st.depthMap(None, torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda(), p.patchsize, p.depthmax,
                     p.iterations, 4, trace=tr)
    torch.cuda.synchronize()
    return dm.cpu().numpy(), {k: v.cpu().numpy() for k, v in tr.items()}


@pytest.mark.parametrize("W,H,patch", [(1, 1, 1), (1, 40, 3), (31, 5, 2), (32, 16, 1), (33, 17, 4), (39, 15, 6),
                                       (64, 33, 5), (65, 9, 31), (70, 50, 17), (97, 4, 9)])
@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("route", list(PER_PIXEL))
def test_route_bits(cuda, oracle, W, H, patch, exact, route):
    sc = scenes.make_scene(max(W, 6), max(H, 6), 2, 9.0, seed=W * 7 + H)
    left, right = np.ascontiguousarray(sc.left[:H, :W]), np.ascontiguousarray(sc.right[:H, :W])
    p = P.default_params(P.PRESET_REFERENCE if exact else P.PRESET_BASELINE, patchsize=patch, depthmax=9.0, iterations=7,
                         pd_iterations=4)
    if exact:
        p.rng = P.RNG_MWC64X if W % 2 else P.RNG_PHILOX
    got, ex = _run(route, p, left, right)
    want, wex = oracle.depthmap(p, left, right, trace=True)
    assert np.array_equal(ex["winners"], wex["winners"])
    assert np.array_equal(ex["valid"], wex["valid"])
    assert not bit_diff(ex["states"], wex["states"]).any()
    assert not bit_diff(got, want).any()


@pytest.mark.parametrize("route", ["taps", "windows", "pixel"])
@pytest.mark.parametrize("what", ["nan_image", "inf_cap", "nan_cap"])
def test_route_special_values(cuda, oracle, route, what):
    """NaN and infinite pixels; a truncation that is not finite (the first two
    routes mark a tap outside the images by a NaN term)."""
    sc = scenes.make_scene(50, 20, 2, 9.0, seed=3)
    left, right = sc.left.copy(), sc.right.copy()
    left[4, 7, 1], left[9, 30, 0], right[9, 20, 2] = np.nan, np.inf, np.nan
    p = P.default_params(P.PRESET_BASELINE, patchsize=4, depthmax=9.0, iterations=3, pd_iterations=2)
    if what == "inf_cap":
        p.color_maxdiff = float("inf")
    elif what == "nan_cap":
        p.grad_maxdiff = float("nan")
    got, ex = _run(route, p, left, right)
    want, wex = oracle.depthmap(p, left, right, trace=True)
    assert np.array_equal(ex["winners"], wex["winners"])
    assert not bit_diff(ex["states"], wex["states"]).any()
    assert not bit_diff(got, want).any()


@pytest.mark.parametrize("W,H,patch", [(33, 7, 3), (301, 203, 2), (64, 941, 1)])      # below and above 60000 pixels
@pytest.mark.parametrize("exact", [False, True])
def test_cost_field_bits(cuda, oracle, W, H, patch, exact):
    from cvt_gb300.stereo import PMHuberStereo
    rng = np.random.default_rng(W + H)
    left, right = rng.random((H, W, 4), np.float32), rng.random((H, W, 4), np.float32)
    s = np.zeros((H, W, 4), np.float32)
    s[..., 0] = rng.choice([1.0, 0.9, 1.4, -0.7, np.nan], (H, W))
    s[..., 1] = rng.uniform(-0.3, 0.3, (H, W))
    s[..., 2] = rng.uniform(-4, W / 3, (H, W))
    p = P.default_params(P.PRESET_REFERENCE if exact else P.PRESET_BASELINE, patchsize=patch)
    got = PMHuberStereo(0, p).cost(*(torch.from_numpy(t).cuda() for t in (left, right, s)))
    assert not bit_diff(got.cpu().numpy(), oracle.cost_field(p, left, right, s)).any()
