"""Images narrower than a warp's 32 pixels, on either side of the lines between
the routes, against the oracle: depthMap and the cost bit for bit, the adjoint
within 1e-3 of the FP64 entry plus 1e-5 of the largest away from kinks."""
import numpy as np
import pytest
import torch

from bitcmp import bit_diff
from cvt_gb300 import params as P
from cvt_gb300 import scenes

pytestmark = pytest.mark.gpu
SIZES = [(1, 70, 5), (2, 45, 9), (3, 400, 2), (5, 33, 17), (7, 90, 4), (12, 350, 6), (20, 340, 3), (33, 40, 31)]


def _pair(W, H):
    sc = scenes.make_scene(max(W, 8), max(H, 8), 2, 5.0, seed=W + H)
    return np.ascontiguousarray(sc.left[:H, :W]), np.ascontiguousarray(sc.right[:H, :W])


@pytest.mark.parametrize("W,H,patch", SIZES)
@pytest.mark.parametrize("exact", [False, True])
def test_depthmap_and_cost(cuda, oracle, W, H, patch, exact):
    from cvt_gb300.stereo import PMHuberStereo
    left, right = _pair(W, H)
    p = P.default_params(P.PRESET_REFERENCE if exact else P.PRESET_BASELINE, patchsize=patch, depthmax=5.0, iterations=3,
                         pd_iterations=3)
    st = PMHuberStereo(0, p)
    L, R = torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda()
    tr = {}
    dm = st.depthMap(None, L, R, patch, 5.0, 3, 4, trace=tr)
    want, wex = oracle.depthmap(p, left, right, trace=True)
    assert not bit_diff(tr["states"].cpu().numpy(), wex["states"]).any()
    assert np.array_equal(tr["winners"].cpu().numpy(), wex["winners"])
    assert not bit_diff(dm.cpu().numpy(), want).any()
    s = np.zeros((H, W, 4), np.float32)
    rng = np.random.default_rng(W)
    s[..., 0], s[..., 1] = rng.choice([1.0, 0.8, 1.5, -0.6], (H, W)), rng.uniform(-0.2, 0.2, (H, W))
    s[..., 2] = rng.uniform(-2, 2, (H, W))
    got = st.cost(L, R, torch.from_numpy(s).cuda())
    assert not bit_diff(got.cpu().numpy(), oracle.cost_field(p, left, right, s)).any()


@pytest.mark.parametrize("W,H,patch", SIZES)
@pytest.mark.parametrize("images", [False, True])
def test_adjoint(cuda, oracle, W, H, patch, images):
    from cvt_gb300.stereo import PMHuberStereo
    rng = np.random.default_rng(W * 100 + H)
    L, R = _pair(W, H)
    pl = np.zeros((H, W, 4), np.float32)
    yy, xx = np.mgrid[0:H, 0:W]
    pl[..., 0], pl[..., 1] = rng.choice([0.02, 0.9, -1.3, 1.6], (H, W)), rng.uniform(-0.2, 0.2, (H, W))
    pl[..., 2] = rng.uniform(0, 3, (H, W)) - pl[..., 0] * xx - pl[..., 1] * yy
    g = rng.normal(0, 1, (H, W)).astype(np.float32)
    p = P.default_params(P.PRESET_BASELINE, patchsize=patch)
    st = PMHuberStereo(0, p)
    C, dpl, d1, d2 = st.cost_adjoint(*(torch.from_numpy(t).cuda() for t in (L, R, pl)), 1,
                                     dcost=torch.from_numpy(g).cuda(), want_images=images)
    fwd = st.cost_adjoint(*(torch.from_numpy(t).cuda() for t in (L, R, pl)), 1)[0]
    assert not bit_diff(C.cpu().numpy(), fwd.cpu().numpy()).any()
    C64, dpl64, d164, d264, amb = oracle.cost_adjoint_f64(p, L, R, pl, g, lr=1, kink_eps=3e-6)
    for got, want, m in ((dpl, dpl64, amb[0]),) + (((d1, d164, amb[1]), (d2, d264, amb[2])) if images else ()):
        got, want, ok = got.cpu().numpy()[..., :3], want[..., :3], ~np.asarray(m, bool)
        bad = np.abs(got - want)[ok] > 1e-3 * np.abs(want)[ok] + 1e-5 * np.abs(want).max()
        assert not bad.any(), (int(bad.sum()), int(ok.sum()))
