"""An infinite upstream gradient: a tap whose colour distance is exactly 0 has
0 times an infinite term in the image-1 gradient, a NaN, in every channel of
its window, as the terms added one by one give it."""
import numpy as np
import pytest
import torch

from cvt_gb300.params import PRESET_BASELINE, default_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("g", [np.inf, -np.inf])
@pytest.mark.parametrize("sx,sy", [(0.002, 0.001), (-0.002, 0.001), (0.001, -0.002), (-0.001, -0.002)])
@pytest.mark.parametrize("W,H", [(40, 9), (13, 9)])
def test_infinite_gradient(cuda, g, sx, sy, W, H):
    from cvt_gb300.stereo import PMHuberStereo
    left = np.full((H, W, 4), 0.5, np.float32)
    yy, xx = np.mgrid[0:H, 0:W]
    right = left + (0.01 + sx * (xx - 6) + sy * (yy - 4))[..., None].astype(np.float32)
    right[..., 3] = 0.5
    planes = np.zeros((H, W, 4), np.float32)
    planes[..., 2] = 0.25
    up = np.zeros((H, W), np.float32)
    up[4, 6] = g
    p = default_params(PRESET_BASELINE, patchsize=1, color_maxdiff=1.0, grad_maxdiff=1.0)
    st = PMHuberStereo(0, p)
    _, _, d1, _ = st.cost_adjoint(*(torch.from_numpy(t).cuda() for t in (left, right, planes)), 1,
                                  dcost=torch.from_numpy(up).cuda())
    d1 = d1.cpu().numpy()[..., :3]
    assert np.isnan(d1[3:6, 5:8]).all()
    assert (d1[:2] == 0).all() and (d1[7:] == 0).all()


@pytest.mark.parametrize("alpha", [np.nan, np.inf])
def test_alpha_not_finite(cuda, alpha):
    """A colour share that is not finite leaves NaN gradients at every pixel with
    support (a cost that is not 1e5), also where residuals are 0 or truncated."""
    from cvt_gb300.stereo import PMHuberStereo
    H, W = 9, 40
    rng = np.random.default_rng(3)
    left = rng.random((H, W, 4), np.float32)
    planes = np.zeros((H, W, 4), np.float32)
    p = default_params(PRESET_BASELINE, patchsize=1, color_alpha=float(alpha))
    st = PMHuberStereo(0, p)
    L = torch.from_numpy(left).cuda()
    C, dpl, d1, d2 = st.cost_adjoint(L, L, torch.from_numpy(planes).cuda(), 1, dcost=torch.ones((H, W), device="cuda"))
    m = C != 1e5
    assert m.any()
    for t in (dpl, d1, d2):
        assert torch.isnan(t[..., :3][m]).all()
