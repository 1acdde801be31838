"""cost_adjoint where its row bookkeeping can go wrong — widths around the
32-lane rows, windows wider than the image, planes whose samples stand still,
jump several columns or run backwards — against the FP64 adjoint on entries
that no tap near a kink reaches, within 1e-3 of the entry plus 1e-5 of the
largest (FP32 sums of at most a few hundred terms)."""
import numpy as np
import pytest
import torch

from cvt_gb300 import scenes
from cvt_gb300.params import PRESET_BASELINE, default_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,patch", [(1, 1, 2), (5, 30, 3), (31, 7, 2), (32, 6, 4), (33, 9, 3), (66, 5, 6), (70, 12, 1),
                                       (301, 203, 2)])      # above 60000 pixels: a thread per pixel
@pytest.mark.parametrize("lr", [1, 0])
def test_adjoint_edges(cuda, oracle, W, H, patch, lr):
    from cvt_gb300.stereo import PMHuberStereo
    rng = np.random.default_rng(W * 100 + H)
    sc = scenes.make_scene(max(W, 8), max(H, 8), 2, 4.0, seed=W + H)
    L, R = np.ascontiguousarray(sc.left[:H, :W]), np.ascontiguousarray(sc.right[:H, :W])
    pl = np.zeros((H, W, 4), np.float32)
    a = rng.choice([0.02, 0.9, -1.3, 1.6], (H, W))       # x' = x - d: slopes 0.98, 0.1, 2.3 and -0.6
    pl[..., 0] = a
    pl[..., 1] = rng.uniform(-0.2, 0.2, (H, W))
    yy, xx = np.mgrid[0:H, 0:W]
    pl[..., 2] = rng.uniform(0, 3, (H, W)) - pl[..., 0] * xx - pl[..., 1] * yy
    if lr == 0:
        pl[..., :3] = -pl[..., :3]
    g = rng.normal(0, 1, (H, W)).astype(np.float32)
    g[rng.random((H, W)) < 0.1] = 0.0
    p = default_params(PRESET_BASELINE, patchsize=patch)
    st = PMHuberStereo(0, p)
    C, dpl, d1, d2 = (t.cpu().numpy() for t in st.cost_adjoint(
        *(torch.from_numpy(t).cuda() for t in (L, R, pl)), lr, dcost=torch.from_numpy(g).cuda()))
    C64, dpl64, d164, d264, amb = oracle.cost_adjoint_f64(p, L, R, pl, g, lr=lr, kink_eps=3e-6)
    for got, want, m in ((dpl, dpl64, amb[0]), (d1, d164, amb[1]), (d2, d264, amb[2])):
        got, want, ok = got[..., :3], want[..., :3], ~np.asarray(m, bool)
        scale = np.abs(want).max() if want.size else 0.0
        bad = np.abs(got - want)[ok] > 1e-3 * np.abs(want)[ok] + 1e-5 * scale
        assert not bad.any(), (int(bad.sum()), int(ok.sum()))
