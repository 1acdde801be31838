"""Resumed states that are not finite, in whole blocks of 32 pixels of a row
among finite ones: both refinements of such a block have no plane to evaluate.
The tap-parallel routes against the per-pixel one (a memory budget of 0), bit
for bit."""
import numpy as np
import pytest
import torch

from bitcmp import bit_diff
from cvt_gb300 import params as P
from cvt_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(70, 20), (161, 120)])       # all candidates by taps; the refinements alone
@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("what", ["all", "some"])
def test_nonfinite_states(cuda, W, H, exact, what):
    from cvt_gb300.stereo import PMHuberStereo
    sc = scenes.make_scene(W, H, 2, 9.0, seed=W)
    L, R = torch.from_numpy(sc.left).cuda(), torch.from_numpy(sc.right).cuda()
    p = P.default_params(P.PRESET_REFERENCE if exact else P.PRESET_BASELINE, patchsize=3, depthmax=9.0, iterations=3,
                         pd_iterations=4)
    st = PMHuberStereo(0, p)
    _, cp = st.depthMapResumable(None, L, R, 3, 9.0, 3, stop=1, save=True)
    s = cp["states"]
    if what == "all":
        s[..., 0], s[..., 3] = float("nan"), -1.0             # a cost below every other: the state stays
    else:
        s[:, ::3, 32:64, 2], s[:, ::3, 32:64, 3] = float("inf"), -1.0
        s[:, 1::5, :, 1] = float("nan")
    out = []
    for budget in (1 << 40, 0):
        st.set_memory_budget(budget)
        tr = {}
        dm, end = st.depthMapResumable(None, L, R, 3, 9.0, 3, resume=cp, save=True, trace=tr)
        torch.cuda.synchronize()
        out.append([t.cpu().numpy() for t in (dm, end["states"], end["smooth"], tr["winners"], tr["valid"])])
    assert what == "some" or not np.isfinite(out[0][1][..., :3]).all(-1).any()
    for a, b in zip(*out):
        assert not bit_diff(a, b).any()
