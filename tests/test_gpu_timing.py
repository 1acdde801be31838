"""propagate_ms is the time of the propagation launches: with timing on, all of
them lie in the timed intervals, also where the views' passes would overlap
otherwise.  Compared with a memory budget that rules the overlap out (24 bytes
per pixel), best of three runs each; and timing changes no result."""
import pytest
import torch

from bitcmp import bit_diff
from cvt_gb300 import params as P
from cvt_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_propagate_ms_covers_the_passes(cuda):
    from cvt_gb300.stereo import PMHuberStereo
    W, H = 321, 243
    sc = scenes.make_scene(W, H, 5, 40.0, seed=9)
    L, R = torch.from_numpy(sc.left).cuda(), torch.from_numpy(sc.right).cuda()
    p = P.default_params(P.PRESET_BASELINE, patchsize=17, depthmax=40.0, iterations=4, pd_iterations=250)
    ms, maps = [], []
    for budget in (1 << 40, 24 * W * H):
        st = PMHuberStereo(0, p)
        st.set_memory_budget(budget)
        maps.append(st.depthMap(None, L, R, 17, 40.0, 4, 4).cpu().numpy())
        st.set_timing(True)
        best = float("inf")
        for _ in range(3):
            st.reset_stats()
            dm = st.depthMap(None, L, R, 17, 40.0, 4, 4)
            s = st.stats()
            assert s["propagate_launches"] == 8
            best = min(best, s["propagate_ms"])
        maps.append(dm.cpu().numpy())
        ms.append(best)
    assert all(not bit_diff(m, maps[0]).any() for m in maps)
    assert abs(ms[0] / ms[1] - 1.0) < 0.05, ms
