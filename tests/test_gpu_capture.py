"""depthMap under stream capture: a captured graph stays valid when the context
then runs smaller pairs, whose tap-parallel passes take more scratch than the
captured pair's shared windows, and such a pair can be captured after a larger
one alone."""
import pytest
import torch

from bitcmp import bit_diff
from cvt_gb300 import params as P
from cvt_gb300 import scenes

pytestmark = pytest.mark.gpu


def _pair(W, H):
    sc = scenes.make_scene(W, H, 3, 12.0, seed=W)
    return torch.from_numpy(sc.left).cuda(), torch.from_numpy(sc.right).cuda()


@pytest.mark.parametrize("exact", [False, True])
def test_graph_and_other_sizes(cuda, exact):
    from cvt_gb300.stereo import PMHuberStereo
    p = P.default_params(P.PRESET_REFERENCE if exact else P.PRESET_BASELINE, patchsize=3, depthmax=12.0, iterations=3,
                         pd_iterations=8)
    st = PMHuberStereo(0, p)
    pairs = [_pair(160, 120), _pair(90, 60), _pair(64, 48)]
    want = []
    for L, R in pairs:                       # other contexts: their scratch is not this one's
        want.append(PMHuberStereo(0, p).depthMap(None, L, R, 3, 12.0, 3, 4).cpu().numpy())
    outs = [torch.zeros(L.shape[:2], device="cuda") for L, _ in pairs]
    st.depthMap(outs[0], *pairs[0], 3, 12.0, 3, 4)
    torch.cuda.synchronize()
    graphs = []
    for (L, R), o in zip(pairs[:2], outs):   # the second pair's size was never run
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            st.depthMap(o, L, R, 3, 12.0, 3, 4)
        graphs.append(g)
    st.depthMap(outs[2], *pairs[2], 3, 12.0, 3, 4)
    torch.cuda.synchronize()
    junk = [torch.full((1 << 18,), float("nan"), device="cuda") for _ in range(16)]
    for i in (0, 1, 0):
        outs[i].zero_()
        graphs[i].replay()
        torch.cuda.synchronize()
        assert not bit_diff(outs[i].cpu().numpy(), want[i]).any(), i
    assert not bit_diff(outs[2].cpu().numpy(), want[2]).any()
    del junk
