"""A batch whose pairs take different routes (shared windows; too narrow for
them; small) in both modes, against the plain calls, bit for bit."""
import pytest
import torch

from bitcmp import bit_diff
from cvt_gb300 import params as P
from cvt_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [0, 1])
@pytest.mark.parametrize("preset", [P.PRESET_REFERENCE, P.PRESET_BASELINE])
def test_mixed_routes(cuda, lanes, preset):
    from cvt_gb300.stereo import PMHuberStereo
    p = P.default_params(preset, patchsize=5, iterations=3, pd_iterations=6)
    pairs = []
    for W, H in ((120, 90), (3, 400), (40, 30), (64, 200)):
        sc = scenes.make_scene(max(W, 8), H, 2, 4.0, seed=W)
        pairs.append((torch.from_numpy(sc.left[:, :W].copy()).cuda(), torch.from_numpy(sc.right[:, :W].copy()).cuda(), 4.0))
    st = PMHuberStereo(0, p)
    if lanes:
        st.set_batch_lanes(lanes)
    else:
        st.set_batch_knobs(1, 16, 4)          # pinned knobs: the phase-batched schedule
    outs = st.depthMapBatched(pairs)
    outs = st.depthMapBatched(pairs, outs=outs)
    torch.cuda.synchronize()
    one = PMHuberStereo(0, p)
    for (L, R, d), got in zip(pairs, outs):
        want = one.depthMap(None, L, R, 5, d, 3, 4)
        assert not bit_diff(got.cpu().numpy(), want.cpu().numpy()).any(), tuple(L.shape)
