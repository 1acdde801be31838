"""The blocked PD smoother against the oracle's steps, bit for bit, where its
tiling and its branches can go wrong: image sizes around the tile (56 x 16) and
column-pair edges, step counts that are no multiple of the steps per launch,
warm starts that reach the scaled divisions (values below 2^-100, alone and
beside norms above 1) and the IEEE ones (1e30, not finite) and a non-finite image weight."""
import numpy as np
import pytest
import torch

from bitcmp import bit_diff
from cvt_gb300 import params as P
from cvt_gb300 import scenes

pytestmark = pytest.mark.gpu


def _warm(kind, rng, shape):
    u = rng.uniform(-1.0, 1.0, shape).astype(np.float32)
    u[..., 3] = 1.0
    if kind == "zeros":
        u[:] = 0.0
    elif kind == "tiny":                     # exact zeros beside 1e-33 .. 1e-42
        u[..., :3] *= (10.0 ** rng.uniform(-42, -33, shape[:-1] + (3,))).astype(np.float32)
        u[rng.random(shape[:-1]) < 0.3, :3] = 0.0
    elif kind == "steep":                    # norms well above 1
        u[..., :3] *= 300.0
    elif kind == "steeptiny":                # norms above 1 beside components of 1e-20 .. 1e-44
        u[..., 0] *= 300.0
        u[..., 1:3] *= (10.0 ** rng.uniform(-44, -20, shape[:-1] + (2,))).astype(np.float32)
    elif kind == "huge":
        u[rng.random(shape[:-1]) < 0.02, :3] = 1e30
    elif kind == "nonfinite":
        m = rng.random(shape[:-1])
        u[m < 0.01, 0] = np.inf
        u[m > 0.99, 2] = np.nan
    return u


@pytest.mark.parametrize("W,H", [(1, 1), (2, 3), (3, 40), (55, 15), (56, 16), (57, 17), (61, 33), (113, 49)])
@pytest.mark.parametrize("kind,steps", [("mixed", 3), ("zeros", 30), ("tiny", 9), ("steep", 8), ("steeptiny", 2),
                                        ("huge", 6),                                         ("nonfinite", 5)])
def test_smoother_bits(cuda, oracle, W, H, kind, steps):
    from cvt_gb300.stereo import PMHuberStereo
    rng = np.random.default_rng(W * 1000 + H * 10 + steps)
    sc = scenes.make_scene(max(W, 4), max(H, 4), 2, 6.0, seed=W + H)
    left, right = sc.left[:H, :W].copy(), sc.right[:H, :W].copy()
    if kind == "nonfinite":
        left[H // 2, W // 2, 0] = np.nan
    p = P.default_params(P.PRESET_BASELINE, patchsize=2, depthmax=6.0, iterations=2, pd_iterations=steps)
    st = PMHuberStereo(0, p)
    cl, cr = torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda()
    _, cp = st.depthMapResumable(None, cl, cr, 2, 6.0, 2, stop=0, save=True)
    warm = np.stack([_warm(kind, rng, (H, W, 4)) for _ in range(2)])
    cp["smooth"] = torch.from_numpy(warm).cuda()
    _, out = st.depthMapResumable(None, cl, cr, 2, 6.0, 2, resume=cp, stop=1, save=True)
    torch.cuda.synchronize()
    S = out["states"].cpu().numpy()
    for v, img in ((0, left), (1, right)):
        chk = oracle.consistency(S[v], S[1 - v], p.maxdispdiff, p.maxanglediff, 1 - v)
        chk = chk[0] if isinstance(chk, tuple) else chk
        f = oracle.fill_state(chk, 6.0, 1 - v)
        want = oracle.pd_apply(warm[v].copy(), f, oracle.edge_weight(img), 5.0, steps)
        got = out["smooth"][v].cpu().numpy()
        bad = bit_diff(got, want)
        assert not bad.any(), (v, kind, np.argwhere(bad)[:4])


@pytest.mark.parametrize("W,H", [(56, 16), (59, 18), (120, 33)])
def test_inpaint_tile_edges(cuda, oracle, W, H):
    from cvt_gb300.stereo import PMHuberStereo
    sc = scenes.make_scene(W, H, 2, 6.0, seed=W + H)
    p = P.default_params(P.PRESET_BASELINE, patchsize=2, depthmax=6.0, iterations=3)
    st = PMHuberStereo(0, p)
    dm = torch.empty(0, device="cuda")
    st.depthMapInpaint(dm, torch.from_numpy(sc.left).cuda(), torch.from_numpy(sc.right).cuda(), 2, 6.0, 3, 4)
    torch.cuda.synchronize()
    want, _ = oracle.depthmap_inpaint(p, sc.left, sc.right)
    assert not bit_diff(dm.cpu().numpy(), want).any()
