"""The ray cast's empty-brick stepping (taken for many rays) against the
oracle's plain march, bit for bit: extents that are no multiple of the bricks,
weights that are NaN, below and above 1, cameras inside and outside the volume."""
import numpy as np
import pytest
import torch

from bitcmp import bit_diff
from cvt_gb300 import tsdf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,cam", [((97, 70, 45), 0.0), ((66, 131, 35), 1.6), ((160, 9, 64), -0.4), ((64, 64, 64), 0.3)])
def test_raycast_bricks_larger(cuda, oracle, dims, cam):
    Wv, Hv, Dv = dims
    iw, ih = 1000, 700                      # beyond the ray count that takes the bricks
    rng = np.random.default_rng(sum(dims))
    g2w = np.eye(4, dtype=np.float32)
    g2w[0, 0], g2w[1, 1], g2w[2, 2] = 2.0 / Wv, 2.0 / Hv, 2.0 / Dv
    g2w[:3, 3] = (-1.0, -1.0, 1.0)
    K = np.array([[0.8 * iw, 0, iw / 2], [0, 0.8 * iw, ih / 2], [0, 0, 1]], np.float32)
    E = np.eye(4, dtype=np.float32)
    c, s = np.cos(0.05), np.sin(0.05)
    E[:3, :3] = np.array([[c, 0, s], [0, 1, 0], [-s, 0, c]])
    E[:3, 3] = (0.05, -0.03, -cam)
    v = tsdf.TSDFVolume(g2w, Wv, Hv, Dv, 0.15)
    v.clear()
    depth = (1.8 + 0.3 * np.sin(np.arange(iw) / 60.0)[None, :] + 0.2 * rng.random((ih, 1))).astype(np.float32) - cam
    v.addDepthMap(K, E, torch.from_numpy(np.maximum(depth, 0.0)).cuda(), 1.0)
    vol = v.volume()
    idx = torch.from_numpy(rng.integers(0, vol[..., 1].numel(), 60)).cuda()
    flat = vol.view(-1, 2)
    flat[idx[:20], 1] = float("nan")
    flat[idx[20:40], 1] = 0.5
    flat[idx[40:], 0], flat[idx[40:], 1] = -0.3, 2.0
    got = v.rayCastDepthMap(K, E, iw, ih, -1.0)
    torch.cuda.synchronize()
    T, Ti = oracle.tsdf_matrices(tsdf.projection(K, E), g2w)
    want = oracle.tsdf_raycast(vol.cpu().numpy(), iw, ih, Ti, T, -1.0)
    bad = bit_diff(got.cpu().numpy(), want)
    assert not bad.any(), int(bad.sum())
    assert (want > 0).mean() > 0.05         # surfaces were met
