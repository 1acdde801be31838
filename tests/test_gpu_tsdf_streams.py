"""Ray casts of one volume on two streams at once, from different cameras, are
those of the casts one after the other: a cast only reads the volume, and the
brick marks that casts of many rays share are never cleared under a march."""
import numpy as np
import pytest
import torch

from bitcmp import bit_diff
from cvt_gb300 import tsdf

pytestmark = pytest.mark.gpu


def test_casts_on_two_streams(cuda, oracle):
    n, iw, ih = 96, 1000, 700               # beyond the ray count that takes the bricks
    g2w = np.eye(4, dtype=np.float32)
    g2w[0, 0] = g2w[1, 1] = g2w[2, 2] = 2.0 / n
    g2w[:3, 3] = (-1.0, -1.0, 1.0)
    K = np.array([[0.8 * iw, 0, iw / 2], [0, 0.8 * iw, ih / 2], [0, 0, 1]], np.float32)
    cams = []
    for x in (0.05, -0.2):
        E = np.eye(4, dtype=np.float32)
        E[:3, 3] = (x, -0.03, 0.1)
        cams.append(E)
    v = tsdf.TSDFVolume(g2w, n, n, n, 0.1)
    v.clear()
    depth = (1.9 + 0.3 * np.sin(np.arange(iw) / 60.0)[None, :] + np.zeros((ih, 1))).astype(np.float32)
    v.addDepthMap(K, cams[0], torch.from_numpy(depth).cuda(), 1.0)
    torch.cuda.synchronize()
    vol = v.volume().cpu().numpy()
    want = []
    for E in cams:
        T, Ti = oracle.tsdf_matrices(tsdf.projection(K, E), g2w)
        want.append(oracle.tsdf_raycast(vol, iw, ih, Ti, T, -1.0))
        assert (want[-1] > 0).mean() > 0.2
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = [[], []]
    for _ in range(40):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                outs[i].append(v.rayCastDepthMap(K, cams[i], iw, ih, -1.0))
    torch.cuda.synchronize()
    for i in range(2):
        for o in outs[i]:
            assert not bit_diff(o.cpu().numpy(), want[i]).any()
