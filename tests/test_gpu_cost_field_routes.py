"""The FAST cost field on either side of the line to two pixels a thread
(2600 blocks of 32 pixels of a row, windows from 13x13), odd heights and ragged
widths among them, and the evaluator that allocates nothing, against the
oracle, bit for bit."""
import ctypes

import numpy as np
import pytest
import torch

from bitcmp import bit_diff
from cvt_gb300 import _lib
from cvt_gb300 import params as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,patch", [(40, 1300, 6), (40, 1301, 6), (40, 1299, 6), (40, 1301, 5), (97, 653, 7)])
def test_cost_field(cuda, oracle, W, H, patch):
    from cvt_gb300.stereo import PMHuberStereo
    rng = np.random.default_rng(W + H)
    left, right = rng.random((H, W, 4), np.float32), rng.random((H, W, 4), np.float32)
    s = np.zeros((H, W, 4), np.float32)
    s[..., 0] = rng.choice([1.0, 0.9, 1.4, -0.7, np.nan], (H, W))
    s[..., 1] = rng.uniform(-0.3, 0.3, (H, W))
    s[..., 2] = rng.uniform(-4, W / 3, (H, W))
    p = P.default_params(P.PRESET_BASELINE, patchsize=patch)
    L, R, S = (torch.from_numpy(t).cuda() for t in (left, right, s))
    want = oracle.cost_field(p, left, right, s)
    assert not bit_diff(PMHuberStereo(0, p).cost(L, R, S).cpu().numpy(), want).any()
    out = torch.empty((H, W), device="cuda")
    rc = _lib.lib().cvtpm_cost_eval_noalloc(ctypes.byref(p), L.data_ptr(), R.data_ptr(), W, H, W * 16, S.data_ptr(),
                                            out.data_ptr(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    assert not bit_diff(out.cpu().numpy(), want).any()
