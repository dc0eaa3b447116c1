"""The path pairs in one launch: image shapes around the rule that picks one or four scanlines per block (an SM's
share of scanlines below or above twelve: 1776 in all), wide and tall images, last blocks of one to four scanlines,
4 and 8 paths, plane counts whose reduction tree drops planes; bit for bit against the FP32 oracle."""
import ctypes

import numpy as np
import pytest

import oracle
from test_gpu_stages import bits, config, vp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("W,H,D,paths", [(3, 3, 32, 8), (5, 67, 64, 8), (67, 5, 32, 8), (130, 41, 96, 4), (41, 130, 64, 8),
                                         (300, 292, 32, 8), (300, 293, 32, 8), (293, 302, 32, 8), (301, 295, 32, 8),
                                         (887, 888, 32, 4), (889, 890, 32, 4),
                                         # planes that the reduction tree leaves out
                                         (45, 31, 96, 8), (45, 31, 160, 8), (31, 45, 192, 4), (45, 31, 224, 8)])
def test_sgm_bit_exact(pm_lib, W, H, D, paths):
    rng = np.random.default_rng(W * H)
    p = oracle.Params(W=W, H=H, D=D, drho=0.03, num_paths=paths)
    ref = rng.integers(0, 255, size=(H, W)).astype(np.uint8)
    cost = rng.uniform(0.0, 60.0, size=(H, W, D)).astype(np.float32)
    cost[rng.integers(0, H, 9), rng.integers(0, W, 9), rng.integers(0, D, 9)] = -1.0   # pixels without a measurement
    want = oracle.sgm(p, ref, cost, "f32")
    cfg = config(p)
    dref, dcost = torch.from_numpy(ref.astype(np.float32)).cuda() * p.intensity_scale, torch.from_numpy(cost).cuda()
    out = torch.empty_like(dcost)
    scratch = torch.empty((max(1, paths // 2 - 1),) + tuple(dcost.shape), dtype=torch.float32, device="cuda")
    assert pm_lib.pm_stage_sgm(ctypes.byref(cfg), vp(dcost), vp(dref), vp(out), vp(scratch), None) == 0
    torch.cuda.synchronize()
    assert (bits(out.cpu().numpy()) == bits(want)).all()
