"""pm_stage_calc_cost on images with more rows than a grid has blocks along y (65535), where its sources become quads
in the volume's first rows: bit for bit against the FP32 oracle."""
import ctypes

import numpy as np
import pytest

import oracle
from test_gpu_stages import bits, config, fptr, vp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("W,H,mode", [(4, 65535, 1), (4, 65536, 0), (5, 131101, 1)])
def test_tall_images(pm_lib, W, H, mode):
    rng = np.random.default_rng(H)
    S, D = 2, 32
    ref = rng.integers(0, 256, size=(H, W)).astype(np.uint8)
    srcs = rng.integers(0, 256, size=(S, H, W)).astype(np.uint8)
    p = oracle.Params(W=W, H=H, D=D, rho0=0.0, drho=0.05, cost_mode=mode, num_paths=4)
    homs = np.zeros((S, 12), np.float32)
    homs[:, [0, 4, 8]] = 1.0
    homs[:, 9:] = [[0.3, -5.5, 0.0], [-0.7, 3.25, 0.0]]
    want, cnt = oracle.calc_cost(p, ref, srcs, homs, "f32")
    assert (want >= 0).any() and (want < 0).any()
    rf, sf = torch.from_numpy(ref).cuda().float(), torch.from_numpy(srcs).cuda().float()
    cost = torch.empty((H, W, D), dtype=torch.float32, device="cuda")
    inv = torch.empty((H, W), dtype=torch.uint8, device="cuda")
    cfg = config(p)
    st = pm_lib.pm_stage_calc_cost(ctypes.byref(cfg), vp(rf), vp(sf), S, fptr(homs.reshape(-1)), vp(cost), None, vp(inv), None)
    assert st == 0
    torch.cuda.synchronize()
    assert (bits(cost.cpu().numpy()) == bits(want)).all()
    assert (inv.cpu().numpy().astype(bool) == (cnt == 0).any(axis=2)).all()
