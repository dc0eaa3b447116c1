"""The four-pixel winner-take-all kernel at its edges: every plane count, pixel counts that leave one, two
or three pixels in the last group, ties, planes that take no part, NaN and infinities; bit for bit
against the FP32 oracle, and against the one-pixel kernel that unaligned volumes take."""
import ctypes

import numpy as np
import pytest

import oracle
from test_gpu_stages import bits, config, vp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def volume(W, H, D, seed):
    rng = np.random.default_rng(seed)
    vol = rng.uniform(0.5, 2.0, size=(H, W, D)).astype(np.float32)
    for y in range(H):
        for x in range(W):
            kind = rng.integers(0, 6)
            at = rng.choice(D, size=int(rng.integers(1, 6)), replace=False)
            if kind < 3:
                vol[y, x, at] = 0.25           # ties, or one clear minimum
            elif kind == 3:
                vol[y, x, at[0]] = 0.0         # no overlap
            elif kind == 4:
                vol[y, x, 0 if at[0] % 2 else D - 1] = 0.1   # border planes
    return vol


def run_filter(lib, cfg, vol, offset, W, H, D, pad=0):
    buf = torch.empty(vol.size + 8, dtype=torch.float32, device="cuda")
    buf[offset:offset + vol.size] = torch.from_numpy(vol.reshape(-1)).cuda()
    depth = torch.zeros((H, W + pad), dtype=torch.float32, device="cuda")
    idx = torch.full((H, W), -7, dtype=torch.int32, device="cuda")
    p = ctypes.c_void_p(buf.data_ptr() + 4 * offset)
    assert lib.pm_stage_filter(ctypes.byref(cfg), p, vp(depth), 4 * (W + pad), vp(idx), None) == 0
    torch.cuda.synchronize()
    assert (depth.cpu().numpy()[:, W:] == 0).all()
    return depth.cpu().numpy()[:, :W], idx.cpu().numpy()


@pytest.mark.parametrize("D", [32, 64, 96, 128, 160, 192, 224, 256])
@pytest.mark.parametrize("W,H,compat,uniq", [(7, 5, 1, 0.95), (9, 5, 0, 0.0), (45, 42, 1, 0.0), (3, 3, 1, 0.95)])
def test_filter_bit_exact(pm_lib, D, W, H, compat, uniq):
    p = oracle.Params(W=W, H=H, D=D, drho=0.03, num_paths=4, tree_compat=compat, uniqueness=uniq)
    vol = volume(W, H, D, seed=D + W)
    want_depth, want_idx = oracle.filter_cost(p, vol, "f32")
    depth, idx = run_filter(pm_lib, config(p), vol, 0, W, H, D, pad=W % 2)
    assert (idx == want_idx).all()
    assert (bits(depth) == bits(want_depth)).all()


@pytest.mark.parametrize("D,offset", [(32, 1), (64, 2), (96, 3), (160, 1)])
def test_unaligned_and_special_values(pm_lib, D, offset):
    """The same volume through both kernels (the offset leaves it unaligned), special values included."""
    W, H = 45, 21
    p = oracle.Params(W=W, H=H, D=D, drho=0.03, num_paths=4, uniqueness=0.95)
    vol = volume(W, H, D, seed=3)
    rng = np.random.default_rng(4)
    for v in (np.nan, np.inf, -np.inf, np.float32(-3.4028235e38), np.float32(3.4028235e38)):
        for _ in range(40):
            vol[rng.integers(H), rng.integers(W), rng.integers(D)] = v
    vol[0, 0], vol[0, 1], vol[0, 2] = np.nan, np.inf, -np.inf
    a = run_filter(pm_lib, config(p), vol, 0, W, H, D)
    b = run_filter(pm_lib, config(p), vol, offset, W, H, D)
    assert (a[1] == b[1]).all()
    assert (bits(a[0]) == bits(b[0])).all()
