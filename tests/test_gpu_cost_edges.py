"""The cost kernel's rules at their edges, bit for bit against the FP32 oracle: sums of exactly zero (identical
saturated images), sums around and below the bound under which the running mean's division is looked at one
voxel at a time, and an image whose width and size leave the default floor bias no room (set_floor_bias)."""
import numpy as np
import pytest

import oracle
from probabilistic_mapping_b200 import scene
from probabilistic_mapping_b200.mapper import StereoMapper
from test_gpu_stages import bits

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def cost_of(W, H, D, ref, srcs, poses, K, drho, scale, mode):
    from cuda.bindings import runtime as rt
    m = StereoMapper(W, H, D, cost_mode=mode, intensity_scale=scale, max_sources=max(1, len(srcs)))
    m.initIntrinsic(K, 0.0, drho)
    m.initReference(ref)
    for img, (R, T) in zip(srcs, poses):
        m.update(img, np.eye(3), np.zeros(3), R, T)
    m.output()
    vol = torch.empty((H, W, D), dtype=torch.float32, device="cuda")
    err, = rt.cudaMemcpy(vol.data_ptr(), m.buffers().cost, vol.numel() * 4, rt.cudaMemcpyKind.cudaMemcpyDeviceToDevice)
    assert err == rt.cudaError_t.cudaSuccess
    homs = np.stack([m.homography(i) for i in range(len(srcs))])
    out = vol.cpu().numpy()
    m.close()
    return out, homs


def setup(W, H, S, seed):
    fs = scene.make_frameset(W, H, 0.8125 * W, S, seed)
    poses = [(fs.R_ref.T @ fs.R_srcs[s], fs.R_ref.T @ (fs.T_srcs[s] - fs.T_ref)) for s in range(S)]
    return fs, poses


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("scale", [1.0, 1e-28, 1e-30, 3e-32, 1e-36])
def test_zero_and_tiny_sums(mode, scale):
    W, H, D, S = 61, 43, 32, 3
    fs, poses = setup(W, H, S, 7)
    ref, srcs = fs.ref.copy(), fs.srcs.copy()
    for img in [ref] + list(srcs):   # a saturated band, identical in all frames, and a black one
        img[10:24] = 255
        img[30:36] = 0
    drho = 0.06
    p = oracle.Params(W=W, H=H, D=D, rho0=0.0, drho=drho, intensity_scale=scale, cost_mode=mode, num_paths=4)
    got, homs = cost_of(W, H, D, ref, srcs, poses, fs.K, drho, scale, mode)
    want, _ = oracle.calc_cost(p, ref, srcs, homs, "f32")
    # (reference mode samples every pixel near the corner of the source too, so only corrected sums are exactly 0)
    assert ((want == 0).any() or mode == 0) and (want > 0).any() and (want < 0).any()
    assert (bits(got) == bits(want)).all()


def test_floor_bias():
    """bits(1.5 * 2^23) * (W + 1) = 1023 * 2^22 modulo 2^32 for this width: with more than 2^22 pixels the default
    bias would let the index wrap."""
    W, D = 346, 32
    H = (1 << 22) // W + 3
    assert (0x4B400000 * (W + 1)) % (1 << 32) + W * H >= 1 << 32
    rng = np.random.default_rng(1)
    ref = rng.integers(0, 256, (H, W)).astype(np.uint8)
    src = rng.integers(0, 256, (H, W)).astype(np.uint8)
    K = np.array([[0.8 * W, 0, W / 2], [0, 0.8 * W, H / 2], [0, 0, 1.0]])
    R = scene.rodrigues(np.array([0.0, 0.0, 1.0]), 0.002)
    p = oracle.Params(W=W, H=H, D=D, rho0=0.0, drho=0.04, intensity_scale=1.0, cost_mode=1, num_paths=4)
    got, homs = cost_of(W, H, D, ref, [src], [(R, np.array([0.05, -0.03, 0.01]))], K, 0.04, 1.0, 1)
    want, _ = oracle.calc_cost(p, ref, src[None], homs, "f32")
    assert (bits(got) == bits(want)).all()


@pytest.mark.parametrize("W,H,D,S,mode", [(203, 151, 64, 3, 0), (97, 263, 96, 5, 0), (401, 305, 32, 7, 0), (203, 57, 64, 3, 0),
                                          (333, 251, 64, 5, 1), (401, 305, 32, 9, 0)])
def test_stage_cost_through_the_volume(pm_lib, W, H, D, S, mode):
    """pm_stage_calc_cost keeps the sources' quads in the first rows of the volume where the other rows are worth it
    (all but the fourth case, which is too small, and the last, whose quads would take every row)."""
    import ctypes
    from test_gpu_stages import config, upload_images, vp
    fs, poses = setup(W, H, S, 11)
    p = oracle.Params(W=W, H=H, D=D, rho0=0.05, drho=0.03, intensity_scale=1.0, cost_mode=mode, num_paths=4)
    homs = np.stack([oracle.compose_homography(fs.K, np.eye(3), np.zeros(3), R, T) for R, T in poses]).astype(np.float32)
    want, _ = oracle.calc_cost(p, fs.ref, fs.srcs, homs, "f32")
    rf, sf = upload_images(pm_lib, fs, 1.0)
    buf = torch.full((W * H * D + 64,), 7.0, dtype=torch.float32, device="cuda")
    inv = torch.full((H, W), 9, dtype=torch.uint8, device="cuda")
    cfg = config(p)
    hp = np.ascontiguousarray(homs).ctypes.data_as(ctypes.POINTER(ctypes.c_float))
    for guard in (0, 1):   # 16-byte aligned, and not
        cost = ctypes.c_void_p(buf.data_ptr() + 4 * guard)
        assert pm_lib.pm_stage_calc_cost(ctypes.byref(cfg), vp(rf), vp(sf), S, hp, cost, None, vp(inv), None) == 0
        torch.cuda.synchronize()
        got = buf[guard:guard + W * H * D].cpu().numpy().reshape(H, W, D)
        assert (bits(got) == bits(want)).all()
        assert (inv.cpu().numpy() == (want < 0).any(-1)).all()
        assert (buf[guard + W * H * D:] == 7.0).all()
