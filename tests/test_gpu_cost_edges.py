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
