"""The differentiation form's samples on the image's last row and column, where the bilinear taps beside and below
lie outside: rectified poses (no rotation, a shift along x or y only), whose samples have an exactly integer
coordinate there.

Finite images: against the FP64 adjoint, with the bounds of test_gpu_diff.py (2 % of the pose gradient's norm, 5 %
of the image gradient's, 1e-3 of the loss).  Images with an infinite pixel, and a temperature whose reciprocal
overflows, give gradients that are not finite; they stay inside the caller's tensor: the words around it keep
their values.
"""
import ctypes

import numpy as np
import pytest

import oracle
from probabilistic_mapping_b200 import scene
from probabilistic_mapping_b200.diff import DepthLossEngine

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

F = 64.0   # a power of two: the homographies of the shifts have no rounding


def rectified(W, H, shifts, seed):
    """ref, srcs, K, R, t, rho_gt of a scene seen with the camera shifted, not turned; the images without their
    quantisation, so that no sample equals its reference value."""
    rng = np.random.default_rng(seed)
    cam = scene.Camera(W, H, F)
    world = scene.Scene(cam, seed, np.eye(3), np.zeros(3))
    ref, depth = world.render(np.eye(3), np.zeros(3), rng)
    srcs = np.stack([world.render(np.eye(3), np.asarray(b, np.float64), rng)[0] for b in shifts])
    R, t = np.stack([np.eye(3)] * len(shifts)), -np.asarray(shifts, np.float64)
    ref, srcs = (np.float32((x + rng.uniform(-0.5, 0.5, x.shape)) / 255.0) for x in (ref, srcs))
    return ref, srcs, cam.K, R, t, np.float32(1.0 / depth)


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


SHIFTS = [(0.1, 0.0, 0.0), (0.0, 0.1, 0.0), (-0.12, 0.0, 0.0), (0.0, -0.08, 0.0)]


# 8-row tiles and (from 283x175x128 on) 16-row tiles
@pytest.mark.parametrize("W,H,D,S,store", [(57, 31, 64, 2, False), (54, 33, 128, 4, True), (283, 175, 128, 2, True)])
def test_gradients_on_the_last_row_and_column(W, H, D, S, store):
    ref, srcs, K, R, t, rgt = rectified(W, H, SHIFTS[:S], 17)
    rho0, drho = scene.plane_range(D)
    p = oracle.DiffParams(W=W, H=H, D=D, S=S, rho0=rho0, drho=drho, temperature=0.05)
    e = DepthLossEngine(W, H, D, S, store_paths=store, rho0=rho0, rho_step=drho, temperature=0.05)
    loss, _ = e.forward(cu(ref), cu(srcs), K, R, t, cu(rgt))
    gs, gp = e.backward()
    gs = gs.cpu().numpy()
    e.close()
    loss64 = oracle.diff_forward(p, ref, srcs, K, R, t, rgt)[0]
    _, gs64, gp64 = oracle.diff_backward(p, ref, srcs, K, R, t, rgt)
    assert loss == pytest.approx(loss64, rel=1e-3)
    assert np.linalg.norm(gs64[0::2, -1]) > 0 and np.linalg.norm(gs64[1::2, :, -1]) > 0
    assert np.linalg.norm(gs - gs64) < 0.05 * np.linalg.norm(gs64)
    assert np.linalg.norm(gp - gp64) < 0.02 * np.linalg.norm(gp64)


# The source shifted along x reads the last row exactly.  An infinite pixel is taken in by the reference or by the
# other source, shifted in both directions (a sample on a row or column of its own gives 0 * infinity: not measured).
@pytest.mark.parametrize("W,H,D,store", [(57, 31, 32, False), (283, 175, 128, True)])
@pytest.mark.parametrize("where", ["ref", "first source", "last source", "temperature"])
def test_non_finite_adjoints_stay_inside(W, H, D, store, where):
    S, along = 2, 1 if where == "first source" else 0
    shifts = [(0.1, 0.07, 0.0), (0.1, 0.07, 0.0)]
    shifts[along] = (0.1, 0.0, 0.0)
    ref, srcs, K, R, t, rgt = rectified(W, H, shifts, 23)
    if where == "ref":
        ref[H // 2, W // 2] = np.inf
    elif where != "temperature":
        srcs[1 - along, H // 2, W // 2] = np.inf
    rho0, drho = scene.plane_range(D)
    e = DepthLossEngine(W, H, D, S, store_paths=store, rho0=rho0, rho_step=drho,
                        temperature=1e-39 if where == "temperature" else 0.05)
    e.forward(cu(ref), cu(srcs), K, R, t, cu(rgt))
    pad, n = W + 8, S * W * H
    buf = torch.full((n + 2 * pad,), 1234.5, dtype=torch.float32, device="cuda")
    gp = np.zeros(6 * S)
    st = e.lib.pm_diff_backward(e.h, ctypes.c_void_p(buf.data_ptr() + 4 * pad),
                                gp.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), None)
    assert st == 0
    torch.cuda.synchronize()
    out = buf.cpu().numpy()
    e.close()
    assert (out[:pad] == 1234.5).all() and (out[pad + n:] == 1234.5).all()
    assert not np.isfinite(out[pad:pad + n].reshape(S, H, W)[along, -1]).all()
