"""The differentiation form at the edges of its kernels' tiles: the cost adjoint's 28 x 8 and 28 x 16
position tiles, image sizes around them, every source count and plane count, against the FP64 adjoint.

The bounds are those of test_gpu_diff.py (the FP32 forward routes some minima and signs otherwise
than FP64): 2 % of the pose gradient's norm, 5 % of the image gradient's, 1e-3 of the loss.
"""
import numpy as np
import pytest

import oracle
from probabilistic_mapping_b200 import scene
from probabilistic_mapping_b200.diff import DepthLossEngine

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def run(W, H, D, S, store, seed=5, keep=None):
    fs = scene.make_frameset(W, H, 0.8125 * W, S, seed=seed)
    rho0, drho = scene.plane_range(D)
    p = oracle.DiffParams(W=W, H=H, D=D, S=S, rho0=rho0, drho=drho, temperature=0.05)
    ref, srcs = np.float32(fs.ref / 255.0), np.float32(fs.srcs / 255.0)
    rgt = np.float32(1.0 / fs.gt_depth)
    R = np.stack([fs.R_srcs[s].T @ fs.R_ref for s in range(S)])
    t = np.stack([fs.R_srcs[s].T @ (fs.T_ref - fs.T_srcs[s]) for s in range(S)])
    e = DepthLossEngine(W, H, D, S, store_paths=store, rho0=rho0, rho_step=drho, temperature=0.05)
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    loss, _ = e.forward(cu(ref), cu(srcs), fs.K, R, t, cu(rgt))
    gs, gp = e.backward()
    gs = gs.cpu().numpy()
    again, gp2 = e.backward()   # a second backward of the same forward
    np.testing.assert_allclose(again.cpu().numpy(), gs, rtol=1e-4, atol=1e-9)
    np.testing.assert_allclose(gp2, gp, rtol=1e-4, atol=1e-9)
    e.close()
    loss64 = oracle.diff_forward(p, ref, srcs, fs.K, R, t, rgt)[0]
    _, gs64, gp64 = oracle.diff_backward(p, ref, srcs, fs.K, R, t, rgt)
    return loss, gs, gp, loss64, gs64, gp64


@pytest.mark.parametrize("W,H,D,S,store", [
    (27, 14, 32, 1, False), (26, 15, 32, 2, True), (29, 16, 64, 3, False), (54, 17, 32, 4, True),
    (57, 31, 128, 2, False), (55, 33, 256, 1, True), (283, 175, 128, 1, False), (281, 159, 128, 2, True)])
def test_gradients_at_tile_edges(W, H, D, S, store):
    loss, gs, gp, loss64, gs64, gp64 = run(W, H, D, S, store)
    assert loss == pytest.approx(loss64, rel=1e-3)
    assert np.linalg.norm(gs - gs64) < 0.05 * np.linalg.norm(gs64)
    assert np.linalg.norm(gp - gp64) < 0.02 * np.linalg.norm(gp64)


@pytest.mark.parametrize("W,H,D,S,store,side", [(61, 40, 32, 1, False, False), (130, 90, 64, 2, True, True)])
def test_async_calls_give_the_same(W, H, D, S, store, side):
    """forward_async / backward_async leave on the device what forward / backward return, on the default stream
    and on another one, also when the next forward is queued before they are read."""
    fs = [scene.make_frameset(W, H, 0.8125 * W, S, seed=s) for s in (3, 4)]
    rho0, drho = scene.plane_range(D)
    e = DepthLossEngine(W, H, D, S, store_paths=store, rho0=rho0, rho_step=drho, temperature=0.05)
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(np.float32(a))).cuda()  # noqa: E731
    args = []
    for f in fs:
        R = np.stack([f.R_srcs[s].T @ f.R_ref for s in range(S)])
        t = np.stack([f.R_srcs[s].T @ (f.T_ref - f.T_srcs[s]) for s in range(S)])
        args.append((cu(f.ref / 255.0), cu(f.srcs / 255.0), f.K, R, t, cu(1.0 / f.gt_depth)))
    want = []
    for a in args:
        loss, rho = e.forward(*a)
        want.append((loss, rho, *e.backward()))
    torch.cuda.synchronize()
    got = []
    stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
    with torch.cuda.stream(stream):
        for a in args:
            loss, rho = e.forward_async(*a)
            got.append((loss, rho, *e.backward_async()))
    torch.cuda.synchronize()
    for (l0, r0, g0, p0), (l1, r1, g1, p1) in zip(want, got):
        assert l1.is_cuda and l1.dtype == torch.float64 and l1.item() == l0
        assert torch.equal(r0, r1)
        np.testing.assert_allclose(g1.cpu().numpy(), g0.cpu().numpy(), rtol=1e-4, atol=1e-9)
        np.testing.assert_allclose(p1.cpu().numpy(), p0, rtol=1e-4, atol=1e-9)
    e.close()
