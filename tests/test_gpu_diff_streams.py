"""One loss engine used from several streams: its calls run in their order, the tensors that a call reads stay valid
until its stream has read them, and a captured forward and backward replay with the same results.  The loss and the
inverse-depth map are compared bit for bit with the synchronous calls; the gradients as in test_gpu_diff.py (atomic
sums: rtol 1e-4, atol 1e-9).  A sleep on a stream keeps its next launch back, so that calls out of order would meet
the wrong state."""
import numpy as np
import pytest

from probabilistic_mapping_b200 import scene
from probabilistic_mapping_b200.diff import DepthLossEngine, depth_loss

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SLEEP = 20_000_000   # clock cycles, about 10 ms


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(np.float32(a))).cuda()


def case(W, H, D, S, seeds):
    rho0, drho = scene.plane_range(D)
    args = []
    for seed in seeds:
        f = scene.make_frameset(W, H, 0.8125 * W, S, seed=seed)
        R = np.stack([f.R_srcs[s].T @ f.R_ref for s in range(S)])
        t = np.stack([f.R_srcs[s].T @ (f.T_ref - f.T_srcs[s]) for s in range(S)])
        args.append((cu(f.ref / 255.0), cu(f.srcs / 255.0), f.K, R, t, cu(1.0 / f.gt_depth)))
    return args, dict(rho0=rho0, rho_step=drho, temperature=0.05)


def same(got, want):
    (l1, r1, g1, p1), (l0, r0, g0, p0) = got, want
    assert float(l1) == l0 and torch.equal(r1, r0)
    np.testing.assert_allclose(g1.cpu().numpy(), g0.cpu().numpy(), rtol=1e-4, atol=1e-9)
    np.testing.assert_allclose(torch.as_tensor(p1).cpu().numpy(), p0, rtol=1e-4, atol=1e-9)


SIZES = [(61, 40, 32, 1, False), (320, 240, 64, 2, False), (130, 90, 64, 2, True)]


@pytest.mark.parametrize("W,H,D,S,store", SIZES)
def test_two_streams_in_turn(W, H, D, S, store):
    args, kw = case(W, H, D, S, (3, 4))
    e = DepthLossEngine(W, H, D, S, store_paths=store, **kw)
    want = []
    for a in args:
        loss, rho = e.forward(*a)
        want.append((loss, rho, *e.backward()))
    torch.cuda.synchronize()
    s = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = []
    for turn in range(2):
        with torch.cuda.stream(s[0]):
            fwd = e.forward_async(*args[0])
            torch.cuda._sleep(SLEEP)
            got.append((0, (*fwd, *e.backward_async())))
        with torch.cuda.stream(s[1]):
            fwd = e.forward_async(*args[1])
            bwd = e.backward_async()
            got.append((1, (*fwd, *bwd)))
        # forward on one stream, the synchronous backward on the other
        with torch.cuda.stream(s[0]):
            torch.cuda._sleep(SLEEP)
            fwd = e.forward_async(*args[0])
        with torch.cuda.stream(s[1]):
            got.append((0, (*fwd, *e.backward())))
    torch.cuda.synchronize()
    for i, g in got:
        same(g, want[i])
    e.close()


@pytest.mark.parametrize("W,H,D,S,store", SIZES)
def test_loss_function_on_two_streams(W, H, D, S, store):
    args, kw = case(W, H, D, S, (5, 6))
    e = DepthLossEngine(W, H, D, S, store_paths=store, **kw)
    want = []
    for a in args:
        loss, _ = e.forward(*a)
        want.append((loss, *e.backward()))
    torch.cuda.synchronize()
    s = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = []
    for i in (0, 1, 0, 1):
        ref, srcs, K, R, t, rgt = args[i]
        with torch.cuda.stream(s[i]):
            x, xi = srcs.clone().requires_grad_(True), torch.zeros((S, 6), dtype=torch.float64, device="cuda", requires_grad=True)
            loss = depth_loss(x, xi, e, ref, K, R, t, rgt)
            torch.cuda._sleep(SLEEP)
            gx, gxi = torch.autograd.grad(loss, (x, xi))
            got.append((i, loss, gx, gxi))
    torch.cuda.synchronize()
    for i, loss, gx, gxi in got:
        assert loss.item() == want[i][0]
        np.testing.assert_allclose(gx.cpu().numpy(), want[i][1].cpu().numpy(), rtol=1e-4, atol=1e-9)
        np.testing.assert_allclose(gxi.cpu().numpy(), want[i][2], rtol=1e-4, atol=1e-9)
    e.close()


def test_inputs_outlive_their_last_reference():
    W, H, D, S = 320, 240, 64, 2
    args, kw = case(W, H, D, S, (7, 8))
    e = DepthLossEngine(W, H, D, S, **kw)
    want = [e.forward(*a)[0] for a in args]
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    losses = []
    for a in args:
        ref, srcs, K, R, t, rgt = a
        tmp = [x.clone() for x in (ref, srcs, rgt)]   # of the default stream
        sizes = [x.shape for x in tmp]
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            torch.cuda._sleep(SLEEP)
            losses.append(e.forward_async(tmp[0], tmp[1], K, R, t, tmp[2])[0])
        del tmp
        e._keep = None   # as the next forward does
        junk = [torch.full(n, 0.5, device="cuda") for n in sizes for _ in range(3)]
        torch.cuda.current_stream().synchronize()
        del junk
    torch.cuda.synchronize()
    assert [x.item() for x in losses] == want
    e.close()


@pytest.mark.parametrize("W,H,D,S,store", SIZES[:2])
def test_captured_calls(W, H, D, S, store):
    args, kw = case(W, H, D, S, (9, 10))
    e = DepthLossEngine(W, H, D, S, store_paths=store, **kw)
    want = []
    for a in args:
        loss, rho = e.forward(*a)
        want.append((loss, rho, *e.backward()))
    ref, srcs, K, R, t, rgt = args[0]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = (*e.forward_async(ref, srcs, K, R, t, rgt), *e.backward_async())
    for _ in range(3):
        g.replay()
        between = (*e.forward_async(*args[1]), *e.backward_async())   # after the replay, on the same engine
        torch.cuda.synchronize()
        same(out, want[0])
        same(between, want[1])
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):   # an ordinary call on another stream waits for a replay, and a replay for it
        torch.cuda._sleep(SLEEP)
        other = (*e.forward_async(*args[1]), *e.backward_async())
    g.replay()
    with torch.cuda.stream(s):
        third = (*e.forward_async(*args[1]), *e.backward_async())
    torch.cuda.synchronize()
    same(other, want[1])
    same(out, want[0])
    same(third, want[1])
    e.close()
