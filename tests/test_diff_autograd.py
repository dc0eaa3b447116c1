"""The torch.autograd side of the differentiable loss (DepthLoss) around an engine that stands in for the library:
gradients for one and for several output gradients at once (is_grads_batched), for output gradients that need a
gradient themselves, and repeated backwards of one forward."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from probabilistic_mapping_b200.diff import depth_loss  # noqa: E402

S, H, W = 2, 5, 7


class Engine:
    """A loss whose gradients are fixed arrays, returned in new tensors as the library's are."""

    def __init__(self):
        rng = np.random.default_rng(0)
        self.gs = torch.from_numpy(rng.normal(size=(S, H, W)).astype(np.float32))
        self.gp = torch.from_numpy(rng.normal(size=(S, 6)))

    def forward_async(self, ref, srcs, K, R, t, rho_gt):
        return torch.tensor(0.25, dtype=torch.float64), rho_gt

    def backward_async(self):
        return self.gs.clone(), self.gp.clone()


def loss_of(e, dtype=torch.float64):
    srcs = torch.zeros((S, H, W), requires_grad=True)
    xi = torch.zeros((S, 6), dtype=dtype, requires_grad=True)
    img = torch.zeros((H, W))
    loss = depth_loss(srcs, xi, e, img, np.eye(3), np.stack([np.eye(3)] * S), np.zeros((S, 3)), img)
    return loss, srcs, xi


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_one_output_gradient(dtype):
    e = Engine()
    loss, srcs, xi = loss_of(e, dtype)
    for _ in range(2):   # a second backward of the same forward
        gs, gp = torch.autograd.grad(loss, (srcs, xi), torch.tensor(3.0, dtype=torch.float64), retain_graph=True)
        assert gs.dtype == torch.float32 and gp.dtype == dtype
        assert torch.equal(gs, e.gs * 3.0) and torch.equal(gp, e.gp.to(dtype) * 3.0)


def test_several_output_gradients_at_once():
    e = Engine()
    loss, srcs, xi = loss_of(e)
    g = torch.tensor([1.0, -2.0, 0.5], dtype=torch.float64)
    gs, gp = torch.autograd.grad(loss, (srcs, xi), g, is_grads_batched=True)
    assert torch.equal(gs, e.gs * g.float().reshape(3, 1, 1, 1)) and torch.equal(gp, e.gp * g.reshape(3, 1, 1))


def test_output_gradient_that_needs_a_gradient():
    e = Engine()
    loss, srcs, xi = loss_of(e)
    g = torch.tensor(2.0, dtype=torch.float64, requires_grad=True)
    gs, gp = torch.autograd.grad(loss, (srcs, xi), g, create_graph=True)
    dg, = torch.autograd.grad(gs.double().sum() + gp.sum(), g)
    assert dg.item() == pytest.approx(float(e.gs.double().sum() + e.gp.sum()), rel=1e-6)
