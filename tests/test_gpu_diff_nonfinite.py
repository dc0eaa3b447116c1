"""A NaN adjoint of the loss does not get lost on its way to the gradients.

The costs that take in an infinite pixel of the second source are NaN, and so is the adjoint of the SGM sum at their
pixels.  Along each path the predecessor's minimum plane receives minus the sum of the step's adjoints, NaN if one of
them is, so the NaN reaches the scanline's end.  The first source is shifted along x or not at all, so its samples
stay on their rows, and the vertical paths take the NaN to every row of its gradient: also where its samples equal
their reference values, whose terms have the sign 0 (0 times NaN is NaN), and also in images of noise, where hardly a
plane but the minimum passes its adjoint on by itself."""
import numpy as np
import pytest

from probabilistic_mapping_b200 import scene
from probabilistic_mapping_b200.diff import DepthLossEngine
from test_gpu_diff_border import cu, rectified

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("W,H,D,store", [(57, 121, 32, False), (90, 133, 128, False), (90, 133, 128, True), (64, 90, 256, True)])
@pytest.mark.parametrize("images", ["scene", "the first source is the reference", "noise"])
def test_every_row_receives_it(W, H, D, store, images):
    same = images == "the first source is the reference"
    ref, srcs, K, R, t, rgt = rectified(W, H, [(0.0 if same else 0.1, 0.0, 0.0), (0.1, 0.07, 0.0)], 31)
    if same:
        srcs[0] = ref
    if images == "noise":
        rng = np.random.default_rng(41)
        ref, srcs = np.float32(rng.random((H, W))), np.float32(rng.random((2, H, W)))
    srcs[1, H // 2, W // 2] = np.inf
    rho0, drho = scene.plane_range(D)
    e = DepthLossEngine(W, H, D, 2, store_paths=store, rho0=rho0, rho_step=drho, temperature=0.05)
    e.forward(cu(ref), cu(srcs), K, R, t, cu(rgt))
    gs, gp = e.backward()
    gs = gs.cpu().numpy()
    e.close()
    assert (~np.isfinite(gs[0])).any(axis=1).all()
    assert not np.isfinite(gp[0]).any()
