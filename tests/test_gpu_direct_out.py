"""Results in the caller's device memory: packed and pitched float maps (which the kernels write themselves), maps off
the floats' boundaries and host maps (which take a copy) hold the same bytes, for the winner-take-all depth and both
fusion variants, the first keyframe's zeros included; nothing beside a pitched map's rows is written."""
import ctypes

import numpy as np
import pytest

from probabilistic_mapping_b200 import _lib, scene
from probabilistic_mapping_b200.mapper import StereoMapper

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


class Dst:
    """A W x H float map at a byte offset with a byte pitch, on the device or the host."""

    def __init__(self, W, H, offset, pitch, device):
        self.W, self.H, self.offset, self.pitch = W, H, offset, pitch
        self.buf = torch.full((offset + pitch * H + 16,), 0x5A, dtype=torch.uint8, device="cuda" if device else "cpu")

    def ptr(self):
        return ctypes.c_void_p(self.buf.data_ptr() + self.offset)

    def read(self):
        b = self.buf.cpu().numpy()
        rows = np.stack([b[self.offset + y * self.pitch:self.offset + y * self.pitch + 4 * self.W] for y in range(self.H)])
        mask = np.ones(len(b), bool)
        for y in range(self.H):
            mask[self.offset + y * self.pitch:self.offset + y * self.pitch + 4 * self.W] = False
        assert (b[mask] == 0x5A).all()
        return rows.tobytes()


@pytest.mark.parametrize("W,H,D,prec", [(61, 43, 64, 0), (64, 48, 96, 0), (47, 33, 256, 0), (61, 43, 128, 1)])
@pytest.mark.parametrize("variant", [None, _lib.PM_FUSION_GPU, _lib.PM_FUSION_CPU_PATH])
def test_same_bytes_everywhere(W, H, D, prec, variant):
    seq = scene.make_sequence(W, H, 0.8125 * W, 2, 3, 9)
    kinds = [(0, 4 * W, False), (0, 4 * W, True), (16, 4 * W + 20, True), (4, 4 * W, True), (2, 4 * W + 6, True), (0, 4 * W + 12, False)]
    got = []
    for offset, pitch, device in kinds:
        m = StereoMapper(W, H, D, precision=prec, num_paths=8, fusion_variant=variant or 0, max_sources=2, rho0=0.1)
        m.initIntrinsic(seq[0].K, 0.0, 0.02)
        out = []
        for fs in seq:
            m.initReference(fs.ref)
            for s in range(2):
                m.update(fs.srcs[s], fs.R_ref, fs.T_ref, fs.R_srcs[s], fs.T_srcs[s])
            d, v = Dst(W, H, offset, pitch, device), Dst(W, H, offset, pitch, device)
            if variant is None:
                assert m.lib.pm_output(m.h, d.ptr(), pitch) == 0
                m.synchronize()
                out.append(d.read())
            else:
                dp = lambda a: np.ascontiguousarray(a, np.float64).ctypes.data_as(ctypes.POINTER(ctypes.c_double))  # noqa: E731
                R, T = np.ascontiguousarray(fs.R_ref), np.ascontiguousarray(fs.T_ref)
                f = float(fs.K[0, 0])
                assert m.lib.pm_output_fusion(m.h, d.ptr(), pitch, v.ptr(), pitch, dp(R), dp(T), f, f, W / 2, H / 2) == 0
                m.synchronize()
                out += [d.read(), v.read()]
            out.append(m.wta_depth().tobytes())
        got.append(out)
        m.close()
    assert any(np.frombuffer(x, np.float32).any() for x in got[0])
    for k, out in zip(kinds[1:], got[1:]):
        assert out == got[0], k
