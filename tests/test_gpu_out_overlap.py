"""Fused depth and variance into device memory that the two maps share in part or in whole: the variance is written
after the depth, as for maps in the host's memory."""
import ctypes

import numpy as np
import pytest

from probabilistic_mapping_b200 import _lib, scene
from probabilistic_mapping_b200.mapper import StereoMapper

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# (pitch of the depth, of the variance, offset of the variance) in floats
@pytest.mark.parametrize("layout", ["same", "a row on", "between the rows", "a pixel on", "other pitch"])
@pytest.mark.parametrize("variant", [_lib.PM_FUSION_GPU, _lib.PM_FUSION_CPU_PATH])
def test_shared_memory(layout, variant):
    W, H, D, S = 161, 123, 64, 2
    pd, pv, off = {"same": (W, W, 0), "a row on": (W, W, W), "between the rows": (2 * W, 2 * W, W), "a pixel on": (W, W, 1),
                   "other pitch": (W + 3, W, 5)}[layout]
    seq = scene.make_sequence(W, H, 0.8125 * W, S, 4, 11)
    dp = lambda a: np.ascontiguousarray(a, np.float64).ctypes.data_as(ctypes.POINTER(ctypes.c_double))  # noqa: E731
    results = []
    for shared in (False, True):
        m = StereoMapper(W, H, D, num_paths=8, fusion_variant=variant, max_sources=S, rho0=0.1)
        m.initIntrinsic(seq[0].K, 0.0, 0.02)
        out = []
        for fs in seq:
            m.initReference(fs.ref)
            for s in range(S):
                m.update(fs.srcs[s], fs.R_ref, fs.T_ref, fs.R_srcs[s], fs.T_srcs[s])
            R, T, f = np.ascontiguousarray(fs.R_ref), np.ascontiguousarray(fs.T_ref), float(fs.K[0, 0])
            n = off + max(pd, pv) * H + 8
            if shared:
                buf = torch.full((n,), -7.0, device="cuda")
                d, v = buf.data_ptr(), buf.data_ptr() + 4 * off
            else:
                bd, bv = torch.empty((H, pd), device="cuda"), torch.empty((H, pv), device="cuda")
                d, v = bd.data_ptr(), bv.data_ptr()
            assert m.lib.pm_output_fusion(m.h, ctypes.c_void_p(d), 4 * pd, ctypes.c_void_p(v), 4 * pv, dp(R), dp(T), f, f,
                                          W / 2, H / 2) == 0
            m.synchronize()
            if shared:
                out.append(buf.cpu().numpy())
            else:
                want = np.full(n, -7.0, np.float32)
                for y in range(H):
                    want[y * pd:y * pd + W] = bd[y, :W].cpu().numpy()
                for y in range(H):
                    want[off + y * pv:off + y * pv + W] = bv[y, :W].cpu().numpy()
                out.append(want)
        results.append(out)
        m.close()
    assert any((o != -7.0).any() and o.any() for o in results[0])
    for a, b in zip(*results):
        assert a.tobytes() == b.tobytes()
