"""Child process of tests/test_gpu_bounds_sites.py: the calls that tests/bounds_workload.py leaves out -- the
differentiation form (both layouts of its volumes, both tile heights of its cost adjoint, one to eight planes per
lane), the stage cost call (float images, quads in the volume's first rows, running means), the stored sum and
results written to the caller's device memory -- through the library that PM_STEREO_LIB names.  Saves every output and,
when the library keeps them, the bounds record and the sites reached, to the .npz given as argv[1].  Outputs that atomics
add up in any order are saved under names with a leading "~"."""
import ctypes
import os
import sys

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import torch  # noqa: E402

from probabilistic_mapping_b200 import _lib, scene  # noqa: E402
from probabilistic_mapping_b200.diff import DepthLossEngine  # noqa: E402
from probabilistic_mapping_b200.mapper import StereoMapper  # noqa: E402

LOSS = [   # width, height, planes, sources, store_paths, shift along x only
    (61, 40, 32, 1, False, False),
    (57, 31, 64, 2, False, True),        # samples exactly on the last row
    (130, 133, 64, 2, False, False),     # three volumes
    (283, 175, 128, 2, True, True),      # 16-row tiles
    (33, 35, 256, 4, False, False),
]
STAGE = [   # width, height, planes, sources, cost mode, with a count
    (67, 41, 32, 2, 0, False),
    (200, 150, 64, 5, 0, False),         # quads in the volume
    (201, 180, 128, 5, 1, False),        # (corrected mode)
    (67, 41, 32, 2, 1, True),
]
MAPPERS = [(97, 61, 96, 0, 0), (64, 49, 128, 1, 1)]   # width, height, planes, precision, fusion variant


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(np.float32(a))).cuda()


def vp(t):
    return ctypes.c_void_p(t.data_ptr() if t is not None else 0)


def losses(out):
    for n, (W, H, D, S, store, along_x) in enumerate(LOSS):
        rho0, drho = scene.plane_range(D)
        f = scene.make_frameset(W, H, 0.8125 * W, S, seed=500 + n)
        R = np.stack([f.R_srcs[s].T @ f.R_ref for s in range(S)])
        t = np.stack([f.R_srcs[s].T @ (f.T_ref - f.T_srcs[s]) for s in range(S)])
        if along_x:
            R[:], t[:, 1:] = np.eye(3), 0.0
        e = DepthLossEngine(W, H, D, S, store_paths=store, rho0=rho0, rho_step=drho, temperature=0.05)
        loss, rho = e.forward(cu(f.ref / 255.0), cu(f.srcs / 255.0), f.K, R, t, cu(1.0 / f.gt_depth))
        gs, gp = e.backward()
        out[f"d{n}_rho"], out[f"~d{n}_loss"] = rho.cpu().numpy(), np.array([loss])
        out[f"~d{n}_gs"], out[f"~d{n}_gp"] = gs.cpu().numpy(), gp
        e.close()


def stages(lib, out):
    for n, (W, H, D, S, mode, count) in enumerate(STAGE):
        rho0, drho = scene.plane_range(D)
        f = scene.make_frameset(W, H, 0.8125 * W, S, seed=600 + n)
        R = [f.R_srcs[s].T @ f.R_ref for s in range(S)]
        t = [f.R_srcs[s].T @ (f.T_ref - f.T_srcs[s]) for s in range(S)]
        hom = np.stack([np.concatenate([(f.K @ R[s] @ np.linalg.inv(f.K)).ravel(), f.K @ t[s]]) for s in range(S)])
        hom = np.ascontiguousarray(hom, np.float32)
        cfg = _lib.default_config(W, H, D)
        cfg.rho0, cfg.rho_step, cfg.cost_mode, cfg.num_paths = rho0, drho, mode, 8
        ref, srcs = cu(f.ref / 255.0), cu(f.srcs / 255.0)
        cost = torch.full((H, W, D), -1.0, device="cuda")
        cnt = torch.zeros((H, W, D), device="cuda") if count else None
        inv = torch.empty((H, W), dtype=torch.uint8, device="cuda")
        assert lib.pm_stage_calc_cost(ctypes.byref(cfg), vp(ref), vp(srcs), S, hom.ctypes.data_as(ctypes.POINTER(ctypes.c_float)),
                                      vp(cost), vp(cnt), vp(inv), None) == 0
        out[f"s{n}_cost"], out[f"s{n}_inv"] = cost.cpu().numpy(), inv.cpu().numpy()


def mappers(out):
    for n, (W, H, D, prec, variant) in enumerate(MAPPERS):
        rho0, drho = scene.plane_range(D)
        seq = scene.make_sequence(W, H, 0.8 * W, 2, 3, seed=700 + n)
        m = StereoMapper(W, H, D, rho0=rho0, precision=prec, sampler=0, num_paths=8, fusion_variant=variant, max_sources=2,
                         intensity_scale=1 / 255, p1=0.003, p2=0.01, tau_so=3.5 / 255)
        K = seq[0].K
        m.initIntrinsic(K, 0.0, drho)
        m.enable_stats(True)
        for k, fs in enumerate(seq):
            m.initReference(fs.ref)
            for s in range(2):
                m.update(fs.srcs[s], fs.R_ref, fs.T_ref, fs.R_srcs[s], fs.T_srcs[s])
            pitch = W + 3   # pitched maps of the caller
            a, b, c = (torch.full((H, pitch), -7.0, device="cuda") for _ in range(3))
            m.store_sgm(k == 1)
            assert m.lib.pm_output(m.h, vp(c), 4 * pitch) == 0
            dp = lambda x: np.ascontiguousarray(x, np.float64).ctypes.data_as(ctypes.POINTER(ctypes.c_double))  # noqa: E731
            R, T = np.ascontiguousarray(fs.R_ref, np.float64), np.ascontiguousarray(fs.T_ref, np.float64)
            assert m.lib.pm_output_fusion(m.h, vp(a), 4 * pitch, vp(b), 4 * pitch, dp(R), dp(T), K[0, 0], K[1, 1], K[0, 2],
                                          K[1, 2]) == 0
            m.synchronize()
            for name, x in (("fused", a), ("var", b), ("wta", c)):
                out[f"m{n}_k{k}_{name}"] = x.cpu().numpy()
        m.close()


def main(out_path):
    out = {}
    lib = _lib.load()
    losses(out)
    stages(lib, out)
    mappers(out)
    rec, sites = (ctypes.c_uint64 * 4)(), (ctypes.c_uint64 * 2)()
    st = [lib.pm_debug_bounds(rec, 1), lib.pm_debug_bounds_sites(sites, 1)]
    out["bounds_status"] = np.array(st, np.int64)
    out["bounds"] = np.array(list(rec), np.uint64)
    out["bounds_sites"] = np.array(list(sites), np.uint64)
    np.savez_compressed(out_path, **out)


if __name__ == "__main__":
    main(sys.argv[1])
