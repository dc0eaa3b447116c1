"""Performance cases of the motion-stereo library: what users of it run, through its public
entry points, over the range of sizes it takes.

`listed()` gives the fixed cases, `draw(rng)` one more of the same ranges.  `prepare(case, seed)`
makes what a program holds before the call (frames and poses of a synthetic scene, the mapper,
batch or engine), `run(state)` is one pass of it, `work(case)` the bytes and operations of a pass,
and `exact(case, seed)` the pass in 64 bits where its outputs are continuous in the inputs.

The kinds:
  map    a StereoMapper, one keyframe per pass: initReference, an update per source frame, then
         output (fuse "none") or outputFusion (fuse "gpu" or "cpu", the two fusion variants).
         host: numpy frames and results, as a camera node has them; else CUDA tensors.
  stage  the stage-level calls that stand in for the reference's launch wrappers, on CUDA tensors:
         cost volume, SGM sum, winner-take-all and one fusion step.
  batch  a StereoBatch of several sequences, one keyframe of each per pass.
  diff   the differentiable depth loss: a training step (loss, gradients of the source images and
         of the poses) or, with train false, its evaluation only.

Scenes are six textured planes 1 to 8 m away, ray-cast to noisy 8-bit frames; sources lie 5 to 15
cm from the reference frame with rotations up to 2 degrees.  A state holds two keyframes and passes
alternate between them, so that the fusion step has a moving camera.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from probabilistic_mapping_b200 import _lib
from probabilistic_mapping_b200.batch import StereoBatch
from probabilistic_mapping_b200.diff import DepthLossEngine, depth_loss
from probabilistic_mapping_b200.mapper import StereoMapper

KEYFRAMES = 2
RHO_MIN, RHO_MAX = 0.1, 2.0   # inverse-depth range of the planes


# ---- the cases --------------------------------------------------------------------------------

def _map(name, W, H, D, S, paths=8, precision="fp32", sampler="exact", mode="reference", fuse="none", host=False,
         scaled=True):
    return dict(name=name, kind="map", W=W, H=H, D=D, S=S, paths=paths, precision=precision, sampler=sampler,
                mode=mode, fuse=fuse, host=host, scaled=scaled)


def _batch(name, sizes, count, S, host, persistent=False):
    return dict(name=name, kind="batch", sizes=sizes, count=count, S=S, paths=8, precision="fp16",
                sampler="texture_f32", mode="reference", host=host, persistent=persistent)


def _diff(name, W, H, D, S, train=True, store=False):
    return dict(name=name, kind="diff", W=W, H=H, D=D, S=S, train=train, store=store)


def listed():
    return [
        # the smallest useful map: a thumbnail keyframe of a tracker's preview, bound by latency
        _map("map_96x64x32_s1", 96, 64, 32, 1, paths=4),
        # the reference node's own configuration (64 planes, 3 sources, 4 paths, 0..255 intensities, its
        # CPU fusion variant) with frames and results in host memory
        _map("node_640x480x64_s3", 640, 480, 64, 3, paths=4, fuse="cpu", host=True, scaled=False),
        # the plain FP32 form at the benchmark's size, with the fusion step
        _map("map_640x480x128_s5", 640, 480, 128, 5, fuse="gpu"),
        # the FP16 form on camera frames of the precision tests' width, the reference's own sampling
        _map("fp16_752x480x128_s5", 752, 480, 128, 5, precision="fp16", sampler="texture_f32", fuse="gpu"),
        # odd sizes and a plane count that is no power of two, corrected 3x3 patches
        _map("odd_333x251x96_s2", 333, 251, 96, 2, mode="corrected"),
        # the largest single map of the benchmark's mixed batch, FP32 with the texture sampler
        _map("map_1280x720x192_s4", 1280, 720, 192, 4, sampler="texture_f32", fuse="gpu"),
        # the stage-level calls at the size that the reference's launch wrappers are compiled for
        dict(name="stage_640x480x64_s5", kind="stage", W=640, H=480, D=64, S=5, paths=4, mode="reference"),
        # the benchmark's batched form: 8 equal sequences, FP16, one CUDA-graph launch per step
        _batch("batch_8x640x480x128", "640x480x128", 8, 5, False),
        # sequences of three sizes, frames and results in host memory
        _batch("mixed_3x2_host", "320x240x64,640x480x128,1280x720x192", 2, 4, True),
        # gradients at the differentiation form's tested size, path states recomputed
        _diff("train_320x240x64_s2", 320, 240, 64, 2),
        # the smallest loss worth a gradient, and the largest with the path states kept
        _diff("train_96x64x32_s1", 96, 64, 32, 1),
        _diff("train_640x480x128_s3", 640, 480, 128, 3, store=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["map", "map", "map", "stage", "batch", "diff", "diff"])
    if kind == "batch":
        sizes = []
        for _ in range(rng.choice([1, 2])):
            w = _log_int(rng, 97, 500)
            sizes.append("%dx%dx%d" % (w, max(48, int(w * rng.uniform(0.5, 0.8))), 64 * rng.choice([1, 1, 2, 3])))
        c = _batch("", ",".join(sizes), rng.choice([1, 2, 3, 4]), rng.choice([2, 3, 4, 5]), rng.random() < 0.4,
                   rng.random() < 0.2)
        c["precision"] = rng.choice(["fp16", "fp16", "fp32"])
        c["sampler"] = rng.choice(["texture_f32", "exact"])
        c["paths"] = rng.choice([4, 8, 8])
    else:
        w = _log_int(rng, 64, 1100 if kind != "diff" else 560)
        h = max(48, int(w * rng.uniform(0.45, 0.85)))
        if kind == "diff":
            c = _diff("", w, h, rng.choice([32, 64, 64, 128]), rng.choice([1, 2, 2, 3]), rng.random() < 0.7,
                      rng.random() < 0.5)
        elif kind == "stage":
            c = dict(kind="stage", W=w, H=h, D=32 * rng.choice([1, 2, 2, 3, 4]), S=rng.choice([1, 2, 3, 5]),
                     paths=rng.choice([4, 8]), mode=rng.choice(["reference", "corrected"]))
        else:
            prec = rng.choice(["fp32", "fp32", "fp16"])
            d = 64 * rng.choice([1, 2, 2, 3]) if prec == "fp16" else 32 * rng.choice([1, 2, 2, 3, 4, 4, 6])
            c = _map("", w, h, d, rng.choice([1, 2, 3, 4, 5]), rng.choice([4, 8, 8]), prec,
                     rng.choice(["exact", "texture_f32"]), rng.choice(["reference", "reference", "corrected"]),
                     rng.choice(["none", "gpu", "gpu", "cpu"]), rng.random() < 0.3, rng.random() < 0.7)
    c.pop("name", None)
    return c


# ---- scenes -----------------------------------------------------------------------------------

def _rotation(axis, angle):
    axis = axis / np.linalg.norm(axis)
    k = np.array([[0, -axis[2], axis[1]], [axis[2], 0, -axis[0]], [-axis[1], axis[0], 0]])
    return np.eye(3) + np.sin(angle) * k + (1 - np.cos(angle)) * (k @ k)


class _Scene:
    """Six textured planes in front of a camera at the origin, ray-cast on the GPU in float64."""

    PLANES, OCTAVES, LATTICE = 6, 3, 128

    def __init__(self, W, H, seed):
        self.W, self.H, self.f = W, H, 0.8125 * W   # f = 520 at 640 columns
        self.K = np.array([[self.f, 0.0, W / 2], [0.0, self.f, H / 2], [0.0, 0.0, 1.0]])
        self.rng = np.random.default_rng(seed)
        r = self.rng
        Kinv = np.linalg.inv(self.K)
        n, c, e1, e2 = [], [], [], []
        for _ in range(self.PLANES):
            th, ph = np.deg2rad(40.0) * np.sqrt(r.uniform()), r.uniform(0, 2 * np.pi)
            normal = np.array([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), -np.cos(th)])
            a = np.cross(normal, [1.0, 0.0, 0.0])
            n.append(normal)
            c.append(r.uniform(1.0, 8.0) * (Kinv @ np.array([r.uniform(0, W), r.uniform(0, H), 1.0])))
            e1.append(a / np.linalg.norm(a))
            e2.append(np.cross(normal, e1[-1]))
        up = lambda v: torch.tensor(np.array(v), dtype=torch.float64, device="cuda")  # noqa: E731
        self.n, self.c, self.e1, self.e2 = up(n), up(c), up(e1), up(e2)
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(int(seed) * 7919 + 11)
        self.tables = torch.rand(self.PLANES, self.OCTAVES, self.LATTICE * self.LATTICE, generator=self.gen,
                                 device="cuda", dtype=torch.float64)
        v, u = torch.meshgrid(torch.arange(H, dtype=torch.float64, device="cuda"),
                              torch.arange(W, dtype=torch.float64, device="cuda"), indexing="ij")
        self.rays = torch.stack([(u - W / 2) / self.f, (v - H / 2) / self.f, torch.ones_like(u)], -1)

    def render(self, R, T):
        """(uint8 frame, depth) of the camera-to-world pose (R, T), both CUDA tensors."""
        T = torch.tensor(T, dtype=torch.float64, device="cuda")
        rays = self.rays @ torch.tensor(R, dtype=torch.float64, device="cuda").T
        t = ((self.c - T) * self.n).sum(-1) / (rays @ self.n.T)
        t, k = torch.where(t > 1e-6, t, torch.inf).min(-1)
        hit = torch.isfinite(t)
        X = T + rays * torch.where(hit, t, 1.0)[..., None] - self.c[k]
        s, q = (X * self.e1[k]).sum(-1), (X * self.e2[k]).sum(-1)
        out, tot = torch.zeros_like(t), 0.0
        tables = self.tables.reshape(-1)
        for o in range(self.OCTAVES):
            cell, L = 0.24 / 2 ** o, self.LATTICE
            base = (k * self.OCTAVES + o) * L * L
            i, j = torch.floor(s / cell), torch.floor(q / cell)
            a, b = s / cell - i, q / cell - j
            a, b = a * a * (3 - 2 * a), b * b * (3 - 2 * b)
            at = lambda di, dj: tables[base + ((j.long() + dj) % L) * L + (i.long() + di) % L]  # noqa: B023,E731
            top = torch.lerp(at(0, 0), at(1, 0), a)
            out += 0.5 ** o * torch.lerp(top, torch.lerp(at(0, 1), at(1, 1), a), b)
            tot += 0.5 ** o
        img = 255.0 * (0.5 + 1.6 * (out / tot - 0.5)).clamp(0.0, 1.0)
        img = torch.where(hit, img, 0.0)
        img = img + 2.0 * torch.randn(img.shape, generator=self.gen, device="cuda", dtype=torch.float64)
        return img.round().clamp(0, 255).to(torch.uint8), torch.where(hit, t, 0.0)


def _unit(rng):
    v = rng.normal(size=3)
    return v / np.linalg.norm(v)


def _keyframes(W, H, S, seed, count=KEYFRAMES):
    """The scene and `count` keyframes: (reference frame, its depth, pose, source frames and poses)."""
    sc = _Scene(W, H, seed)
    r, out = sc.rng, []
    for k in range(count):
        R, T = _rotation(np.array([0.0, 1.0, 0.0]), np.deg2rad(0.5) * k), np.array([0.04 * k, 0.0, 0.0])
        ref, depth = sc.render(R, T)
        srcs, Rs, Ts = [], [], []
        for _ in range(S):
            Ts.append(T + r.uniform(0.05, 0.15) * (R @ _unit(r)))
            Rs.append(R @ _rotation(_unit(r), np.deg2rad(2.0) * r.uniform()))
            srcs.append(sc.render(Rs[-1], Ts[-1])[0])
        out.append(dict(ref=ref, depth=depth, R=R, T=T, srcs=srcs, Rs=Rs, Ts=Ts))
    return sc, out


def _planes(D):
    return RHO_MIN, (RHO_MAX - RHO_MIN) / (D - 1)


def _params(case, D, scaled=True):
    """pm_config fields: the reference's parameters on 0..255 intensities, or the benchmark's on 0..1."""
    p = dict(rho0=_planes(D)[0], num_paths=case["paths"],
             cost_mode=_lib.PM_COST_CORRECTED if case["mode"] == "corrected" else _lib.PM_COST_REFERENCE,
             precision=_lib.PM_PREC_FP16 if case.get("precision") == "fp16" else _lib.PM_PREC_FP32,
             sampler=_lib.PM_SAMPLER_TEXTURE_F32 if case.get("sampler") == "texture_f32" else _lib.PM_SAMPLER_EXACT,
             max_sources=max(1, case["S"]))
    if scaled:
        p.update(intensity_scale=1 / 255, p1=0.003, p2=0.01, tau_so=3.5 / 255, uniqueness_ratio=0.95)
    return p


# ---- map: StereoMapper ------------------------------------------------------------------------

def _prepare_map(case, seed):
    W, H, D = case["W"], case["H"], case["D"]
    sc, frames = _keyframes(W, H, case["S"], seed)
    p = _params(case, D, case["scaled"])
    p["fusion_variant"] = _lib.PM_FUSION_CPU_PATH if case["fuse"] == "cpu" else _lib.PM_FUSION_GPU
    m = StereoMapper(W, H, D, **p)
    m.initIntrinsic(sc.K, 0.0, _planes(D)[1])
    if not case["host"]:
        m.set_stream(torch.cuda.current_stream().cuda_stream)
        out = [torch.empty(H, W, device="cuda") for _ in range(2)]
    else:
        for f in frames:
            f["ref"], f["srcs"] = f["ref"].cpu().numpy(), [x.cpu().numpy() for x in f["srcs"]]
        out = [np.empty((H, W), np.float32) for _ in range(2)]
    torch.cuda.synchronize()
    st = dict(kind="map", m=m, sc=sc, frames=frames, fuse=case["fuse"] != "none", out=out, at=0)
    if st["fuse"]:
        _run_map(st)   # the first keyframe only starts the fusion state
    return st


def _run_map(st):
    m, f, sc = st["m"], st["frames"][st["at"]], st["sc"]
    st["at"] = (st["at"] + 1) % KEYFRAMES
    m.initReference(f["ref"])
    for img, R, T in zip(f["srcs"], f["Rs"], f["Ts"]):
        m.update(img, f["R"], f["T"], R, T)
    if not st["fuse"]:
        return m.output(st["out"][0])
    return m.outputFusion(f["R"], f["T"], sc.f, sc.f, sc.W / 2, sc.H / 2, out=st["out"][0], variance=st["out"][1])


# ---- stage: the launch-wrapper calls ----------------------------------------------------------

def _homography(K, Rl, Tl, Rr, Tr):
    """H1 = K Rr^T Rl K^-1 and H2 = K Rr^T (Tl - Tr) (stereo_mapper.cpp:79-80)."""
    A = K @ Rr.T
    return np.concatenate([(A @ Rl @ np.linalg.inv(K)).reshape(-1), A @ (Tl - Tr)]).astype(np.float32)


def _stage_inputs(case, seed):
    sc, frames = _keyframes(case["W"], case["H"], case["S"], seed)
    f = frames[1]
    ref = f["ref"].float()
    srcs = torch.stack(f["srcs"]).float().contiguous()
    homs = np.stack([_homography(sc.K, f["R"], f["T"], R, T) for R, T in zip(f["Rs"], f["Ts"])])
    # a fusion state left by the previous keyframe
    g = sc.gen
    shape = (case["H"], case["W"])
    rand = lambda lo, hi: torch.rand(shape, generator=g, device="cuda") * (hi - lo) + lo  # noqa: E731
    state = [rand(0.0, 20.0), rand(1.0, 12.0), (frames[0]["depth"].float() * rand(0.95, 1.05)).contiguous(), rand(0.01, 4.0)]
    state[0] = torch.where(state[0] < 4.0, -1.0, state[0]).contiguous()   # cells without a state
    return sc, frames, ref.contiguous(), srcs, homs, state


def _prepare_stage(case, seed):
    W, H, D = case["W"], case["H"], case["D"]
    sc, frames, ref, srcs, homs, state = _stage_inputs(case, seed)
    cfg = _lib.default_config(W, H, D)
    for k, v in _params(case, D, False).items():
        setattr(cfg, k, v)
    cfg.rho_step = _planes(D)[1]
    dev = lambda *shape, dtype=torch.float32: torch.empty(shape, dtype=dtype, device="cuda")  # noqa: E731
    poses = []
    for a, b in ((0, 1), (1, 0)):   # previous keyframe a seen from b
        R = frames[b]["R"].T @ frames[a]["R"]
        t = frames[b]["R"].T @ (frames[a]["T"] - frames[b]["T"])
        poses.append((ctypes.c_float * 12)(*R.reshape(-1), *t))
    state2 = [torch.zeros(H, W, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    return dict(kind="stage", lib=_lib.load(), cfg=cfg, W=W, H=H, S=case["S"], ref=ref, srcs=srcs, homs=homs,
                cost=dev(H, W, D), sgm=dev(H, W, D), scratch=dev(case["paths"] // 2 - 1, H, W, D), depth=dev(H, W),
                fused=dev(H, W), index=dev(H, W, dtype=torch.int32), ztable=dev(H, W, dtype=torch.int64),
                table=dev(H, W, dtype=torch.int32), states=[state, state2], poses=poses,
                cam=(ctypes.c_float * 4)(sc.f, sc.f, W / 2, H / 2), at=0)


def _run_stage(st):
    lib, cfg, W, H = st["lib"], st["cfg"], st["W"], st["H"]
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    homs = st["homs"].ctypes.data_as(ctypes.POINTER(ctypes.c_float))
    _lib.check(lib.pm_stage_calc_cost(ctypes.byref(cfg), p(st["ref"]), p(st["srcs"]), st["S"], homs, p(st["cost"]),
                                      None, None, stream), None, "pm_stage_calc_cost")
    _lib.check(lib.pm_stage_sgm(ctypes.byref(cfg), p(st["cost"]), p(st["ref"]), p(st["sgm"]), p(st["scratch"]),
                                stream), None, "pm_stage_sgm")
    _lib.check(lib.pm_stage_filter(ctypes.byref(cfg), p(st["sgm"]), p(st["depth"]), 0, p(st["index"]), stream), None,
               "pm_stage_filter")
    st["fused"].copy_(st["depth"])
    pre, cur = st["states"][st["at"]], st["states"][1 - st["at"]]
    ptrs = lambda s: (ctypes.c_void_p * 4)(*[t.data_ptr() for t in s])  # noqa: E731
    _lib.check(lib.pm_stage_depth_fuse(W, H, st["poses"][st["at"]], st["cam"], p(st["fused"]), ptrs(pre), ptrs(cur),
                                       p(st["ztable"]), p(st["table"]), stream), None, "pm_stage_depth_fuse")
    st["at"] = 1 - st["at"]
    return dict(cost=st["cost"], sgm=st["sgm"], depth=st["depth"], index=st["index"], fused=st["fused"],
                table=st["table"], state=list(cur))


# ---- batch: StereoBatch -----------------------------------------------------------------------

def _batch_sizes(case):
    shapes = [tuple(int(x) for x in s.split("x")) for s in case["sizes"].split(",")]
    return [s for s in shapes for _ in range(case["count"])]


def _prepare_batch(case, seed):
    sizes = _batch_sizes(case)
    b = StereoBatch([dict(width=W, height=H, num_planes=D, **_params(case, D)) for W, H, D in sizes], case["S"],
                    host_io=case["host"], persistent=case["persistent"])
    seqs = []
    for i, (W, H, D) in enumerate(sizes):
        sc, frames = _keyframes(W, H, case["S"], seed * 101 + i)
        b.init_intrinsic(i, sc.K, _planes(D)[1])
        if case["host"]:
            for f in frames:
                f["ref"], f["srcs"] = f["ref"].cpu().numpy(), [x.cpu().numpy() for x in f["srcs"]]
            out = [np.empty((H, W), np.float32) for _ in range(2)]
        else:
            out = [torch.empty(H, W, device="cuda") for _ in range(2)]
        seqs.append((frames, out))
    torch.cuda.synchronize()
    st = dict(kind="batch", b=b, seqs=seqs, at=0)
    _run_batch(st)   # the first keyframe builds the graph and starts the fusion states
    return st


def _run_batch(st):
    b = st["b"]
    for i, (frames, _) in enumerate(st["seqs"]):
        f = frames[st["at"]]
        b.set_frame(i, 0, f["ref"])
        for s, img in enumerate(f["srcs"]):
            b.set_frame(i, 1 + s, img)
        b.set_poses(i, f["R"], f["T"], f["Rs"], f["Ts"])
    st["at"] = (st["at"] + 1) % KEYFRAMES
    b.run()
    b.synchronize()
    return [b.copy_output(i, *out) for i, (_, out) in enumerate(st["seqs"])]


# ---- diff: the differentiable depth loss ------------------------------------------------------

def _diff_inputs(case, seed):
    sc, frames = _keyframes(case["W"], case["H"], case["S"], seed, 1)
    f = frames[0]
    ref, srcs = f["ref"].float() / 255, (torch.stack(f["srcs"]).float() / 255).contiguous()
    rho_gt = torch.where(f["depth"] > 0, 1.0 / f["depth"].clamp(min=1e-3), 0.0).float().contiguous()
    R0 = np.stack([R.T @ f["R"] for R in f["Rs"]])   # source from reference
    t0 = np.stack([R.T @ (f["T"] - T) for R, T in zip(f["Rs"], f["Ts"])])
    # pose estimates a few millimetres and a few hundredths of a degree off
    xi = torch.tensor(sc.rng.normal(size=(case["S"], 6)) * 5e-4, dtype=torch.float32, device="cuda")
    return sc.K, ref.contiguous(), srcs, rho_gt, R0, t0, xi


def _prepare_diff(case, seed):
    K, ref, srcs, rho_gt, R0, t0, xi = _diff_inputs(case, seed)
    e = DepthLossEngine(case["W"], case["H"], case["D"], case["S"], store_paths=case["store"])
    torch.cuda.synchronize()
    return dict(kind="diff", e=e, K=K, ref=ref, srcs=srcs.requires_grad_(case["train"]),
                xi=xi.requires_grad_(case["train"]), rho_gt=rho_gt, R0=R0, t0=t0, train=case["train"])


def _run_diff(st):
    if not st["train"]:
        return st["e"].forward(st["ref"], st["srcs"], st["K"], st["R0"], st["t0"], st["rho_gt"])
    st["srcs"].grad = st["xi"].grad = None
    loss = depth_loss(st["srcs"], st["xi"], st["e"], st["ref"], st["K"], st["R0"], st["t0"], st["rho_gt"])
    total = loss.float()   # the sum with a program's other losses, in the type of its parameters
    total.backward()
    return total.detach(), st["srcs"].grad, st["xi"].grad


def prepare(case, seed):
    return {"map": _prepare_map, "stage": _prepare_stage, "batch": _prepare_batch, "diff": _prepare_diff}[case["kind"]](case, seed)


def run(state):
    return {"map": _run_map, "stage": _run_stage, "batch": _run_batch, "diff": _run_diff}[state["kind"]](state)


# ---- work -------------------------------------------------------------------------------------

def _map_work(W, H, D, S, paths, fused):
    """Frames in, depth (and variance) out; 144 operations per voxel and source for the nine warps, bilinear
    samples and differences, and 9 per voxel and path for the recurrence, the sum and the minimum."""
    N = W * H
    return N * (1 + S) + (8 if fused else 4) * N, N * D * (144 * S + 9 * paths)


def work(case):
    S = case["S"]
    if case["kind"] == "map":
        b, f = _map_work(case["W"], case["H"], case["D"], S, case["paths"], case["fuse"] != "none")
    elif case["kind"] == "batch":
        each = [_map_work(W, H, D, S, case["paths"], True) for W, H, D in _batch_sizes(case)]
        b, f = sum(x for x, _ in each), sum(x for _, x in each)
    elif case["kind"] == "stage":
        N, V = case["W"] * case["H"], case["W"] * case["H"] * case["D"]
        # float images in, the two volumes, index, depths and table, four state maps in and out
        b, f = 4 * N * (1 + S) + 8 * V + 16 * N + 32 * N, V * (144 * S + 9 * case["paths"])
    else:
        N, V = case["W"] * case["H"], case["W"] * case["H"] * case["D"]
        # images and ground truth in; the gradients (or the inverse-depth map) out
        b, f = 4 * N * (2 + S) + (4 * N * S if case["train"] else 4 * N), V * (144 * S + 9 * 8 + 10)
        if case["train"]:
            f += V * (2 * 144 * S + 9 * 8 + 10)
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits ----------------------------------------------------------------------

def _sample(img, x, y, z, t, rho):
    """img (H, W) at the warp of the homogeneous points (x, y, z) + t * rho; NaN outside the image."""
    H, W = img.shape
    w = z + t[2] * rho
    u, v = (x + t[0] * rho) / w, (y + t[1] * rho) / w
    ok = (w >= 0) & (u >= 0) & (u <= W - 1) & (v >= 0) & (v <= H - 1)
    u, v = torch.where(ok, u, 0.0), torch.where(ok, v, 0.0)
    i, j = u.detach().floor(), v.detach().floor()
    a, b = u - i, v - j
    i, j = i.long(), j.long()
    pad = torch.nn.functional.pad(img, (0, 1, 0, 1)).reshape(-1)
    at = lambda di, dj: pad[(j + dj) * (W + 1) + i + di]  # noqa: E731
    top, bot = torch.lerp(at(0, 0), at(1, 0), a), torch.lerp(at(0, 1), at(1, 1), a)
    return torch.lerp(top, bot, b), ok


def _grid(H, W, halo):
    v, u = torch.meshgrid(torch.arange(-halo, H + halo, dtype=torch.float64, device="cuda"),
                          torch.arange(-halo, W + halo, dtype=torch.float64, device="cuda"), indexing="ij")
    return u, v


#: (du, dv) of the warped neighbour and of the reference pixel that it is compared with
_PATCH = [((0, 0), (0, 0)), ((0, -1), (0, -1)), ((0, 1), (0, 1)), ((-1, 0), (-1, 0)), ((1, 0), (1, 0)),
          ((-1, -1), (-1, -1)), ((1, 1), (1, 1)), ((-1, 1), (-1, 1)), ((1, -1), (1, -1))]
#: the reference's samples: the rows above and below swapped, the fifth and ninth from a corrupted warp
_QUIRKS = [((0, 0), (0, 0)), ((0, -1), (0, 1)), ((0, 1), (0, -1)), ((-1, 0), (-1, 0)), (4, (1, 0)),
           ((-1, -1), (-1, -1)), ((1, 1), (1, 1)), ((-1, 1), (-1, 1)), (8, (1, -1))]


def _cost(ref, srcs, warps, rhos, mode):
    """The cost volume (H, W, D) in float64: the mean over the measuring sources of the nine absolute
    differences' mean, -1 where no source measures.  warps: per source (point (3, H+2, W+2) of the halo grid, t
    (3), r (9))."""
    H, W = ref.shape
    rp = torch.nn.functional.pad(ref, (1, 1, 1, 1))
    total, count = [], []
    cut = lambda t, du, dv: t[1 + dv:1 + dv + H, 1 + du:1 + du + W]  # noqa: E731
    for rho in rhos:
        acc, cnt = torch.zeros_like(ref), torch.zeros_like(ref)
        for img, (P, t, r) in zip(srcs, warps):
            s, ok = _sample(img, P[0], P[1], P[2], t, rho)
            term, good = torch.zeros_like(ref), torch.ones_like(ref, dtype=torch.bool)
            for at, (du, dv) in _QUIRKS if mode == "reference" else _PATCH:
                if isinstance(at, tuple):
                    val, o = cut(s, *at), cut(ok, *at)
                else:   # the neighbour's point built from the centre's x alone (calc_cost.cu:49-51, 69-71)
                    xc = cut(P[0], 0, 0)
                    q = [xc + r[0], xc + r[3], xc + r[6]]
                    if at == 8:
                        q = [q[0] - r[1], q[0] - r[4], q[0] - r[7]]
                    val, o = _sample(img, q[0], q[1], q[2], t, rho)
                term = term + (cut(rp, du, dv) - val).abs()
                good = good & o
            acc = acc + torch.where(good, term / 9, 0.0)
            cnt = cnt + good
        total.append(torch.where(cnt > 0, acc / cnt.clamp(min=1), -1.0))
    return torch.stack(total, -1)


_DIRS = [(1, 0), (-1, 0), (0, 1), (0, -1), (1, 1), (-1, -1), (-1, 1), (1, -1)]


def _paths(C, bad, ref, count, p1, p2, tau, q1, q2):
    """The sum over `count` SGM paths of the volume C (H, W, D), whose pixels `bad` cost 0 (what
    the sum is at such pixels is left to the caller)."""
    H, W, D = C.shape
    C = torch.where(bad[..., None], 0.0, C)
    inf = torch.full((1, 1), math.inf, dtype=C.dtype, device=C.device)
    out = None
    for dx, dy in _DIRS[:count]:
        T = dy == 0   # rows are the steps, or columns for the horizontal paths
        c, g = (C.transpose(0, 1), ref.T) if T else (C, ref)
        n, sh = c.shape[0], 0 if T else dx
        order = range(n) if (dx if T else dy) > 0 else range(n - 1, -1, -1)
        prev, rows = None, [None] * n
        for k in order:
            if prev is None:
                L = c[k]
            else:
                Lp, gp = prev
                if sh:   # the predecessor's column is one to the side; the image's edge starts a path
                    Lp, gp = torch.roll(Lp, sh, 0), torch.roll(gp, sh, 0)
                pen = ((g[k] - gp).abs() < tau)[:, None]
                P1, P2 = torch.where(pen, p1 * q1, p1), torch.where(pen, p2 * q2, p2)
                m, _ = Lp.min(-1, keepdim=True)
                edge = inf.expand(Lp.shape[0], 1)
                left, right = torch.cat([edge, Lp[:, :-1]], 1), torch.cat([Lp[:, 1:], edge], 1)
                nb = torch.where(left <= right, left, right) + P1
                far = (m + P2).expand_as(Lp)
                best = torch.where((Lp <= nb) & (Lp <= far), Lp, torch.where(nb <= far, nb, far))
                L = c[k] + best - m
                if sh:
                    first = 0 if sh > 0 else -1
                    keep = torch.ones(L.shape[0], 1, dtype=torch.bool, device=L.device)
                    keep[first] = False
                    L = torch.where(keep, L, c[k])
            rows[k] = L
            prev = (L, g[k])
        S = torch.stack(rows)
        S = S.transpose(0, 1) if T else S
        out = S if out is None else out + S
    return out


def _exact_stage(case, seed):
    sc, _, ref, srcs, homs, _ = _stage_inputs(case, seed)
    H, W, D = case["H"], case["W"], case["D"]
    u, v = _grid(H, W, 1)
    warps = []
    for h in homs.astype(np.float64):
        P = [h[3 * i] * u + h[3 * i + 1] * v + h[3 * i + 2] for i in range(3)]
        warps.append((P, h[9:], h[:9]))
    rho0, drho = (float(np.float32(x)) for x in _planes(D))
    cost = _cost(ref.double(), srcs.double(), warps, [rho0 + d * drho for d in range(D)], case["mode"])
    bad = (cost < 0).any(-1)
    sgm = _paths(cost, bad, ref.double(), case["paths"], 8.0, 24.0, 4.0, 2.0, 3.0)
    sgm = torch.where(bad[..., None], 0.0, sgm)   # an unmeasured plane makes the pixel's sums 0
    # the choice of a plane, and the fusion that follows it, jump with the last bit of a sum
    return dict(cost=cost, sgm=sgm, depth=None, index=None, fused=None, table=None, state=None)


def _exact_diff(case, seed):
    K, ref, srcs, rho_gt, R0, t0, xi = _diff_inputs(case, seed)
    H, W, D = case["H"], case["W"], case["D"]
    ref, rho_gt = ref.double(), rho_gt.double()
    srcs = srcs.double().requires_grad_(case["train"])
    step = torch.zeros(case["S"], 6, dtype=torch.float64, device="cuda", requires_grad=case["train"])
    u, v = _grid(H, W, 1)
    Kd = torch.tensor(K, dtype=torch.float64, device="cuda")
    rays = torch.stack([(u - K[0, 2]) / K[0, 0], (v - K[1, 2]) / K[1, 1], torch.ones_like(u)])
    warps = []
    for s in range(case["S"]):
        R, t = R0[s], t0[s]
        if case["train"]:
            x = xi[s].double().cpu().numpy()
            E = _rotation(x[:3], np.linalg.norm(x[:3]))
            R, t = E @ R, E @ t + x[3:]
        R, t = (torch.tensor(y, dtype=torch.float64, device="cuda") for y in (R, t))
        p = torch.einsum("ij,jhw->ihw", R, rays)
        w = step[s, :3, None, None].expand(3, H + 2, W + 2)
        # exp([omega]) P + upsilon, to the first order
        p = torch.einsum("ij,jhw->ihw", Kd, p + torch.cross(w, p, dim=0))
        warps.append((p, Kd @ (t + torch.linalg.cross(step[s, :3], t) + step[s, 3:]), None))
    rho0, drho = float(np.float32(0.1)), float(np.float32(1.9 / (D - 1)))
    rhos = [rho0 + d * drho for d in range(D)]
    with torch.set_grad_enabled(case["train"]):
        C = _cost(ref, srcs, warps, rhos, "corrected")
        bad = (C < 0).any(-1)
        tau = float(np.float32(3.5 / 255))
        S = _paths(C, bad, ref, 8, float(np.float32(0.003)), float(np.float32(0.01)), tau, 2.0, 3.0)
        rho = torch.tensor(rhos, dtype=torch.float64, device="cuda")
        rho_hat = (torch.softmax(-S / float(np.float32(0.05)), -1) * rho).sum(-1)
        use = ~bad & (rho_gt > 0)
        loss = torch.where(use, (rho_hat - rho_gt).abs(), 0.0).sum() / use.sum()
        if not case["train"]:
            return loss, torch.where(use, rho_hat, 0.0)
        loss.backward()
    return loss.detach(), srcs.grad, step.grad


def exact(case, seed):
    if case["kind"] == "stage":
        return _exact_stage(case, seed)
    if case["kind"] == "diff" and case["W"] * case["H"] * case["D"] <= 640 * 480 * 64:   # memory of the saved states
        return _exact_diff(case, seed)
    return None   # a map is its choice of planes, which jumps with the last bit of a sum
