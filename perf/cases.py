"""Performance cases of the RGB-D registration path: what its callers run, over the
sizes they run it at.

A case names one public entry point (a stage of the C ABI, a one-shot alignment, a
reusable plan, the streaming tracker or the adjoint) and its sizes.  ``prepare`` makes
the inputs on the GPU from a seed, ``run`` is one pass through the entry point, ``work``
the bytes that pass cannot do without, and ``exact`` what it computes in 64 bits, in
plain torch.

The clouds are samples of a furnished room (walls, boxes, cylinders) with 3 mm position
noise and a smooth colour field; frames are ray-cast views of a procedural scene with
sensor noise and missing pixels.
"""
from __future__ import annotations

import ctypes as C
import math
import weakref
from types import SimpleNamespace

import numpy as np
import torch

from cuda_3d_gb300 import native as N
from cuda_3d_gb300 import synth

LAMBDA = float(np.float32(0.968))  # weight of the geometric term, everywhere
# voxel, iterations, max_corr, normal radius, gradient radius of the coarse-to-fine schedule
SCALES = [(0.04, 50, 0.06, 0.08, 0.08), (0.02, 30, 0.03, 0.04, 0.04), (0.01, 14, 0.015, 0.02, 0.02)]
# the frame-to-frame registration of the tracker (the last value: at most 30 neighbours)
TRACK_SCALE = (0.01, 30, 0.03, 0.02, 0.02, 30)
DEPTH_SCALE, T_MIN, T_MAX = 0.001, 0.2, 10.0


# --------------------------------------------------------------------------- #
# the cases
# --------------------------------------------------------------------------- #
def listed():
    return [
        # the smallest cloud of the batch workload, downsampled once: a latency-bound call
        dict(name="voxel_20k", kind="voxel", n=20_011, voxel=0.04, per_voxel=4.0),
        # a full fragment at the finest scale
        dict(name="voxel_300k", kind="voxel", n=300_000, voxel=0.01, per_voxel=1.5),
        # one camera frame to a cloud: the 5x5 filter of the tracker
        dict(name="frame_640_fixed", kind="frame", w=640, h=480, filter="fixed", radius=2),
        # the larger camera mode with the reference demo's adaptive filter
        dict(name="frame_1280_adaptive", kind="frame", w=1280, h=720, filter="adaptive", radius=0),
        # normals of a downsampled frame, neighbours capped as the tracker does
        dict(name="normals_206k", kind="normals", n=206_443, voxel=0.01, radius=0.02, max_nn=30),
        # correspondences between two downsampled fragments of different size
        dict(name="nn_250k", kind="nn", n_query=250_000, n_ref=200_003, voxel=0.01, radius=0.03),
        # cleaning of a frame before it joins the reconstruction (the reference demo's settings)
        dict(name="outlier_180k", kind="outlier", n=180_000, voxel=0.008, radius=0.01, min_neighbors=4),
        # the reference's own call: two downsampled fragments aligned in one shot
        dict(name="align_64k", kind="align", n=64_365, voxel=0.02, max_corr=0.05, grad_radius=0.04, max_iter=100),
        # the gradient through five unrolled steps
        dict(name="vjp_100k", kind="vjp", n=100_000, voxel=0.02, max_corr=0.05, steps=5),
        # a tracked camera: two frames pushed, each registered onto the one before
        dict(name="track_640", kind="track", w=640, h=480, rot_deg=2.0, trans=0.03),
        # one fragment pair, coarse to fine, on a plan that the caller keeps
        dict(name="pair_250k", kind="register", pairs=1, n_min=250_000, n_max=250_000),
        # the batch workload: 64 pairs of uneven size in one plan
        dict(name="batch_64", kind="register", pairs=64, n_min=20_000, n_max=300_000),
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["voxel", "frame", "normals", "gradient", "nn", "outlier", "align", "vjp", "track", "register"])
    n = int(log(5_000, 300_000))
    voxel = round(log(0.008, 0.04), 4)
    if kind == "voxel":
        return dict(kind=kind, n=n, voxel=voxel, per_voxel=round(log(1.2, 8.0), 2))
    if kind == "frame":
        w = int(log(160, 1280))
        return dict(kind=kind, w=w, h=int(w * rng.uniform(0.5, 0.8)), filter=rng.choice(["none", "fixed", "adaptive"]),
                    radius=rng.randint(1, 4))
    if kind == "normals":
        return dict(kind=kind, n=n, voxel=voxel, radius=round(voxel * rng.uniform(1.8, 3.0), 4),
                    max_nn=rng.choice([0, 16, 30]))
    if kind == "gradient":
        return dict(kind=kind, n=n, voxel=voxel, radius=round(voxel * rng.uniform(1.8, 3.0), 4))
    if kind == "nn":
        return dict(kind=kind, n_query=n, n_ref=int(log(5_000, 300_000)), voxel=voxel,
                    radius=round(voxel * rng.uniform(1.5, 3.0), 4))
    if kind == "outlier":
        return dict(kind=kind, n=n, voxel=voxel, radius=round(voxel * rng.uniform(1.25, 2.5), 4),
                    min_neighbors=rng.randint(2, 8))
    if kind == "align":
        return dict(kind=kind, n=n, voxel=voxel, max_corr=round(2.5 * voxel, 4), grad_radius=round(2.0 * voxel, 4),
                    max_iter=rng.randint(10, 100))
    if kind == "vjp":
        return dict(kind=kind, n=n, voxel=voxel, max_corr=round(2.5 * voxel, 4), steps=rng.randint(2, 6))
    if kind == "track":
        w = int(log(320, 1280))
        return dict(kind=kind, w=w, h=int(w * rng.uniform(0.5, 0.8)), rot_deg=round(rng.uniform(0.5, 2.0), 2),
                    trans=round(rng.uniform(0.01, 0.03), 3))
    n_min = int(log(5_000, 100_000))
    return dict(kind=kind, pairs=int(log(1, 32)), n_min=n_min, n_max=int(n_min * rng.uniform(1.0, 3.0)))


def work(case):
    """Bytes of one pass: each input read once (16 bytes per position, colour, normal or
    gradient of a cloud), each output written once.  The path is neighbour searches and
    reductions, bound by memory and latency; its arithmetic is not counted."""
    k = case["kind"]
    if k == "voxel":
        b = case["n"] * 32 + case["n"] / case["per_voxel"] * 32
    elif k == "frame":
        b = case["w"] * case["h"] * (2 + 3 + 0.95 * 32)
    elif k == "normals":
        b = case["n"] * (16 + 16)
    elif k == "gradient":
        b = case["n"] * (16 + 16 + 16)
    elif k == "nn":
        b = (case["n_query"] + case["n_ref"]) * 16 + case["n_query"] * 4
    elif k == "outlier":
        b = case["n"] * (32 + 32)
    elif k == "align":
        b = case["n"] * (16 + 32)
    elif k == "vjp":
        b = case["n"] * (16 + 48 + 24)
    elif k == "track":
        b = 2 * case["w"] * case["h"] * (2 + 3)
    else:
        lo, hi = case["n_min"], case["n_max"]
        mean = (hi - lo) / math.log(hi / lo) if hi > lo else lo
        b = case["pairs"] * 2 * mean * 32
    return {"bytes": float(b), "flops": 0.0}


# --------------------------------------------------------------------------- #
# inputs
# --------------------------------------------------------------------------- #
class Gen:
    """seeded draws on the GPU"""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed) & 0x7FFFFFFF)

    def rand(self, *shape, lo=0.0, hi=1.0):
        return lo + (hi - lo) * torch.rand(*shape, generator=self.g, device="cuda", dtype=torch.float64)

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda", dtype=torch.float64)


def surfaces():
    """the room's faces as (origin, u, v) triples (n x 3 x 3, float64, on the GPU), the
    cylinders as 16-sided prisms"""
    W, D, H = synth.ROOM
    scene = synth.room_scene()
    f = [((0, 0, 0), (W, 0, 0), (0, D, 0)), ((0, 0, H), (W, 0, 0), (0, D, 0)), ((0, 0, 0), (W, 0, 0), (0, 0, H)),
         ((0, D, 0), (W, 0, 0), (0, 0, H)), ((0, 0, 0), (0, D, 0), (0, 0, H)), ((W, 0, 0), (0, D, 0), (0, 0, H))]
    for lo, hi in scene.boxes:
        s = hi - lo
        f += [((lo[0], lo[1], hi[2]), (s[0], 0, 0), (0, s[1], 0)), (tuple(lo), (s[0], 0, 0), (0, 0, s[2])),
              ((lo[0], hi[1], lo[2]), (s[0], 0, 0), (0, 0, s[2])), (tuple(lo), (0, s[1], 0), (0, 0, s[2])),
              ((hi[0], lo[1], lo[2]), (0, s[1], 0), (0, 0, s[2]))]
    for cx, cy, r, h in scene.cylinders:
        a = [2 * math.pi * i / 16 for i in range(17)]
        p = [(cx + r * math.cos(t), cy + r * math.sin(t)) for t in a]
        f += [((x, y, 0), (x2 - x, y2 - y, 0), (0, 0, h)) for (x, y), (x2, y2) in zip(p, p[1:])]
    return torch.tensor(np.array(f, np.float64), device="cuda")


def sample_room(gen, n, scale=1.0, noise=0.003):
    """n points of the room, uniform by area and with position noise, and their surface
    normals; scale enlarges the room"""
    f = surfaces() * scale
    area = torch.linalg.cross(f[:, 1], f[:, 2])
    size = area.norm(dim=1)
    edge = torch.cumsum(size, 0) / size.sum()
    k = torch.searchsorted(edge, gen.rand(n)).clamp(max=len(f) - 1)
    p = f[k, 0] + gen.rand(n, 1) * f[k, 1] + gen.rand(n, 1) * f[k, 2]
    nrm = (area / size[:, None])[k]
    nrm = torch.where(nrm[:, 2:] > 0, -nrm, nrm)
    return p + noise * gen.normal(n, 3), nrm


ROOM_AREA = 118.0  # of the faces above, about


class Colors:
    """a smooth colour field: three octaves of sinusoids"""

    def __init__(self, gen):
        self.k = torch.cat([gen.normal(4, 3) * s for s in (2.0, 4.0, 8.0)])
        self.a = torch.cat([gen.rand(4, 3, lo=0.3) * s for s in (0.10, 0.05, 0.025)])
        self.p = gen.rand(12, 3, hi=2 * math.pi)

    def __call__(self, x):
        out = torch.full_like(x, 0.5)
        for k, a, p in zip(self.k, self.a, self.p):
            out += a * torch.sin((x @ k)[:, None] + p)
        return out.clamp(0, 1)

    def intensity_gradient(self, x):
        w = torch.tensor([0.2126, 0.7152, 0.0722], dtype=torch.float64, device="cuda")
        out = torch.zeros_like(x)
        for k, a, p in zip(self.k, self.a, self.p):
            out += ((w * a) * torch.cos((x @ k)[:, None] + p)).sum(1, keepdim=True) * k
        return out


def thinned(gen, n, voxel):
    """about one room point per voxel, as a downsampled cloud holds them: n points, and
    their normals"""
    layers = 1.0 + 0.006 / voxel  # the noise spreads a face over more than one layer of voxels
    p, nrm = sample_room(gen, 4 * n, scale=math.sqrt(1.1 * n * voxel * voxel / layers / ROOM_AREA))
    c = torch.floor(p / voxel).to(torch.int64) + (1 << 19)
    _, inv = torch.unique((c[:, 0] << 40) | (c[:, 1] << 20) | c[:, 2], return_inverse=True)
    first = torch.full((int(inv.max()) + 1,), len(p), dtype=torch.int64, device="cuda")
    first.scatter_reduce_(0, inv, torch.arange(len(p), device="cuda"), "amin")
    keep = first.sort().values[:n]
    return p[keep], nrm[keep]


def rigid(gen, angle_deg, trans, center):
    """a rotation by angle_deg about a random axis through center, and a shift of length
    trans (4 x 4, float64)"""
    axis, d = gen.normal(3), gen.normal(3)
    R = torch.matrix_exp(hat(axis / axis.norm() * math.radians(angle_deg)))
    T = torch.eye(4, dtype=torch.float64, device="cuda")
    T[:3, :3] = R
    T[:3, 3] = center + d / d.norm() * trans - R @ center
    return T


def moved(T, p):
    return p @ T[:3, :3].T + T[:3, 3]


def thinned_pair(gen, case):
    """two downsampled views of a room that share 70 % of it, a small motion apart: the
    source's points and colours, the target's, and the target's normals and gradients"""
    n, out = case["n"], []
    for part in (0, 1):
        p, nrm = thinned(gen, int(n / 0.7), case["voxel"])
        order = p[:, 0].argsort()
        keep = (order[:n] if part == 0 else order[-n:]).sort().values
        out.append((p[keep], nrm[keep]))
    (s, _), (t, nrm) = out
    col = Colors(gen)
    T = rigid(gen, 0.3, 0.4 * case["max_corr"], t.mean(0))
    a = SimpleNamespace(sx=moved(torch.linalg.inv(T), s).float(), sc=col(s).float(), tx=t.float(), tc=col(t).float(),
                        tn=nrm.float(), tg=col.intensity_gradient(t).float())
    return a


def room_pairs(gen, case):
    """fragment pairs: sizes log-uniform, overlap 40-90 %, rotation 0-15 deg, translation
    0-15 cm per pair; a lone pair has overlap 60 %, 10 deg and 10 cm"""
    P = case["pairs"]
    u = gen.rand(P, 5).cpu().numpy()
    col, W, D = Colors(gen), synth.ROOM[0], synth.ROOM[1]
    center = torch.tensor([v / 2 for v in synth.ROOM], dtype=torch.float64, device="cuda")
    out = []
    for k in range(P):
        n = int(math.exp(math.log(case["n_min"]) + u[k, 0] * math.log(case["n_max"] / case["n_min"])))
        overlap, rot, trans = (0.6, 10.0, 0.1) if P == 1 else (0.4 + 0.5 * u[k, 1], 15 * u[k, 2], 0.15 * u[k, 3])
        a = 2 * math.pi * u[k, 4]
        d = torch.tensor([math.cos(a), math.sin(a)], dtype=torch.float64, device="cuda")
        half = 0.5 * (abs(math.cos(a)) * W + abs(math.sin(a)) * D)
        view = 2 * half / (2 - overlap)
        clouds = []
        for lo in (half - view, -half):  # target, source
            p, _ = sample_room(gen, int(1.35 * n * 2 * half / view))
            s = (p[:, :2] - center[:2]) @ d
            clouds.append(p[(s >= lo) & (s <= lo + view)][:n])
        t, s = clouds
        T = rigid(gen, rot, trans, center)
        out.append((moved(torch.linalg.inv(T), s).float(), col(s).float(), t.float(), col(t).float()))
    return out


def camera(case):
    w, h = case["w"], case["h"]
    f = 525.0 * w / 640
    return synth.Camera(w, h, f, f, (w - 1) / 2, (h - 1) / 2)


def frames(case, seed, poses):
    """rendered views of the frame scene from the given camera poses: (depth, BGR) on the host"""
    return [synth.render_rgbd_torch(synth.frame_scene(), P, int(seed) * 16 + k, camera(case))
            for k, P in enumerate(poses)]


def inputs(case, seed):
    """the case's inputs as float32 tensors on the GPU (frames: host arrays)"""
    gen, k = Gen(seed), case["kind"]
    if k == "voxel":
        p, _ = sample_room(gen, case["n"], scale=math.sqrt(case["n"] / case["per_voxel"] * case["voxel"] ** 2
                                                           / ROOM_AREA))
        return SimpleNamespace(x=p.float(), c=Colors(gen)(p).float())
    if k == "frame":
        return SimpleNamespace(frames=frames(case, seed, [np.eye(4)]))
    if k in ("normals", "gradient", "outlier"):
        p, nrm = thinned(gen, case["n"], case["voxel"])
        return SimpleNamespace(x=p.float(), c=Colors(gen)(p).float(), nrm=nrm.float())
    if k == "nn":
        n = max(case["n_query"], case["n_ref"])
        q, r = (thinned(gen, n, case["voxel"])[0] for _ in range(2))
        q, r = q[:case["n_query"]], r[:case["n_ref"]]
        return SimpleNamespace(q=q.float(), r=r.float())
    if k in ("align", "vjp"):
        return thinned_pair(gen, case)
    if k == "track":
        rng = np.random.default_rng(int(seed) & 0x7FFFFFFF)
        d = rng.normal(size=3)
        T = synth.make_T(synth.random_rotation(rng, case["rot_deg"]), d / np.linalg.norm(d) * case["trans"])
        return SimpleNamespace(frames=frames(case, seed, [np.eye(4), T]))
    return SimpleNamespace(pairs=room_pairs(gen, case))


# --------------------------------------------------------------------------- #
# what a caller keeps, and one pass
# --------------------------------------------------------------------------- #
_context = None


def context():
    """one library context, shared by the states that are alive"""
    global _context
    ctx = _context() if _context else None
    if ctx is None:
        ctx = N.Context(torch.cuda.current_device())
        _context = weakref.ref(ctx)
    return ctx


class _Memory:
    """device memory of a cloud, which lives as long as a tensor of it does"""

    def __init__(self, cloud, ptr, shape, typestr):
        self.cloud = cloud
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def views(cloud, n):
    """a cloud's positions, colours, normals and count as tensors (no copy)"""
    pos, col, nrm, _, cnt = cloud.device_views()
    v = [torch.as_tensor(_Memory(cloud, p, (n, 4), "<f4"), device="cuda") if p else None for p in (pos, col, nrm)]
    return v + [torch.as_tensor(_Memory(cloud, cnt, (1,), "<i4"), device="cuda")]


def clouds(ctx, sets):
    """clouds of (positions, colours) tensors"""
    out = [ctx.cloud(max(len(x), 1)) for x, _ in sets]
    torch.cuda.synchronize()
    N.upload_many(ctx, out, [x.data_ptr() for x, _ in sets], [c.data_ptr() for _, c in sets],
                  [len(x) for x, _ in sets])
    ctx.sync()
    return out


def empty_cloud(ctx, n):
    """a cloud of capacity n whose unused tail is zero, and its views"""
    c = ctx.cloud(n)
    v = views(c, n)
    for t in v:
        if t is not None:
            t.zero_()
    torch.cuda.synchronize()
    return c, v


FILTERS = {"none": N.FILTER_NONE, "fixed": N.FILTER_FIXED, "adaptive": N.FILTER_ADAPTIVE}


def prepare(case, seed):
    a, k, ctx = inputs(case, seed), case["kind"], context()
    s = SimpleNamespace(case=case, kind=k, ctx=ctx)
    if k in ("voxel", "outlier"):
        s.cloud, = clouds(ctx, [(a.x, a.c)])
        s.out, s.view = empty_cloud(ctx, len(a.x))
    elif k == "frame":
        depth, bgr = a.frames[0]
        s.depth = torch.from_numpy(depth.view(np.int16)).cuda()
        s.bgr = torch.from_numpy(bgr).cuda()
        s.out, s.view = empty_cloud(ctx, case["w"] * case["h"])
        cam = camera(case)
        s.intrin = N.Intrinsics(cam.fx, cam.fy, cam.cx, cam.cy)
        s.filter = N.Filter(FILTERS[case["filter"]], case["radius"], 3.0, 30.0)
    elif k in ("normals", "gradient"):
        s.cloud, = clouds(ctx, [(a.x, a.c)])
        if k == "gradient":
            ctx.check(ctx.L.gca3d_cloud_set_normals(ctx.h, s.cloud.h, a.nrm.data_ptr(), len(a.x)))
            ctx.sync()
        s.n = len(a.x)
    elif k == "nn":
        s.query, s.ref = clouds(ctx, [(a.q, torch.zeros_like(a.q)), (a.r, torch.zeros_like(a.r))])
        s.idx = torch.empty(len(a.q), dtype=torch.int32, device="cuda")
    elif k in ("align", "vjp"):
        s.src, s.tgt = clouds(ctx, [(a.sx, a.sc), (a.tx, a.tc)])
        ctx.check(ctx.L.gca3d_cloud_set_normals(ctx.h, s.tgt.h, a.tn.data_ptr(), len(a.tx)))
        if k == "align":
            s.params = N.icp_params([N.scale(0.0, case["max_iter"], case["max_corr"], 0.0, case["grad_radius"])],
                                    keep_target_normals=True)
        else:
            ctx.check(ctx.L.gca3d_cloud_set_gradients(ctx.h, s.tgt.h, a.tg.data_ptr(), len(a.tx)))
            s.dxyz, s.drgb = (torch.empty(len(a.sx), 3, device="cuda") for _ in range(2))
            s.seed = loss_seed(seed)
        ctx.sync()
    elif k == "track":
        s.frames = a.frames
        s.tracker = N.Tracker(ctx, N.tracker_params(camera(case), [N.scale(*TRACK_SCALE)], depth_scale=DEPTH_SCALE,
                                                    tmin=T_MIN, tmax=T_MAX, use_graph=True, constant_velocity=False))
        for f in (1, 0, 1):  # a tracker that is running: both of its per-frame graphs exist
            s.tracker.push(*s.frames[f])
    else:
        src = clouds(ctx, [p[:2] for p in a.pairs])
        tgt = clouds(ctx, [p[2:] for p in a.pairs])
        s.plan = N.IcpPlan(ctx, src, tgt, N.icp_params([N.scale(*x) for x in SCALES], update_map=N.UPDATE_SE3_EXP,
                                                       use_graph=True))
    torch.cuda.synchronize()
    return s


def registration(results):
    """the results of registrations: poses, statistics, and counts"""
    return {"T": np.stack([r["T"] for r in results]),
            "stats": np.array([[r["rmse_ref"], r["fitness"], r["inlier_rmse"]] for r in results]),
            "counts": np.array([[r["status"], r["iterations"], r["n_src"], r["n_tgt"]] for r in results])}


def run(s):
    case, k, ctx, L = s.case, s.kind, s.ctx, s.ctx.L
    if k == "voxel":
        ctx.check(L.gca3d_voxel_downsample(ctx.h, s.cloud.h, case["voxel"], s.out.h))
        return {"xyz": s.view[0][:, :3], "intensity": s.view[0][:, 3], "rgb": s.view[1][:, :3], "count": s.view[3]}
    if k == "frame":
        ctx.check(L.gca3d_frame_to_cloud(ctx.h, s.depth.data_ptr(), s.bgr.data_ptr(), case["w"], case["h"],
                                         C.byref(s.intrin), None, None, DEPTH_SCALE, T_MIN, T_MAX, C.byref(s.filter),
                                         s.out.h))
        return {"xyz": s.view[0][:, :3], "intensity": s.view[0][:, 3], "rgb": s.view[1][:, :3], "count": s.view[3]}
    if k == "normals":
        ctx.check(L.gca3d_estimate_normals(ctx.h, s.cloud.h, case["radius"], case["max_nn"]))
        return views(s.cloud, s.n)[2][:, :3]
    if k == "gradient":
        ctx.check(L.gca3d_color_gradient(ctx.h, s.cloud.h, case["radius"]))
        return torch.as_tensor(_Memory(s.cloud, s.cloud.device_views()[3], (s.n, 4), "<f4"), device="cuda")[:, :3]
    if k == "nn":
        ctx.check(L.gca3d_nn_search(ctx.h, s.query.h, s.ref.h, case["radius"], s.idx.data_ptr()))
        return s.idx
    if k == "outlier":
        ctx.check(L.gca3d_radius_outlier_removal(ctx.h, s.cloud.h, case["radius"], case["min_neighbors"], s.out.h))
        return {"xyz": s.view[0][:, :3], "rgb": s.view[1][:, :3], "count": s.view[3]}
    if k == "align":
        return registration([N.color_icp(ctx, s.src, s.tgt, s.params)])
    if k == "vjp":
        xi0, dT, dE = s.seed
        r = N.color_icp_vjp(ctx, s.src, s.tgt, xi0, K=case["steps"], max_corr=case["max_corr"], dT=dT, dE=dE,
                            n_src=len(s.dxyz), out={"dxyz": SimpleNamespace(ptr=s.dxyz.data_ptr()),
                                                  "drgb": SimpleNamespace(ptr=s.drgb.data_ptr())})
        return {"T": r["T"], "E": r["E"], "dxi0": r["dxi0"], "dxyz": s.dxyz, "drgb": s.drgb}
    if k == "track":
        return registration([s.tracker.push(*f)[0] for f in s.frames])
    return registration(s.plan.execute())


# --------------------------------------------------------------------------- #
# the same in 64 bits
# --------------------------------------------------------------------------- #
def loss_seed(seed):
    """start of the unrolled steps and cotangents of their pose and objective"""
    rng = np.random.default_rng(int(seed) & 0x7FFFFFFF)
    dT = rng.normal(size=(4, 4))
    dT[3] = 0.0
    return rng.normal(size=6) * 1e-3, dT, 0.3


def hat(w):
    """the cross-product matrix of w, or the 4 x 4 twist of (w, v)"""
    o = torch.zeros((), dtype=w.dtype, device=w.device)
    rows = [[o, -w[2], w[1]], [w[2], o, -w[0]], [-w[1], w[0], o]]
    if len(w) == 6:
        rows = [r + [w[3 + i]] for i, r in enumerate(rows)] + [[o, o, o, o]]
    return torch.stack([torch.stack(r) for r in rows])


def euler(x):
    """Rz Ry Rx with the translation x[3:]"""
    R = torch.eye(3, dtype=x.dtype, device=x.device)
    for a in (2, 1, 0):
        e = torch.zeros(3, dtype=x.dtype, device=x.device)
        e[a] = 1.0
        R = R @ torch.matrix_exp(hat(e * x[a]))
    T = torch.eye(4, dtype=x.dtype, device=x.device)
    T[:3, :3], T[:3, 3] = R, x[3:]
    return T


def dist2(p, q):
    """squared distances in the points' own precision, each operation rounded by itself"""
    d = p - q
    return d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]


def neighbours(q, r, radius):
    """all (query, reference) index pairs closer than radius (float32, as the radius is given)"""
    radius = float(np.float32(radius))
    rr = torch.tensor(radius, device=q.device) ** 2
    mn, cell = r.min(0).values.double(), 1.0001 * radius
    rc = torch.floor((r.double() - mn) / cell).to(torch.int64) + 2
    dim = rc.max(0).values + 3
    qc = torch.floor((q.double() - mn) / cell).to(torch.int64) + 2
    ok = ((qc >= 1) & (qc <= dim - 2)).all(1).nonzero()[:, 0]
    key, order = ((rc[:, 0] * dim[1] + rc[:, 1]) * dim[2] + rc[:, 2]).sort()
    qi, ri = [], []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            k = ((qc[ok, 0] + dx) * dim[1] + qc[ok, 1] + dy) * dim[2] + qc[ok, 2]
            a, b = torch.searchsorted(key, k - 1), torch.searchsorted(key, k + 1, right=True)
            m = b - a
            i = torch.repeat_interleave(ok, m)
            at = torch.arange(len(i), device=q.device) - torch.repeat_interleave(m.cumsum(0) - m, m)
            j = order[torch.repeat_interleave(a, m) + at]
            near = dist2(q[i], r[j]) < rr.to(q.dtype)
            qi.append(i[near])
            ri.append(j[near])
    return torch.cat(qi), torch.cat(ri)


def nearest(q, r, radius):
    """the nearest reference point within radius of every query point, -1 where there is none"""
    i, j = neighbours(q, r, radius)
    d = dist2(q[i], r[j])
    best = torch.full((len(q),), math.inf, dtype=d.dtype, device=q.device).scatter_reduce_(0, i, d, "amin")
    hit = d == best[i]
    out = torch.full((len(q),), len(r), dtype=torch.int64, device=q.device)
    out.scatter_reduce_(0, i[hit], j[hit], "amin")
    return torch.where(out < len(r), out, -1)


def intensity(c):
    return c.double() @ torch.tensor([0.2126, 0.7152, 0.0722], dtype=torch.float64, device=c.device)


def sums(index, values, n):
    return torch.zeros((n,) + values.shape[1:], dtype=torch.float64, device=values.device).index_add_(0, index, values)


def voxels(x, c, voxel):
    """centroids and mean colours of the occupied voxels in (x, y, z) order"""
    k = torch.floor((x - x.min(0).values) / torch.tensor(voxel, dtype=torch.float32, device=x.device)).to(torch.int64)
    _, inv, cnt = torch.unique((k[:, 0] << 42) | (k[:, 1] << 21) | k[:, 2], return_inverse=True, return_counts=True)
    m = sums(inv, torch.cat([x.double(), c.double()], 1), len(cnt)) / cnt[:, None]
    return m[:, :3], m[:, 3:]


def capped(i, d, n, most):
    """the pairs that stay when each of n queries keeps its `most` nearest"""
    order = torch.argsort(d)
    order = order[torch.argsort(i[order], stable=True)]
    first = torch.searchsorted(i[order].contiguous(), torch.arange(n, device=i.device))
    rank = torch.arange(len(i), device=i.device) - first[i[order]]
    return order[rank < most]


def normals64(x, radius, max_nn=0):
    i, j = neighbours(x.float(), x.float(), radius)
    if max_nn:
        keep = capped(i, dist2(x.float()[i], x.float()[j]), len(x), max_nn)
        i, j = i[keep], j[keep]
    d = x.double()[j] - x.double()[i]
    cnt = torch.bincount(i, minlength=len(x)).double()[:, None]
    mean = sums(i, d, len(x)) / cnt
    cov = sums(i, (d[:, :, None] * d[:, None, :]).reshape(-1, 9), len(x)) / cnt
    cov = cov.reshape(-1, 3, 3) - mean[:, :, None] * mean[:, None, :]
    n = torch.linalg.eigh(cov.cpu())[1][:, :, 0].to(x.device)
    n = torch.where(n[:, 2:] > 0, -n, n)
    return torch.where(cnt >= 3, n, torch.zeros_like(n))


def gradients64(x, inten, n, radius):
    i, j = neighbours(x.float(), x.float(), radius)
    d = x.double()[j] - x.double()[i]
    n = n.double()
    v = d - (d * n[i]).sum(1, keepdim=True) * n[i]
    A = sums(i, (v[:, :, None] * v[:, None, :]).reshape(-1, 9), len(x)).reshape(-1, 3, 3)
    b = sums(i, v * (inten[j] - inten[i])[:, None], len(x))
    knn = torch.bincount(i, minlength=len(x)).double()
    w = (knn - 1)[:, None, None] ** 2
    A = A + w * n[:, :, None] * n[:, None, :] + 1e-6 * torch.eye(3, dtype=torch.float64, device=x.device)
    g = torch.linalg.solve(A, b[:, :, None])[:, :, 0]
    return torch.where((knn >= 5)[:, None], g, torch.zeros_like(g))


def system(p, si, q, qi, n, g):
    """residuals (m x 2) and Jacobians (m x 2 x 6) of the colored-ICP objective"""
    lg, lc = math.sqrt(LAMBDA), math.sqrt(1.0 - LAMBDA)
    rg = ((p - q) * n).sum(1)
    t = g - (g * n).sum(1, keepdim=True) * n
    rc = qi + (g * (p - rg[:, None] * n - q)).sum(1) - si
    J = [w * torch.cat([torch.linalg.cross(p, u), u], 1) for w, u in ((lg, n), (lc, t))]
    return torch.stack([lg * rg, lc * rc], 1), torch.stack(J, 1)


def evaluate(T, s, si, t, ti, n, g, max_corr):
    """one evaluation at pose T: H, b, the objective, correspondences and their squared distances"""
    p = moved(T, s)
    # correspondences are defined on float32 points: they are piecewise constant in the pose
    nn = nearest(moved(T.detach().float().double(), s.detach()).float(), t.float(), max_corr)
    m, j = nn >= 0, nn[nn >= 0]
    r, J = system(p[m], si[m], t[j], ti[j], n[j], g[j])
    H, b = torch.einsum("nki,nkj->ij", J, J), torch.einsum("nki,nk->i", J, r)
    return H, b, (r * r).sum(), len(j), dist2(p[m], t[j])


def icp64(s, si, t, ti, n, g, max_corr, max_iter, step, T):
    """Gauss-Newton steps until the reference's convergence test holds: pose and statistics"""
    stats = None
    for _ in range(max_iter):
        H, b, E, m, d2 = evaluate(T, s, si, t, ti, n, g, max_corr)
        U = step(-torch.linalg.solve(H, b))
        T = U @ T
        stats = [float(E) / len(s), m / len(s), float(d2.mean().sqrt())]
        if 0.5 * float(U.diagonal()[:3].sum() - 1.0) >= 1 - 1e-6 and float((U[:3, 3] ** 2).sum()) <= 1e-6:
            break
    return T, stats


def filtered64(depth, case):
    """the bilateral filter of a depth image (float64), and the frame's points in raster order"""
    d = torch.from_numpy(depth.astype(np.int32)).cuda()
    h, w = d.shape
    dv = d.float() * torch.tensor(DEPTH_SCALE, dtype=torch.float32, device="cuda")
    use = (dv >= T_MIN) & (dv <= T_MAX)
    if case["filter"] == "adaptive":
        step = torch.floor((dv - torch.tensor(T_MIN, dtype=torch.float32, device="cuda")) / 0.5).clamp(0, 5).double()
        rad, ss, sd, most = step, 8.0 + step, 100.0 + 10.0 * step, 5
    else:
        most = case["radius"]
        rad, ss, sd = (torch.full((h, w), v, dtype=torch.float64, device="cuda") for v in (float(most), 3.0, 30.0))
    out = d.double()
    if case["filter"] != "none":
        pad = torch.nn.functional.pad(d, (most, most, most, most))
        sw, sv = torch.zeros_like(out), torch.zeros_like(out)
        for dy in range(-most, most + 1):
            for dx in range(-most, most + 1):
                nb = pad[most + dy:most + dy + h, most + dx:most + dx + w].double()
                wgt = torch.exp(-(dx * dx + dy * dy) / ss ** 2) * torch.exp(-((out - nb) ** 2) / sd ** 2)
                wgt = torch.where((nb > 0) & (max(abs(dx), abs(dy)) <= rad), wgt, 0.0)
                sw += wgt
                sv += wgt * nb
        out = torch.where(use, sv / sw, out)
    z = out * float(np.float32(DEPTH_SCALE))
    cam = camera(case)
    v, u = torch.meshgrid(torch.arange(h, device="cuda") - 0.5, torch.arange(w, device="cuda") - 0.5, indexing="ij")
    p = torch.stack([(u - cam.cx) * z / float(np.float32(cam.fx)), (v - cam.cy) * z / float(np.float32(cam.fy)), z], -1)
    return p[(z >= T_MIN) & (z <= T_MAX)]


def padded(x, n):
    out = torch.zeros((n,) + tuple(x.shape[1:]), dtype=torch.float64, device="cuda")
    out[:len(x)] = x
    return out


def as_result(T, stats):
    return {"T": T.cpu().numpy()[None], "stats": np.array([stats]), "counts": None}


def exact(case, seed):
    k = case["kind"]
    # a batch takes minutes here; a tracked frame's colours are read at pixel boundaries, where
    # rounding decides between two pixels, so its poses have no 64-bit value
    if k == "track" or (k == "register" and case["pairs"] > 1):
        return None
    a = inputs(case, seed)
    eye = torch.eye(4, dtype=torch.float64, device="cuda")
    if k == "voxel":
        x, c = voxels(a.x, a.c, case["voxel"])
        n = len(a.x)
        return {"xyz": padded(x, n), "intensity": padded(intensity(c), n), "rgb": padded(c, n), "count": None}
    if k == "frame":
        p = filtered64(a.frames[0][0], case)
        return {"xyz": padded(p, case["w"] * case["h"]), "intensity": None, "rgb": None, "count": None}
    if k == "normals":
        return normals64(a.x, case["radius"], case["max_nn"])
    if k == "gradient":
        return gradients64(a.x, intensity(a.c), a.nrm, case["radius"])
    if k == "nn":
        return nearest(a.q, a.r, case["radius"]).to(torch.int32)
    if k == "outlier":
        i, _ = neighbours(a.x, a.x, case["radius"])
        keep = torch.bincount(i, minlength=len(a.x)) > case["min_neighbors"]
        n = len(a.x)
        return {"xyz": padded(a.x[keep], n), "rgb": padded(a.c[keep], n), "count": None}
    if k == "align":
        s, t, ti = a.sx.double(), a.tx.double(), intensity(a.tc)
        g = gradients64(a.tx, ti, a.tn, case["grad_radius"])
        return as_result(*icp64(s, intensity(a.sc), t, ti, a.tn.double(), g, case["max_corr"], case["max_iter"], euler,
                                eye))
    if k == "vjp":
        xi0, dT, dE = loss_seed(seed)
        x0 = torch.tensor(xi0, device="cuda", requires_grad=True)
        s, c = a.sx.double().requires_grad_(), a.sc.double().requires_grad_()
        si, ti = intensity(c), intensity(a.tc)
        fixed = (s, si, a.tx.double(), ti, a.tn.double(), a.tg.double(), case["max_corr"])
        T = torch.matrix_exp(hat(x0))
        for _ in range(case["steps"]):
            H, b = evaluate(T, *fixed)[:2]
            T = torch.matrix_exp(hat(-torch.linalg.solve(H, b))) @ T
        E = evaluate(T, *fixed)[2]
        ((torch.tensor(dT, device="cuda") * T)[:3].sum() + dE * E).backward()
        # the steps contract, so the start's own gradient is nearly zero: rounding error in any precision
        return {"T": T.detach().cpu().numpy(), "E": float(E), "dxi0": None, "dxyz": s.grad, "drgb": c.grad}
    sx, sc, tx, tc = a.pairs[0]
    T, stats = eye, None
    for voxel, iters, max_corr, rn, rg in SCALES:
        (s, c), (t, ct) = voxels(sx, sc, voxel), voxels(tx, tc, voxel)
        ti = intensity(ct)
        n = normals64(t, rn)
        T, stats = icp64(s, intensity(c), t, ti, n, gradients64(t, ti, n, rg), max_corr, iters,
                         lambda x: torch.matrix_exp(hat(x)), T)
    return as_result(T, stats)
