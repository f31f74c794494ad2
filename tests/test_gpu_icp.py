"""GPU colored ICP through the C ABI against the FP64 oracle.

Pose tolerance: rotation and translation error <= 1e-5 rad / 1e-5 m against the
FP64 oracle run on the same inputs with the same schedule; batched, graph-replayed
and single-pair runs are bit-identical to each other."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

POSE_TOL = 1e-5


@pytest.fixture(scope="module")
def N():
    from cuda_3d_gb300 import build, native

    build.build()
    return native


@pytest.fixture(scope="module")
def ctx(N):
    return N.Context(0)


@pytest.fixture(scope="module")
def synth():
    from cuda_3d_gb300 import synth as S

    return S


def c1_scales(N=None, O=None):
    spec = [(0.04, 50, 0.06, 0.08, 0.08), (0.02, 30, 0.03, 0.04, 0.04), (0.01, 14, 0.015, 0.02, 0.02)]
    if N is not None:
        return [N.scale(*s) for s in spec]
    return [O.Scale(*s) for s in spec]


@pytest.fixture(scope="module")
def pair_c1(synth):
    return synth.room_pair(seed=1, n_points=250_000, rot_deg=10.0, trans=0.10)


def run_gpu(ctx, N, pair, scales, **kw):
    src = ctx.cloud_from(pair.src_xyz, pair.src_rgb)
    tgt = ctx.cloud_from(pair.tgt_xyz, pair.tgt_rgb)
    return N.color_icp(ctx, src, tgt, N.icp_params(scales, **kw))


@pytest.mark.parametrize("update", ["se3", "euler"])
def test_icp_c1_vs_fp64_oracle(ctx, N, orc, synth, pair_c1, update):
    um = N.UPDATE_SE3_EXP if update == "se3" else N.UPDATE_EULER_ZYX
    r = run_gpu(ctx, N, pair_c1, c1_scales(N), update_map=um)
    T64, res = orc.multiscale_f64(pair_c1.src_xyz, pair_c1.src_rgb, pair_c1.tgt_xyz, pair_c1.tgt_rgb,
                                  c1_scales(O=orc), update_map=um)
    rot, tr = synth.pose_error(r["T"], T64)
    assert rot <= POSE_TOL and tr <= POSE_TOL, (rot, tr)
    assert r["iterations"] == sum(x.iterations for x in res)
    assert abs(r["fitness"] - res[-1].fitness) < 1e-3
    assert abs(r["inlier_rmse"] - res[-1].inlier_rmse) < 1e-3 * res[-1].inlier_rmse + 1e-7
    # and the registration itself recovers the ground truth
    rot_gt, tr_gt = synth.pose_error(r["T"], pair_c1.T_gt)
    assert rot_gt < np.radians(0.05) and tr_gt < 0.002


def test_icp_plain_and_compensated_agree(ctx, N, synth, pair_c1):
    rc = run_gpu(ctx, N, pair_c1, c1_scales(N), update_map=N.UPDATE_SE3_EXP, compensated=True)
    rp = run_gpu(ctx, N, pair_c1, c1_scales(N), update_map=N.UPDATE_SE3_EXP, compensated=False)
    rot, tr = synth.pose_error(rc["T"], rp["T"])
    assert rot <= POSE_TOL and tr <= POSE_TOL, (rot, tr)
    assert rc["scale_iterations"] == rp["scale_iterations"]


def test_icp_reference_single_level_align(ctx, N, orc, synth):
    """the reference's color_icp::align: clouds used as given, target normals
    estimated beforehand, colour gradients on the target, Euler ZYX steps"""
    pair = synth.room_pair(seed=5, n_points=120_000, rot_deg=3.0, trans=0.03)
    sx, sc, _, _ = orc.voxel_downsample(pair.src_xyz, pair.src_rgb, 0.02)
    tx, tc, _, _ = orc.voxel_downsample(pair.tgt_xyz, pair.tgt_rgb, 0.02)
    src, tgt = ctx.cloud_from(sx, sc), ctx.cloud_from(tx, tc)
    ctx.check(ctx.L.gca3d_estimate_normals(ctx.h, tgt.h, 0.05, 0))
    tn = tgt.download(xyz=False, rgb=False, normals=True)["normals"].astype(np.float64)
    p = N.icp_params([N.scale(0.0, 100, 0.05, 0.0, 0.04)], keep_target_normals=True)
    r = N.color_icp(ctx, src, tgt, p)
    tg = orc.gradient_f64(tx, tc, tn, 0.04)
    o = orc.color_icp_f64(sx, sc, tx, tc, tn, tg, max_iter=100, max_corr=0.05)
    rot, tr = synth.pose_error(r["T"], o.T)
    assert rot <= POSE_TOL and tr <= POSE_TOL, (rot, tr)
    assert r["iterations"] == o.iterations and r["converged"] == o.converged
    np.testing.assert_allclose(r["rmse_ref"], o.rmse_ref, rtol=1e-3)
    # the reference's own FP32 loop (in-place FP32 transforms) lands close by
    r32 = orc.color_icp_ref32(sx, sc, tx, tc, tn.astype(np.float32), tg.astype(np.float32), 100, 0.05)
    rot32, tr32 = synth.pose_error(r["T"], r32.T)
    assert rot32 < 1e-3 and tr32 < 1e-3


def make_batch(synth, k=6, seed=0):
    rng = np.random.default_rng(seed)
    return [synth.room_pair(seed=100 + i, n_points=int(rng.integers(15_000, 90_000)),
                            overlap=float(rng.uniform(0.5, 0.9)), rot_deg=float(rng.uniform(0, 6)),
                            trans=float(rng.uniform(0, 0.06))) for i in range(k)]


def small_scales(N):
    return [N.scale(0.05, 30, 0.1, 0.1, 0.1), N.scale(0.025, 20, 0.05, 0.05, 0.05)]


def test_batched_bit_identical_to_single(ctx, N, synth):
    pairs = make_batch(synth)
    srcs = [ctx.cloud_from(p.src_xyz, p.src_rgb) for p in pairs]
    tgts = [ctx.cloud_from(p.tgt_xyz, p.tgt_rgb) for p in pairs]
    prm = N.icp_params(small_scales(N), update_map=N.UPDATE_SE3_EXP, use_graph=True)
    batched = N.color_icp_batched(ctx, srcs, tgts, prm)
    for s, t, b in zip(srcs, tgts, batched):
        single = N.color_icp(ctx, s, t, prm)
        np.testing.assert_array_equal(single["T"], b["T"])
        assert single["iterations"] == b["iterations"]
        assert single["fitness"] == b["fitness"]


@pytest.mark.parametrize("k", [63, 64, 65, 129, 4095, 4096])
def test_many_pairs_bit_identical_to_single(ctx, N, synth, k):
    """pair counts around the widths of the item map's search, up to the largest allowed;
    clouds are shared, and empty ones (pairs without work items) lie at the start, at the end
    and in runs between"""
    base = [synth.room_pair(seed=300 + j, n_points=700 + 151 * j, rot_deg=2.0, trans=0.02) for j in range(5)]
    S = [ctx.cloud_from(p.src_xyz, p.src_rgb) for p in base] + [ctx.cloud(16)]
    T = [ctx.cloud_from(p.tgt_xyz, p.tgt_rgb) for p in base] + [ctx.cloud(16)]
    rng = np.random.default_rng(k)
    which = rng.integers(0, 5, k)
    for at in (0, 1, k // 2, k - 1):
        which[at] = 5
    which[k // 3: k // 3 + 35] = 5
    prm = N.icp_params([N.scale(0.15, 4, 0.5, 0.6, 0.6)], use_graph=True)
    single = [N.IcpPlan(ctx, [s], [t], prm).execute()[0] for s, t in zip(S, T)]
    assert all(r["status"] == N.OK for r in single[:5]) and single[5]["status"] == N.ERR_NO_CORRESPONDENCES
    many = N.IcpPlan(ctx, [S[j] for j in which], [T[j] for j in which], prm).execute()
    for j, r in zip(which, many):
        assert r["status"] == single[j]["status"] and r["iterations"] == single[j]["iterations"]
        np.testing.assert_array_equal(r["T"], single[j]["T"])


@pytest.mark.parametrize("compensated", [True, False])
@pytest.mark.parametrize("k", [2, 3, 300])
def test_finalize_forms_give_the_same_poses(ctx, N, synth, k, compensated):
    """the finalize with a cluster per pair and with a block per pair, on either side of the line
    between them (48 blocks of 1024 points a pair, by the clouds' capacity) and far from it,
    against one pair at a time"""
    base = [synth.room_pair(seed=400 + j, n_points=(700, 9_001, 30_000)[j], rot_deg=2.0, trans=0.02)
            for j in range(3)]
    T = [ctx.cloud_from(p.tgt_xyz, p.tgt_rgb) for p in base]
    scales = [N.scale(0.0, 4, 0.3, 0.4, 0.4), N.scale(0.05, 3, 0.2, 0.3, 0.3)]
    prm = N.icp_params(scales, use_graph=True, compensated=compensated)
    want = None
    for blocks in (30, 47, 48, 49) if k < 10 else (30,):
        S = [ctx.cloud_from(p.src_xyz, p.src_rgb, capacity=blocks * 1024) for p in base]
        if want is None:
            want = [N.IcpPlan(ctx, [s], [t], prm).execute()[0] for s, t in zip(S, T)]
            assert all(r["status"] == N.OK for r in want)
        got = N.IcpPlan(ctx, [S[j % 3] for j in range(k)], [T[j % 3] for j in range(k)], prm).execute()
        for j, r in enumerate(got):
            assert r["scale_iterations"] == want[j % 3]["scale_iterations"]
            assert r["fitness"] == want[j % 3]["fitness"] and r["inlier_rmse"] == want[j % 3]["inlier_rmse"]
            np.testing.assert_array_equal(r["T"], want[j % 3]["T"])


@pytest.mark.parametrize("compensated", [True, False])
@pytest.mark.parametrize("n", [1000, 8192, 65_536, 65_537, 131_073])
def test_finalize_sums_of_every_length(ctx, N, synth, n, compensated):
    """the cluster's finalize and the fused one (one block's sums, in the same order) for 1, 8, 64,
    65 and 129 partials: the same poses bit for bit"""
    p = synth.room_pair(seed=5, n_points=n, rot_deg=2.0, trans=0.02)
    S, T = ctx.cloud_from(p.src_xyz, p.src_rgb), ctx.cloud_from(p.tgt_xyz, p.tgt_rgb)
    r = 12.0 / np.sqrt(n)
    got = [N.IcpPlan(ctx, [S], [T], N.icp_params([N.scale(0.0, 5, r, r, r)], use_graph=True, compensated=compensated,
                                                 tuning=N.Tuning(0, 0, 0, 0, fused, 0))).execute()[0] for fused in (0, 1)]
    assert got[0]["status"] == N.OK and got[0]["iterations"] == got[1]["iterations"]
    assert got[0]["fitness"] == got[1]["fitness"] and got[0]["inlier_rmse"] == got[1]["inlier_rmse"]
    np.testing.assert_array_equal(got[0]["T"], got[1]["T"])


def test_plain_sums_cost_no_more_than_compensated(ctx, N, synth):
    """FP32 sums without compensation are the cheaper option of the two: a registration with
    them takes at most a little longer (it took 1.26 times as long when their partials were read
    one after the other)"""
    import time

    p = synth.room_pair(seed=3, n_points=120_000, rot_deg=8.0, trans=0.1)
    S, T = ctx.cloud_from(p.src_xyz, p.src_rgb), ctx.cloud_from(p.tgt_xyz, p.tgt_rgb)

    def best(compensated):
        plan = N.IcpPlan(ctx, [S], [T], N.icp_params([N.scale(0.0, 20, 0.14, 0.05, 0.05)], use_graph=True, rot_eps=1e-30,
                                                     trans_eps=0.0, compensated=compensated))
        times = []
        for _ in range(15):
            t0 = time.perf_counter()
            r = plan.execute()[0]
            times.append(time.perf_counter() - t0)
        assert r["iterations"] == 20
        return min(times)

    assert best(False) < 1.15 * best(True)


def test_one_shot_calls_share_a_workspace(N, synth):
    """one context's one-shot calls reuse one workspace: sizes, pair counts and scales that
    grow and shrink, a refused call and a call without correspondences in between give the
    bits of a fresh context each"""
    pairs = [synth.room_pair(seed=40 + k, n_points=n, rot_deg=2.0, trans=0.02)
             for k, n in enumerate((4_000, 20_000, 9_000))]
    two = [N.scale(0.1, 10, 0.2, 0.2, 0.2), N.scale(0.05, 10, 0.1, 0.1, 0.1)]
    one = [N.scale(0.06, 15, 0.12, 0.12, 0.12)]
    calls = [((0,), one), ((1,), two), ((0, 1, 2), two), ((2,), one), ((1, 0), one), ((0,), two)]

    def run(c, which, scales):
        s = [c.cloud_from(pairs[k].src_xyz, pairs[k].src_rgb) for k in which]
        t = [c.cloud_from(pairs[k].tgt_xyz, pairs[k].tgt_rgb) for k in which]
        return N.color_icp_batched(c, s, t, N.icp_params(scales))

    shared = N.Context(0)
    for k, (which, scales) in enumerate(calls):
        got = run(shared, which, scales)
        want = run(N.Context(0), which, scales)
        for a, b in zip(got, want):
            assert a["status"] == N.OK and a["scale_iterations"] == b["scale_iterations"]
            np.testing.assert_array_equal(a["T"], b["T"])
        if k == 1:
            with pytest.raises(N.GcaError):
                run(shared, (0,), [N.scale(0.1, 10, -1.0, 0.2, 0.2)])
        if k == 3:
            far = shared.cloud_from(pairs[0].src_xyz + 50.0, pairs[0].src_rgb)
            tgt = shared.cloud_from(pairs[0].tgt_xyz, pairs[0].tgt_rgb)
            r = N.color_icp(shared, far, tgt, N.icp_params(one))
            assert r["status"] == N.ERR_NO_CORRESPONDENCES


def test_one_shot_workspace_grows_with_the_pairs(N, synth):
    """a call with more pairs than the kept workspace holds leaves one that holds them: calls
    with three pairs cost the same whether the context's first call had one pair or three (they
    took 1.5 times as long while the small workspace stayed and theirs was made and freed)"""
    import time

    pairs = [synth.room_pair(seed=500 + k, n_points=20_000, rot_deg=2.0, trans=0.02) for k in range(3)]
    prm = N.icp_params([N.scale(0.05, 10, 0.1, 0.1, 0.1)])

    def best(first):
        c = N.Context(0)
        S = [c.cloud_from(p.src_xyz, p.src_rgb) for p in pairs]
        T = [c.cloud_from(p.tgt_xyz, p.tgt_rgb) for p in pairs]
        N.color_icp_batched(c, S[:first], T[:first], prm)
        times = []
        for _ in range(20):
            t0 = time.perf_counter()
            N.color_icp_batched(c, S, T, prm) # waits for its results
            times.append(time.perf_counter() - t0)
        return min(times)

    three = min(best(3), best(3))
    assert min(best(1), best(1)) < 1.3 * three


@pytest.mark.parametrize("k,n_points", [(1, 600), (1, 6_000), (3, 6_000), (2, 530_000)])
@pytest.mark.parametrize("mode", ["shared_grid", "two_grids", "kept_normals", "kept_two_grids", "capped"])
@pytest.mark.parametrize("graph", [False, True])
def test_preparation_branches_equal_serial(N, synth, k, n_points, mode, graph):
    """the preparation on its branches (the last size is above the line up to which the normals
    have one) gives the bits of the preparation on the context stream alone, also on a repeat"""
    if n_points > 100_000 and (mode != "two_grids" or not graph):
        pytest.skip("one form of the large size")
    ctx = N.Context(0)
    pairs = [synth.room_pair(seed=60 + j, n_points=n_points, rot_deg=2.0, trans=0.02) for j in range(k)]
    S = [ctx.cloud_from(p.src_xyz, p.src_rgb) for p in pairs]
    T = [ctx.cloud_from(p.tgt_xyz, p.tgt_rgb) for p in pairs]
    kept = mode.startswith("kept")
    corr = 0.1 if mode in ("two_grids", "kept_two_grids") else 0.3
    kw = dict(max_nn=12) if mode == "capped" else {}
    if kept:
        for t in T:
            ctx.check(ctx.L.gca3d_estimate_normals(ctx.h, t.h, 0.3, 0))
        scales = [N.scale(0.0, 4, corr, 0.3, 0.3), N.scale(0.0, 3, corr / 2, 0.3, 0.3)]
    else:
        scales = [N.scale(v, 4, corr * v / 0.1, 0.3 * v / 0.1, 0.3 * v / 0.1, **kw) for v in (0.1, 0.05, 0.025)]
    got = {}
    for serial in (0, 1):
        prm = N.icp_params(scales, use_graph=graph, keep_target_normals=kept,
                           tuning=N.Tuning(0, 0, 0, 0, 0, serial))
        plan = N.IcpPlan(ctx, S, T, prm)
        got[serial] = [plan.execute() for _ in range(2)]
    for reps in zip(*got[0], *got[1]):
        for r in reps[:-1]:
            assert r["status"] == reps[-1]["status"] and r["scale_iterations"] == reps[-1]["scale_iterations"]
            np.testing.assert_array_equal(r["T"], reps[-1]["T"])
    # 600 points are too sparse to register: there both end with the same status
    assert n_points <= 600 or all(r["scale_iterations"][0] > 0 for r in got[1][0])


@pytest.mark.parametrize("n_points", [(1 << 19) - 1, 1 << 19, (1 << 19) + 1])
def test_item_size_rule_equals_every_item_size(ctx, N, synth, n_points):
    """two pairs around the line at which the default work item of the search doubles: the poses
    of every item size, with a last item of one point or one short of full"""
    pairs = [synth.room_pair(seed=80 + j, n_points=n_points, rot_deg=2.0, trans=0.02) for j in range(2)]
    S = [ctx.cloud_from(p.src_xyz, p.src_rgb) for p in pairs]
    T = [ctx.cloud_from(p.tgt_xyz, p.tgt_rgb) for p in pairs]
    got = [N.IcpPlan(ctx, S, T, N.icp_params([N.scale(0.05, 4, 0.06, 0.1, 0.1)], use_graph=True,
                                             tuning=N.Tuning(item))).execute() for item in (0, 64, 128, 256, 512)]
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert a["status"] == b["status"] == N.OK and a["iterations"] == b["iterations"]
            np.testing.assert_array_equal(a["T"], b["T"])


def test_plan_graph_replay(ctx, N, synth):
    pairs = make_batch(synth, k=4, seed=1)
    srcs = [ctx.cloud_from(p.src_xyz, p.src_rgb) for p in pairs]
    tgts = [ctx.cloud_from(p.tgt_xyz, p.tgt_rgb) for p in pairs]
    eager = N.color_icp_batched(ctx, srcs, tgts, N.icp_params(small_scales(N), use_graph=True))
    plan = N.IcpPlan(ctx, srcs, tgts, N.icp_params(small_scales(N), use_graph=True))
    assert plan.kernels() > 0
    for _ in range(2):
        res = plan.execute()
        for a, b in zip(res, eager):
            np.testing.assert_array_equal(a["T"], b["T"])
            assert a["iterations"] == b["iterations"]
    # initial poses are honoured: starting at the answer converges at once
    Ts = np.stack([r["T"] for r in eager])
    res = plan.execute(T_init=Ts)
    for a, b in zip(res, eager):
        rot, tr = synth.pose_error(a["T"], b["T"])
        assert rot < 1e-4 and tr < 1e-4
    # new cloud contents are picked up by the replay
    p = pairs[0]
    srcs[0].upload(p.src_xyz[: len(p.src_xyz) // 2], p.src_rgb[: len(p.src_xyz) // 2])
    res = plan.execute()
    assert res[0]["n_src"] < eager[0]["n_src"]


def test_plain_mode_matches_graph_mode(ctx, N, synth):
    pairs = make_batch(synth, k=3, seed=2)
    srcs = [ctx.cloud_from(p.src_xyz, p.src_rgb) for p in pairs]
    tgts = [ctx.cloud_from(p.tgt_xyz, p.tgt_rgb) for p in pairs]
    a = N.color_icp_batched(ctx, srcs, tgts, N.icp_params(small_scales(N), use_graph=False))
    b = N.color_icp_batched(ctx, srcs, tgts, N.icp_params(small_scales(N), use_graph=True))
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x["T"], y["T"])


def test_no_correspondences(ctx, N, synth):
    p = synth.room_pair(seed=9, n_points=20_000)
    src = ctx.cloud_from(p.src_xyz + np.float32(50.0), p.src_rgb)
    tgt = ctx.cloud_from(p.tgt_xyz, p.tgt_rgb)
    r = N.color_icp(ctx, src, tgt, N.icp_params([N.scale(0.05, 10, 0.1, 0.1, 0.1)]))
    assert r["status"] == N.ERR_NO_CORRESPONDENCES
    np.testing.assert_allclose(r["T"], np.eye(4), atol=1e-12)
    assert r["iterations"] == 1 and r["converged"]
    assert r["fitness"] == 0.0


def test_empty_source(ctx, N, synth):
    p = synth.room_pair(seed=9, n_points=20_000)
    src = ctx.cloud(100)
    tgt = ctx.cloud_from(p.tgt_xyz, p.tgt_rgb)
    r = N.color_icp(ctx, src, tgt, N.icp_params([N.scale(0.05, 10, 0.1, 0.1, 0.1)]))
    assert r["status"] == N.ERR_NO_CORRESPONDENCES and r["iterations"] == 0
    np.testing.assert_array_equal(r["T"], np.eye(4))


def test_invalid_params(ctx, N):
    src, tgt = ctx.cloud(10), ctx.cloud(10)
    res = N.IcpResult()
    for bad in (N.icp_params([N.scale(0.05, 10, 0.1, 0.1, 0.1)], lam=1.5),
                N.icp_params([N.scale(0.05, 10, -0.1, 0.1, 0.1)]),
                N.icp_params([N.scale(0.05, 10, 0.1, 0.1, 0.1, 65)])):
        assert ctx.L.gca3d_color_icp(ctx.h, src.h, tgt.h, C.byref(bad), None, C.byref(res)) == N.ERR_INVALID_VALUE
    p = N.icp_params([N.scale(0.0, 10, 0.1, 0.0, 0.1)], keep_target_normals=True)
    assert ctx.L.gca3d_color_icp(ctx.h, src.h, tgt.h, C.byref(p), None, C.byref(res)) == N.ERR_INVALID_VALUE


def test_frame_pair_pipeline_vs_oracle(ctx, N, orc, synth):
    """the frame-pair workload: two 640x480 RGB-D frames -> filtered clouds ->
    0.01 m voxels -> normals (r 0.02, at most 30 neighbours) -> single-level ICP"""
    fp = synth.frame_pair(seed=0)
    clouds = []
    for depth, bgr in ((fp.depth1, fp.bgr1), (fp.depth0, fp.bgr0)):
        d, c = ctx.alloc(depth.nbytes), ctx.alloc(bgr.nbytes)
        d.write(depth)
        c.write(bgr)
        out = ctx.cloud(depth.size)
        di = N.Intrinsics(525.0, 525.0, 319.5, 239.5)
        f = N.Filter(N.FILTER_FIXED, 2, 3.0, 30.0)
        ctx.check(ctx.L.gca3d_frame_to_cloud(ctx.h, d.ptr, c.ptr, 640, 480, C.byref(di), None, None, 0.001, 0.2,
                                             10.0, C.byref(f), out.h))
        clouds.append(out)
    src, tgt = clouds
    sc = [N.scale(0.01, 30, 0.03, 0.02, 0.02, 30)]
    r = N.color_icp(ctx, src, tgt, N.icp_params(sc, update_map=N.UPDATE_SE3_EXP))
    s, t = src.download(), tgt.download()
    T64, res = orc.multiscale_f64(s["xyz"], s["rgb"], t["xyz"], t["rgb"], [orc.Scale(0.01, 30, 0.03, 0.02, 0.02, 30)])
    rot, tr = synth.pose_error(r["T"], T64)
    assert rot <= POSE_TOL and tr <= POSE_TOL, (rot, tr)
    # a 2 deg rotation moves points at 2-4 m by 7-14 cm, beyond the 3 cm correspondence
    # limit of this single-level schedule, so it is not expected to reach the ground
    # truth; a coarse-to-fine schedule on the same clouds, run to a tight convergence
    # test (the reference's stops at 1 mm steps), does, which checks the geometry of
    # the frame stage (intrinsics, half-pixel shift, colour lookup)
    sc3 = [N.scale(0.04, 30, 0.15, 0.08, 0.08), N.scale(0.02, 30, 0.06, 0.04, 0.04),
           N.scale(0.01, 30, 0.03, 0.02, 0.02, 30)]
    r3 = N.color_icp(ctx, src, tgt, N.icp_params(sc3, update_map=N.UPDATE_SE3_EXP, rot_eps=1e-10, trans_eps=1e-10))
    rot_gt, tr_gt = synth.pose_error(r3["T"], fp.T_gt)
    assert rot_gt < np.radians(0.05) and tr_gt < 0.001, (np.degrees(rot_gt), tr_gt)


def test_autotune_and_every_launch_shape_give_identical_results(ctx, N, synth):
    """the autotuner returns a valid launch shape, and the shape never changes a bit
    of the result (partials are per 1024-point item and summed in item order)"""
    pairs = synth.batch_pairs(8, seed=3, n_min=20_000, n_max=60_000)
    srcs = [ctx.cloud_from(p.src_xyz, p.src_rgb) for p in pairs]
    tgts = [ctx.cloud_from(p.tgt_xyz, p.tgt_rgb) for p in pairs]
    prm = N.icp_params(c1_scales(N), update_map=N.UPDATE_SE3_EXP, use_graph=True)
    best, ms = N.icp_autotune(ctx, srcs, tgts, prm, reps=1)
    assert best.nn_item_points in (64, 128, 256, 512)
    assert best.nn_blocks_per_sm > 0 and best.accum_blocks_per_sm > 0 and ms > 0
    ref = N.IcpPlan(ctx, srcs, tgts, prm).execute(results=True)
    for tune in (best, N.Tuning(64, 4, 2), N.Tuning(512, 20, 12), N.Tuning(128, 6, 3, 0, 1)):
        p2 = N.icp_params(c1_scales(N), update_map=N.UPDATE_SE3_EXP, use_graph=True, tuning=tune)
        got = N.IcpPlan(ctx, srcs, tgts, p2).execute(results=True)
        for a, b in zip(ref, got):
            np.testing.assert_array_equal(a["T"], b["T"])
            assert a["iterations"] == b["iterations"]


@pytest.mark.parametrize("use_graph", [True, False])
def test_preparation_branch_changes_no_bit(ctx, N, synth, use_graph):
    """Every scale's clouds, grids and normals prepared on a branch of their own that runs
    ahead of the iterations (default) or on the context stream before each scale's
    iterations: the same kernels on the same data, so the same bits."""
    pairs = synth.batch_pairs(10, seed=7, n_min=10_000, n_max=80_000)
    srcs = [ctx.cloud_from(p.src_xyz, p.src_rgb) for p in pairs]
    tgts = [ctx.cloud_from(p.tgt_xyz, p.tgt_rgb) for p in pairs]
    out = []
    for serial in (0, 1):
        prm = N.icp_params(c1_scales(N), update_map=N.UPDATE_SE3_EXP, use_graph=use_graph,
                           tuning=N.Tuning(0, 0, 0, 0, 0, serial))
        plan = N.IcpPlan(ctx, srcs, tgts, prm)
        out.append([plan.execute(results=True) for _ in range(2)])
    for run0, run1 in zip(*out):
        for a, b in zip(run0, run1):
            np.testing.assert_array_equal(a["T"], b["T"])
            for k in ("iterations", "fitness", "inlier_rmse", "rmse_ref", "scale_iterations", "scale_n_src"):
                assert a[k] == b[k], k


def test_queued_executes_read_their_own_results(ctx, N, synth):
    """Two plans executed back to back without waiting: each plan's results() waits
    for its own execute (the state copy queued behind it) and returns that execute's
    results, equal to a waiting execute's; a plan never executed has no results."""
    pairs = synth.batch_pairs(8, seed=6, n_min=20_000, n_max=60_000)
    srcs = [ctx.cloud_from(p.src_xyz, p.src_rgb) for p in pairs]
    tgts = [ctx.cloud_from(p.tgt_xyz, p.tgt_rgb) for p in pairs]
    prm = N.icp_params(c1_scales(N), update_map=N.UPDATE_SE3_EXP, use_graph=True)
    a = N.IcpPlan(ctx, srcs[:4], tgts[:4], prm)
    b = N.IcpPlan(ctx, srcs[4:], tgts[4:], prm)
    res = N.IcpResult * 4
    assert ctx.L.gca3d_icp_plan_results(a.h, res()) == N.ERR_INVALID_VALUE
    ref_a, ref_b = a.execute(results=True), b.execute(results=True)
    for _ in range(3):
        a.execute(results=False)
        b.execute(results=False)
        got_a = a.results()
        got_b = b.results()
        for ref, got in ((ref_a, got_a), (ref_b, got_b)):
            for x, y in zip(ref, got):
                np.testing.assert_array_equal(x["T"], y["T"])
                assert x["iterations"] == y["iterations"]


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("compensated", [True, False])
def test_fused_and_separate_finalize_agree(ctx, N, synth, use_graph, compensated):
    """The finalize run by each pair's last accumulate block and as a launch of its
    own (default) give the same bits: the same partials summed in the same order, the
    same solve.  Pairs converge at different iterations, so the fused path also
    rebuilds the work maps while other pairs are still accumulating."""
    pairs = synth.batch_pairs(12, seed=5, n_min=10_000, n_max=90_000)
    srcs = [ctx.cloud_from(p.src_xyz, p.src_rgb) for p in pairs]
    tgts = [ctx.cloud_from(p.tgt_xyz, p.tgt_rgb) for p in pairs]
    out = []
    for fused in (0, 1):
        prm = N.icp_params(c1_scales(N), update_map=N.UPDATE_SE3_EXP, use_graph=use_graph, compensated=compensated,
                           tuning=N.Tuning(0, 0, 0, 0, fused))
        out.append(N.IcpPlan(ctx, srcs, tgts, prm).execute(results=True))
    iters = set()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a["T"], b["T"])
        for k in ("iterations", "converged", "status", "fitness", "inlier_rmse", "rmse_ref", "scale_iterations"):
            assert a[k] == b[k], k
        iters.add(tuple(a["scale_iterations"]))
    assert len(iters) > 1  # the pairs stop at different iterations
    # a single pair (its last block is the last of the iteration), an empty source
    # alone (no item at all: the iteration still ends the loop) and beside others
    empty = ctx.cloud(100)
    cases = [([srcs[0]], [tgts[0]]), ([empty], [tgts[0]]), ([srcs[1], empty, srcs[2]], tgts[1:4])]
    for cs, ct in cases:
        got = []
        for fused in (0, 1):
            prm = N.icp_params(c1_scales(N), update_map=N.UPDATE_SE3_EXP, use_graph=use_graph,
                               compensated=compensated, tuning=N.Tuning(0, 0, 0, 0, fused))
            got.append(N.IcpPlan(ctx, cs, ct, prm).execute(results=True))
        for a, b in zip(*got):
            np.testing.assert_array_equal(a["T"], b["T"])
            assert a["iterations"] == b["iterations"] and a["status"] == b["status"]
        for r, c in zip(got[0], cs):
            if c is empty:
                assert r["status"] == N.ERR_NO_CORRESPONDENCES and r["iterations"] == 0


@pytest.mark.parametrize("voxels", [(0.04, 0.02, 0.01), (0.08, 0.04, 0.02, 0.01), (0.05, 0.02, 0.01)])
def test_voxel_refinement_changes_no_bit(ctx, N, synth, voxels):
    """Where the voxel sizes halve from scale to scale, one sort at the coarser scale
    carries the finer scales' sub-cell bits and each finer scale only splits the coarser
    voxels' runs; with voxel_resort every scale sorts anew.  Both give the same voxels in
    the same order, so every result is bit-identical (0.05 -> 0.02 does not halve: a new
    sort there, a refinement after it)."""
    pairs = synth.batch_pairs(8, seed=4, n_min=20_000, n_max=80_000)
    srcs = [ctx.cloud_from(p.src_xyz, p.src_rgb) for p in pairs]
    tgts = [ctx.cloud_from(p.tgt_xyz, p.tgt_rgb) for p in pairs]
    scales = [N.scale(v, 20, 1.5 * v, 2 * v, 2 * v) for v in voxels]
    out = []
    for resort in (0, 1):
        prm = N.icp_params(scales, update_map=N.UPDATE_SE3_EXP, use_graph=True, tuning=N.Tuning(0, 0, 0, resort))
        out.append(N.IcpPlan(ctx, srcs, tgts, prm).execute(results=True))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a["T"], b["T"])
        for k in ("iterations", "fitness", "inlier_rmse", "rmse_ref", "scale_iterations", "scale_n_src",
                  "scale_n_tgt"):
            assert a[k] == b[k], k


def test_fp64_pose_routines_vs_cuda(ctx, N):
    """The pose update's short FP64 routines on this device, against CUDA: the Newton
    reciprocal within 1 ulp of IEEE division over 2^-60 .. 2^60, the small-angle
    sine and cosine within 2 ulp of sincos for |x| <= 0.25, and the series of the
    exponential map's coefficients within the rounding bound of the closed forms
    (which cancel at small angles: eps (4 + 8 / t^2))."""
    r = N.selfcheck_fp64(ctx, 1 << 20)
    assert r["rcp_ulp"] <= 1.0
    assert r["sin_ulp"] <= 2.0 and r["cos_ulp"] <= 2.0
    assert r["exp_coeff_vs_bound"] <= 1.0
