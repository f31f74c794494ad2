"""GPU parity of the individual path stages, called through the C ABI.

Bit-exact against the oracle / the reference's own outputs (golden fixtures) for
keys, indices, neighbour lists, the voxel set and the rigid transform; within the
stated tolerances of the FP64 oracle for normals, gradients and the
Gauss-Newton system."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def N():
    from cuda_3d_gb300 import build, native

    build.build()
    return native


@pytest.fixture(scope="module")
def ctx(N):
    return N.Context(0)


@pytest.fixture(scope="module")
def room():
    from cuda_3d_gb300 import synth

    rng = np.random.default_rng(77)
    return synth.sample_room(synth.room_scene(1234), 250_000, rng)


def angle_err(a, b):
    """unsigned angle between line directions, atan2(|a x b|, |a . b|): arccos of a
    dot product near 1 reads sqrt(2 delta) for a rounding delta of the norms"""
    a = a / np.maximum(np.linalg.norm(a, axis=1, keepdims=True), 1e-30)
    b = b / np.maximum(np.linalg.norm(b, axis=1, keepdims=True), 1e-30)
    return np.arctan2(np.linalg.norm(np.cross(a, b), axis=1), np.abs((a * b).sum(1)))


# --------------------------------------------------------------------------- #
# cloud basics
# --------------------------------------------------------------------------- #
def test_upload_download_roundtrip(ctx, golden, orc):
    xyz, rgb = golden["cloud_xyz"], golden["cloud_rgb"]
    c = ctx.cloud_from(xyz, rgb)
    assert len(c) == len(xyz)
    d = c.download()
    np.testing.assert_array_equal(d["xyz"], xyz)
    np.testing.assert_array_equal(d["rgb"], rgb)


def test_intensity_equals_fp64(ctx):
    """the intensity of every point is the FP64 weighted sum rounded to float, bit for bit:
    random, 8-bit, grey, negative, tiny, huge and non-finite colours"""
    rng = np.random.default_rng(4)
    f = np.float32
    parts = [rng.random((200_000, 3)), rng.integers(0, 256, (50_000, 3)) * f(1 / 255),
             np.repeat(rng.integers(0, 256, (256, 1)) * f(1 / 255), 3, 1),
             rng.normal(size=(50_000, 3)) * 10.0 ** rng.integers(-44, 38, (50_000, 1)),
             np.array(np.meshgrid(*[[0.0, -0.0, 1.0, 1e-45, 3e38, np.inf, -np.inf, np.nan]] * 3)).reshape(3, -1).T]
    rgb = np.concatenate([p.astype(f) for p in parts])
    cloud = ctx.cloud_from(np.zeros_like(rgb), rgb)
    pos = np.empty((len(rgb), 4), f)
    ctx.check(ctx.L.gca3d_copy(ctx.h, pos.ctypes.data, cloud.device_views()[0], pos.nbytes))
    with np.errstate(all="ignore"):
        c = rgb.astype(np.float64)
        want = ((0.2126 * c[:, 0] + 0.7152 * c[:, 1]) + 0.0722 * c[:, 2]).astype(f)
    nan = np.isnan(want)
    np.testing.assert_array_equal(np.isnan(pos[:, 3]), nan)
    np.testing.assert_array_equal(pos[~nan, 3].view(np.uint32), want[~nan].view(np.uint32))


def test_upload_from_pinned_and_device_memory(ctx, N, golden):
    """Pinned host buffers and device buffers are read in place by the packing
    kernel; pageable ones go through a staging copy.  All three give the same cloud
    (positions with the intensity the ICP uses, and colours)."""
    torch = pytest.importorskip("torch")
    xyz, rgb = golden["cloud_xyz"], golden["cloud_rgb"]
    n = len(xyz)

    def device_arrays(c):
        pos, col = np.empty((n, 4), np.float32), np.empty((n, 4), np.float32)
        views = c.device_views()
        ctx.check(ctx.L.gca3d_copy(ctx.h, pos.ctypes.data_as(C.c_void_p), C.c_void_p(views[0]), n * 16))
        ctx.check(ctx.L.gca3d_copy(ctx.h, col.ctypes.data_as(C.c_void_p), C.c_void_p(views[1]), n * 16))
        return pos, col

    want = device_arrays(ctx.cloud_from(xyz, rgb))
    pinned = [torch.from_numpy(np.ascontiguousarray(a, np.float32)).pin_memory() for a in (xyz, rgb)]
    device = [t.to("cuda") for t in pinned]
    torch.cuda.synchronize()
    for bufs in (pinned, device):
        c = N.Cloud(ctx, n)
        ctx.check(ctx.L.gca3d_cloud_upload(ctx.h, c.h, C.c_void_p(bufs[0].data_ptr()), C.c_void_p(bufs[1].data_ptr()),
                                           n))
        got = device_arrays(c)
        assert len(c) == n
        np.testing.assert_array_equal(got[0], want[0])
        np.testing.assert_array_equal(got[1], want[1])


@pytest.mark.parametrize("mode", ["in_place", "copy_engine"])
def test_upload_many_matches_single_uploads(ctx, N, golden, mode):
    """One batched call over clouds of mixed sources (pinned, device, pageable, no
    colour, empty) gives the clouds of the single uploads, in both upload modes."""
    torch = pytest.importorskip("torch")
    ctx.check(ctx.L.gca3d_set_upload_mode(ctx.h, N.UPLOAD_COPY_ENGINE if mode == "copy_engine" else N.UPLOAD_IN_PLACE))
    xyz, rgb = golden["cloud_xyz"], golden["cloud_rgb"]
    n = len(xyz)
    parts = [(0, n), (0, 1000), (5, 4000), (100, 100), (7, n)]
    pinned = [torch.from_numpy(np.ascontiguousarray(a, np.float32)).pin_memory() for a in (xyz, rgb)]
    device = [t.to("cuda") for t in pinned]
    torch.cuda.synchronize()
    pageable = [np.ascontiguousarray(a, np.float32) for a in (xyz, rgb)]
    srcs = [pinned, device, pageable, pinned, device]
    clouds, xp, rp, cnt, want = [], [], [], [], []
    for k, ((a, b), bufs) in enumerate(zip(parts, srcs)):
        ptr = (lambda t, off: t.data_ptr() + 12 * off) if bufs is not pageable else \
              (lambda t, off: t.ctypes.data + 12 * off)
        with_rgb = k != 1
        clouds.append(N.Cloud(ctx, max(b - a, 1)))
        xp.append(ptr(bufs[0], a))
        rp.append(ptr(bufs[1], a) if with_rgb else None)
        cnt.append(b - a)
        ref = ctx.cloud_from(xyz[a:b], rgb[a:b] if with_rgb else None, capacity=max(b - a, 1))
        want.append(ref.download())
    N.upload_many(ctx, clouds, xp, rp, cnt)
    ctx.check(ctx.L.gca3d_set_upload_mode(ctx.h, N.UPLOAD_IN_PLACE))
    for c, w, m in zip(clouds, want, cnt):
        assert len(c) == m
        d = c.download()
        np.testing.assert_array_equal(d["xyz"], w["xyz"])
        np.testing.assert_array_equal(d["rgb"], w["rgb"])
    assert ctx.L.gca3d_set_upload_mode(ctx.h, 7) == N.ERR_INVALID_VALUE


def test_upload_many_repeated_cloud_keeps_call_order(ctx, N, golden):
    """A cloud named several times in one call ends with its last entry, whatever the
    sources of the entries (in place or staged)."""
    torch = pytest.importorskip("torch")
    xyz, rgb = golden["cloud_xyz"], golden["cloud_rgb"]
    n = len(xyz)
    pinned = [torch.from_numpy(np.ascontiguousarray(a, np.float32)).pin_memory() for a in (xyz, rgb)]
    pageable = [np.ascontiguousarray(a, np.float32) for a in (xyz, rgb)]
    pin = lambda off: (pinned[0].data_ptr() + 12 * off, pinned[1].data_ptr() + 12 * off)
    page = lambda off: (pageable[0].ctypes.data + 12 * off, pageable[1].ctypes.data + 12 * off)
    # (source, first point, count) per entry, all into one cloud; the last entry wins
    for seq in ([(pin, 0, 500), (page, 10, 300)], [(page, 10, 300), (pin, 0, 500)],
                [(pin, 0, 500), (pin, 20, 200)], [(pin, 0, 500), (page, 3, 50), (pin, 40, 400)]):
        c = N.Cloud(ctx, n)
        xp, rp, cnt = [], [], []
        for src, off, m in seq:
            a, b = src(off)
            xp.append(a)
            rp.append(b)
            cnt.append(m)
        N.upload_many(ctx, [c] * len(seq), xp, rp, cnt)
        _, off, m = seq[-1]
        ref = ctx.cloud_from(xyz[off:off + m], rgb[off:off + m])
        want, got = ref.download(), c.download()
        assert len(c) == m
        np.testing.assert_array_equal(got["xyz"], want["xyz"])
        np.testing.assert_array_equal(got["rgb"], want["rgb"])


def test_bounds_true_max(ctx, golden):
    for pts in (golden["cloud_xyz"], golden.voxel_input("neg05")[0]):
        c = ctx.cloud_from(pts)
        mn, mx = np.zeros(3, np.float32), np.zeros(3, np.float32)
        ctx.check(ctx.L.gca3d_bounds(ctx.h, c.h, mn.ctypes.data, mx.ctypes.data))
        np.testing.assert_array_equal(mn, pts.min(0))
        np.testing.assert_array_equal(mx, pts.max(0))  # the reference's FLT_MIN start is not reproduced


def test_transform_bit_exact(ctx, golden):
    c = ctx.cloud_from(golden.patch_xyz[:3000])
    T = golden["transform_T"].astype(np.float64)
    ctx.check(ctx.L.gca3d_transform(ctx.h, c.h, T.ctypes.data))
    np.testing.assert_array_equal(c.download()["xyz"], golden["transform_out"])


# --------------------------------------------------------------------------- #
# voxel downsample: bit-exact
# --------------------------------------------------------------------------- #
def voxel_gpu(ctx, xyz, rgb, v):
    c = ctx.cloud_from(xyz, rgb)
    out = ctx.cloud(c.capacity)
    ctx.check(ctx.L.gca3d_voxel_downsample(ctx.h, c.h, float(v), out.h))
    return out.download()


@pytest.mark.parametrize("tag", ["v05", "v02", "neg05", "dup", "one"])
def test_voxel_golden(ctx, golden, tag):
    xyz, rgb = golden.voxel_input(tag)
    d = voxel_gpu(ctx, xyz, rgb, golden[f"voxel_{tag}_size"])
    np.testing.assert_array_equal(d["xyz"], golden[f"voxel_{tag}_xyz"])
    np.testing.assert_array_equal(d["rgb"], golden[f"voxel_{tag}_rgb"])


@pytest.mark.parametrize("v", [0.04, 0.02, 0.01, 0.005])
def test_voxel_full_size_vs_oracle(ctx, orc, room, v):
    xyz, rgb = room
    d = voxel_gpu(ctx, xyz, rgb, v)
    ox, oc, cnt, _ = orc.voxel_downsample(xyz, rgb, v)
    np.testing.assert_array_equal(d["xyz"], ox)
    np.testing.assert_array_equal(d["rgb"], oc)


@pytest.mark.parametrize("n", [1, 15, 16, 17, 1023, 16 * 1024, 16 * 1024 + 1, 13 * 16 * 1024, 13 * 16 * 1024 + 1])
@pytest.mark.parametrize("extent,voxel", [(2.0, 0.05), (900.0, 0.002), (900.0, 0.0005)])
def test_voxel_sort_sizes_and_key_widths_vs_oracle(ctx, orc, n, extent, voxel):
    """both sorts around the line between them (13 x 16 x 1024 points) and at the edges of a
    block's share, with keys of 18, 57 (sorted in two parts beside the index) and 63 bits; a
    tenth of the points are repeated, so the order within a voxel shows"""
    rng = np.random.default_rng(n)
    xyz = (rng.random((n, 3)) * extent).astype(np.float32)
    xyz[rng.integers(0, n, n // 10)] = xyz[rng.integers(0, n, n // 10)]
    rgb = rng.random((n, 3)).astype(np.float32)
    src, out = ctx.cloud_from(xyz, rgb), ctx.cloud(n)
    ctx.check(ctx.L.gca3d_voxel_downsample(ctx.h, src.h, voxel, out.h))
    d = out.download()
    ox, oc, _, _ = orc.voxel_downsample(xyz, rgb, voxel)
    np.testing.assert_array_equal(d["xyz"], ox)
    np.testing.assert_array_equal(d["rgb"], oc)


@pytest.mark.parametrize("per", [1, 2, 7, 8, 9, 10, 16, 17, 25, 1000])
def test_voxel_sums_of_every_length(ctx, orc, per):
    """voxels of exactly `per` points (and one fewer, every third), whose points are far apart in the cloud: the
    sums in index order, bit for bit"""
    rng = np.random.default_rng(per)
    cells = np.stack(np.meshgrid(*[np.arange(4)] * 3), -1).reshape(-1, 3)
    counts = np.where(np.arange(64) % 3 == 0, max(per - 1, 1), per)
    xyz = np.repeat(cells, counts, 0) * 0.1 + 0.02 + 0.06 * rng.random((counts.sum(), 3))
    xyz = np.concatenate([[[0.0, 0.0, 0.0]], xyz]).astype(np.float32) # the origin of the voxels
    xyz[1:] = xyz[1:][rng.permutation(len(xyz) - 1)]
    rgb = rng.random(xyz.shape).astype(np.float32)
    src, out = ctx.cloud_from(xyz, rgb), ctx.cloud(len(xyz))
    ctx.check(ctx.L.gca3d_voxel_downsample(ctx.h, src.h, 0.1, out.h))
    d = out.download()
    ox, oc, _, _ = orc.voxel_downsample(xyz, rgb, 0.1)
    assert len(ox) == 64
    np.testing.assert_array_equal(d["xyz"], ox)
    np.testing.assert_array_equal(d["rgb"], oc)


def test_voxel_empty_and_invalid(ctx, N):
    c = ctx.cloud(16)
    out = ctx.cloud(16)
    ctx.check(ctx.L.gca3d_voxel_downsample(ctx.h, c.h, 0.05, out.h))
    assert len(out) == 0
    assert ctx.L.gca3d_voxel_downsample(ctx.h, c.h, 0.0, out.h) == N.ERR_INVALID_VALUE
    assert ctx.L.gca3d_voxel_downsample(ctx.h, c.h, -1.0, out.h) == N.ERR_INVALID_VALUE
    small = ctx.cloud(4)
    assert ctx.L.gca3d_voxel_downsample(ctx.h, c.h, 0.05, small.h) == N.ERR_CAPACITY


def test_voxel_extent_beyond_key_range(ctx, N):
    pts = np.array([[0, 0, 0], [1.0e5, 0, 0]], np.float32)
    c = ctx.cloud_from(pts)
    out = ctx.cloud(2)
    assert ctx.L.gca3d_voxel_downsample(ctx.h, c.h, 0.001, out.h) == N.ERR_CAPACITY


# --------------------------------------------------------------------------- #
# nearest neighbour and radius lists: bit-exact
# --------------------------------------------------------------------------- #
def nn_gpu(ctx, q, r, radius):
    cq, cr = ctx.cloud_from(q), ctx.cloud_from(r)
    buf = ctx.alloc(4 * len(q))
    ctx.check(ctx.L.gca3d_nn_search(ctx.h, cq.h, cr.h, float(radius), buf.ptr))
    return buf.read(np.int32, len(q))


def test_nn_golden(ctx, golden, orc):
    idx = nn_gpu(ctx, golden["nn_q"], golden.nn_r, golden["nn_radius"])
    np.testing.assert_array_equal(idx, golden["nn_idx"])


def test_nn_exact_ties_min_index(ctx, golden, orc):
    q, r, rad = golden["nntie_q"], golden["nntie_r"], float(golden["nntie_radius"])
    idx = nn_gpu(ctx, q, r, rad)
    np.testing.assert_array_equal(idx, orc.nn_search(q, r, rad, tie=orc.TIE_MIN_INDEX))


def test_nn_full_size_vs_oracle(ctx, orc, room):
    xyz = room[0]
    rng = np.random.default_rng(5)
    q = (xyz[:100_000] + rng.normal(scale=0.01, size=(100_000, 3))).astype(np.float32)
    r = xyz[100_000:]
    for rad in (0.015, 0.05):
        idx = nn_gpu(ctx, q, r, rad)
        np.testing.assert_array_equal(idx, orc.nn_search(q, r, rad, tie=orc.TIE_MIN_INDEX))


@pytest.mark.parametrize("n", [17, 16 * 1024 + 1, 13 * 16 * 1024, 13 * 16 * 1024 + 1])
@pytest.mark.parametrize("extent,radius", [(2.0, 0.1), (800.0, 0.0009)])
def test_nn_grid_sort_sizes(ctx, n, extent, radius):
    """grids on both sides of the sorts' line, with short keys and with keys
    that fill a word, against all distances in FP32"""
    rng = np.random.default_rng(n)
    r = (rng.random((n, 3)) * extent).astype(np.float32)
    q = (r[rng.integers(0, n, 300)] + rng.normal(size=(300, 3)) * radius * 0.3).astype(np.float32)
    d2 = np.zeros((len(q), n), np.float32)
    for k in range(3):
        d = q[:, k, None] - r[None, :, k]
        d2 += d * d
    best = d2.argmin(1)
    want = np.where(d2[np.arange(len(q)), best] < np.float32(radius) * np.float32(radius), best, -1)
    assert (want >= 0).mean() > 0.5
    np.testing.assert_array_equal(nn_gpu(ctx, q, r, radius), want)


def test_nn_queries_outside_grid(ctx, orc):
    r = np.random.default_rng(1).random((1000, 3)).astype(np.float32)
    q = np.array([[50, 50, 50], [-50, 0, 0], [0.5, 0.5, 0.5], [np.nan, 0, 0]], np.float32)
    idx = nn_gpu(ctx, q, r, 0.1)
    assert idx[0] == -1 and idx[1] == -1 and idx[3] == -1
    assert idx[2] == orc.nn_search(q[2:3], r, 0.1)[0]


def radius_gpu(ctx, q, r, radius, grid_min):
    cq, cr = ctx.cloud_from(q), ctx.cloud_from(r)
    n = len(q)
    counts, starts = ctx.alloc(4 * n), ctx.alloc(4 * n)
    cap = 256 * n
    lst = ctx.alloc(4 * cap)
    total = C.c_int64()
    gm = None if grid_min is None else np.ascontiguousarray(grid_min, np.float32)
    ctx.check(ctx.L.gca3d_radius_search(ctx.h, cq.h, cr.h, float(radius), None if gm is None else gm.ctypes.data,
                                        counts.ptr, starts.ptr, lst.ptr, cap, C.byref(total)))
    return counts.read(np.int32, n), starts.read(np.int32, n), lst.read(np.int32, total.value)


@pytest.mark.parametrize("given", [True, False])
def test_radius_lists_golden_order(ctx, golden, given):
    pts = golden.patch_xyz
    c, s, l = radius_gpu(ctx, pts, pts, golden["radius_r"], golden["radius_grid_min"] if given else None)
    np.testing.assert_array_equal(c, golden["radius_counts"])
    np.testing.assert_array_equal(s, golden["radius_starts"])
    np.testing.assert_array_equal(l, golden["radius_list"])


def test_radius_capacity_error(ctx, golden, N):
    pts = golden.patch_xyz
    cq = ctx.cloud_from(pts)
    n = len(pts)
    counts, starts, lst = ctx.alloc(4 * n), ctx.alloc(4 * n), ctx.alloc(64)
    total = C.c_int64()
    st = ctx.L.gca3d_radius_search(ctx.h, cq.h, cq.h, float(golden["radius_r"]), None, counts.ptr, starts.ptr,
                                   lst.ptr, 16, C.byref(total))
    assert st == N.ERR_CAPACITY and total.value == golden["radius_list"].size


# --------------------------------------------------------------------------- #
# normals and colour gradients: tolerance vs FP64
# --------------------------------------------------------------------------- #
@pytest.fixture(scope="module")
def room_v01(orc, room):
    vx, vc, _, _ = orc.voxel_downsample(room[0], room[1], 0.01)
    return vx, vc


def normals_gpu(ctx, xyz, radius, max_nn=0):
    c = ctx.cloud_from(xyz)
    ctx.check(ctx.L.gca3d_estimate_normals(ctx.h, c.h, float(radius), int(max_nn)))
    return c.download(xyz=False, rgb=False, normals=True)["normals"]


@pytest.mark.parametrize("max_nn", [0, 30])
def test_normals_vs_f64(ctx, orc, room_v01, max_nn):
    xyz = room_v01[0]
    n = normals_gpu(ctx, xyz, 0.02, max_nn)
    ref = orc.normals_f64(xyz, 0.02, max_nn)
    zero_g, zero_r = np.linalg.norm(n, axis=1) == 0, np.linalg.norm(ref, axis=1) == 0
    np.testing.assert_array_equal(zero_g, zero_r)
    ok = ~zero_r
    err = angle_err(n[ok].astype(np.float64), ref[ok])
    # FP32 moments and closed form (Newton-refined smallest eigenvalue); the points
    # whose relative eigenvalue gap is below 1e-3 come from the FP64 pass.  Just above
    # that gap the FP32 covariance's own rounding (a few eps of its largest entry)
    # bounds the angle at about 1e-6 / gap.  The sign follows n_z <= 0.
    assert np.median(err) < 1e-6, np.percentile(err, [50, 99, 100])
    assert np.percentile(err, 99) < 1e-4, np.percentile(err, [50, 99, 100])
    assert err.max() < 2e-3, np.percentile(err, [50, 99, 100])
    sign_ok = (n[ok, 2] <= 0) | (np.abs(n[ok, 2]) < 1e-6)
    assert sign_ok.all()
    np.testing.assert_allclose(np.linalg.norm(n[ok], axis=1), 1.0, atol=1e-5)


@pytest.mark.parametrize("max_nn", [3, 31, 32, 33, 64])
@pytest.mark.parametrize("density", [300, 3000])
def test_capped_normals_vs_f64(ctx, max_nn, density):
    """neighbourhoods around and far above the cap, within the selection pass's shared list
    (256) and beyond it; repeated points make ties that the index decides.  The FP64 normal of
    the max_nn nearest (FP32 distance, then index) is defined up to the gap between its two
    smallest eigenvalues: FP32 sums of a few dozen terms (about 30 roundings of 2^-24 of the
    largest entry) turn it by at most 2e-6 / relative gap, and a repeated triple (gap zero)
    has none"""
    rng = np.random.default_rng(density + max_nn)
    uv = rng.random((density, 2)) * 0.1
    xyz = np.stack([uv[:, 0], uv[:, 1], 0.5 * uv[:, 0] ** 2 + 0.02 * rng.random(density)], 1).astype(np.float32)
    xyz = np.concatenate([xyz, xyz[:: 7]])
    radius = np.float32(0.04)
    d2 = np.zeros((len(xyz), len(xyz)), np.float32)
    for k in range(3):
        d = xyz[None, :, k] - xyz[:, None, k]
        d2 += d * d
    near = np.argsort(d2, axis=1, kind="stable")[:, :max_nn]
    inside = np.take_along_axis(d2, near, 1) < radius * radius
    assert inside.all(1).mean() > 0.9
    n = normals_gpu(ctx, xyz, radius, max_nn).astype(np.float64)
    off = xyz[near].astype(np.float64) - xyz[:, None].astype(np.float64)
    w = inside[..., None] / inside.sum(1)[:, None, None]
    mu = (off * w).sum(1)
    cov = np.einsum("nki,nkj->nij", off * w, off) - mu[:, :, None] * mu[:, None, :]
    val, vec = np.linalg.eigh(cov)
    gap = (val[:, 1] - val[:, 0]) / np.maximum(val[:, 2] - val[:, 0], 1e-30)
    ok = (inside.sum(1) >= 3) & (gap > 1e-5)
    assert ok.mean() > 0.5 # the repeated points of a triple have no normal
    err = np.linalg.norm(np.cross(n[ok], vec[ok][:, :, 0]), axis=1)
    assert (err <= 2e-6 / gap[ok]).all(), (err * gap[ok]).max()


@pytest.mark.parametrize("near", [225, 255, 256, 257, 289, 480, 481, 2000])
@pytest.mark.parametrize("max_nn", [1, 3, 30, 64])
@pytest.mark.parametrize("order", ["random", "far_first"])
def test_capped_selection_around_its_list(ctx, near, max_nn, order):
    """neighbourhoods (one group of points, every point with all the others in its radius)
    around the sizes at which the selection's list of 256 keys is filled and cut back, and far
    above; the points in random order and with the distances to the first falling.  The kept
    set decides the normal, so it must be the FP64 normal of the max_nn nearest (FP32
    distance, then index) within 2e-6 / relative gap of its two smallest eigenvalues, as above"""
    rng = np.random.default_rng(near + max_nn)
    uv = (rng.random((near, 2)) - 0.5) * 0.02
    xyz = np.stack([uv[:, 0], uv[:, 1], 3.0 * uv[:, 0] ** 2 + 0.004 * rng.random(near)], 1).astype(np.float32)
    if order == "far_first":
        xyz = xyz[np.argsort(-((xyz - xyz[0]) ** 2).sum(1))]
    radius = np.float32(0.06)
    d2 = np.zeros((near, near), np.float32)
    for k in range(3):
        d = xyz[None, :, k] - xyz[:, None, k]
        d2 += d * d
    assert (d2 < radius * radius).all()
    kept = np.argsort(d2, axis=1, kind="stable")[:, :max_nn]
    n = normals_gpu(ctx, xyz, radius, max_nn).astype(np.float64)
    if max_nn < 3:
        assert not n.any() # fewer than three points have no normal
        return
    off = xyz[kept].astype(np.float64) - xyz[:, None].astype(np.float64)
    mu = off.mean(1)
    cov = np.einsum("nki,nkj->nij", off, off) / max_nn - mu[:, :, None] * mu[:, None, :]
    val, vec = np.linalg.eigh(cov)
    gap = (val[:, 1] - val[:, 0]) / np.maximum(val[:, 2] - val[:, 0], 1e-30)
    ok = gap > 1e-5
    assert ok.mean() > 0.5
    err = np.linalg.norm(np.cross(n[ok], vec[ok][:, :, 0]), axis=1)
    assert (err <= 2e-6 / gap[ok]).all(), (err * gap[ok]).max()


def test_capped_normals_cost_grows_with_the_neighbourhood(ctx):
    """a cap of 30 with about 200 and 400 neighbours a point, either side of the selection's
    list: twice the candidates take a few times as long (2.2 measured), not tens of times"""
    import time

    rng = np.random.default_rng(5)
    n = 60_000
    c = ctx.cloud_from(np.stack([rng.random(n), rng.random(n), 0.002 * rng.random(n)], 1).astype(np.float32))

    def best(near):
        radius = float(np.sqrt(near / (np.pi * n)))
        times = []
        for _ in range(6):
            t0 = time.perf_counter()
            ctx.check(ctx.L.gca3d_estimate_normals(ctx.h, c.h, radius, 30)) # waits for its result
            times.append(time.perf_counter() - t0)
        return min(times)

    assert best(400) < 5.0 * best(200)


def test_degenerate_normals_vs_f64(ctx, orc):
    """Points on thin noisy lines: the two smallest eigenvalues of every
    neighbourhood are close, so the FP32 pass queues them and every normal comes
    from the FP64 pass.  Where the gap is resolvable and well inside the FP32
    pass's 1e-3 threshold (relative gap of the two smallest eigenvalues between
    1e-7 and 3e-4) the normal is determined to about 1e-16 / gap and must match the
    oracle's FP64 sweeps."""
    cKDTree = pytest.importorskip("scipy.spatial").cKDTree

    rng = np.random.default_rng(3)
    lines = []
    for _ in range(20):
        o = rng.uniform(-1.0, 1.0, 3)
        d = rng.normal(size=3)
        d /= np.linalg.norm(d)
        t = rng.uniform(0.0, 0.5, 300)
        lines.append(o + t[:, None] * d + rng.normal(size=(300, 3)) * 2e-4)
    xyz = np.concatenate(lines).astype(np.float32)
    n = normals_gpu(ctx, xyz, 0.02)
    ref = orc.normals_f64(xyz, 0.02, 0)
    x64 = xyz.astype(np.float64)
    gap = np.full(len(xyz), np.nan)
    for i, nb in enumerate(cKDTree(x64).query_ball_point(x64, 0.0199)):
        if len(nb) >= 3:
            ev = np.linalg.eigvalsh(np.cov(x64[nb].T, bias=True))
            gap[i] = (ev[1] - ev[0]) / (ev[2] - ev[0])
    sel = (gap > 1e-7) & (gap < 3e-4)
    assert sel.sum() > 500
    err = angle_err(n[sel].astype(np.float64), ref[sel])
    assert err.max() < 1e-6, np.percentile(err, [50, 99, 100])


@pytest.mark.parametrize("lines", [1, 30, 140, 420])
def test_degenerate_normals_many_points_vs_f64(ctx, orc, lines):
    """as above for queues that are shorter and longer than the FP64 pass has warps (one point
    each, several, and more than 32 each, so that a warp takes several rounds), with a queue that is
    no multiple of them; same bound"""
    cKDTree = pytest.importorskip("scipy.spatial").cKDTree
    rng = np.random.default_rng(lines)
    per = 301
    o = rng.uniform(-1.0, 1.0, (lines, 1, 3)) * (lines / 20 + 1) ** (1 / 3)
    d = rng.normal(size=(lines, 1, 3))
    d /= np.linalg.norm(d, axis=2, keepdims=True)
    t = rng.uniform(0.0, 0.5, (lines, per, 1))
    xyz = (o + t * d + rng.normal(size=(lines, per, 3)) * 2e-4).reshape(-1, 3).astype(np.float32)
    n = normals_gpu(ctx, xyz, 0.02)
    ref = orc.normals_f64(xyz, 0.02, 0)
    x64 = xyz.astype(np.float64)
    some = rng.permutation(len(xyz))[:3000]
    gap = np.full(len(xyz), np.nan)
    for i, nb in zip(some, cKDTree(x64).query_ball_point(x64[some], 0.0199)):
        if len(nb) >= 3:
            ev = np.linalg.eigvalsh(np.cov(x64[nb].T, bias=True))
            gap[i] = (ev[1] - ev[0]) / (ev[2] - ev[0])
    sel = (gap > 1e-7) & (gap < 3e-4)
    assert sel.sum() > 25
    err = angle_err(n[sel].astype(np.float64), ref[sel])
    assert err.max() < 1e-6, np.percentile(err, [50, 99, 100])


def test_gradient_vs_f64(ctx, orc, room_v01):
    xyz, rgb = room_v01
    c = ctx.cloud_from(xyz, rgb)
    ctx.check(ctx.L.gca3d_estimate_normals(ctx.h, c.h, 0.02, 0))
    ctx.check(ctx.L.gca3d_color_gradient(ctx.h, c.h, 0.02))
    d = c.download(xyz=False, rgb=False, normals=True, grad=True)
    ref = orc.gradient_f64(xyz, rgb, d["normals"].astype(np.float64), 0.02)
    g = d["grad"].astype(np.float64)
    scale = np.maximum(np.linalg.norm(ref, axis=1), 1e-3)
    rel = np.linalg.norm(g - ref, axis=1) / scale
    assert np.percentile(rel, 99) < 1e-3, np.percentile(rel, [50, 99, 100])
    np.testing.assert_array_equal(np.linalg.norm(g, axis=1) == 0, np.linalg.norm(ref, axis=1) == 0)


def test_gradient_needs_normals(ctx, N, golden):
    c = ctx.cloud_from(golden.patch_xyz, golden.patch_rgb)
    assert ctx.L.gca3d_color_gradient(ctx.h, c.h, 0.05) == N.ERR_INVALID_VALUE


# --------------------------------------------------------------------------- #
# Gauss-Newton system for given correspondences
# --------------------------------------------------------------------------- #
def gn_f64(src, srgb, tx, trgb, tn, tg, nn, lam, orc):
    m = nn >= 0
    p = src[m].astype(np.float64)
    j = nn[m]
    q, n, d = tx[j].astype(np.float64), tn[j].astype(np.float64), tg[j].astype(np.float64)
    Is = orc.intensity(srgb[m]).astype(np.float64)
    It = orc.intensity(trgb[j]).astype(np.float64)
    rg = ((p - q) * n).sum(1)
    proj = p - rg[:, None] * n
    rc = It + ((proj - q) * d).sum(1) - Is
    dt = d - (n * d).sum(1)[:, None] * n
    slg, slc = np.sqrt(np.float32(lam)).astype(np.float64), np.sqrt(np.float32(1) - np.float32(lam)).astype(np.float64)
    Jg = slg * np.concatenate([np.cross(p, n), n], 1)
    Jc = slc * np.concatenate([np.cross(p, dt), dt], 1)
    A = Jg.T @ Jg + Jc.T @ Jc
    b = Jg.T @ (slg * rg) + Jc.T @ (slc * rc)
    r2 = ((slg * rg) ** 2 + (slc * rc) ** 2).sum()
    return A, b, r2


def test_build_gauss_newton(ctx, golden, orc):
    tgt = ctx.cloud_from(golden.patch_xyz, golden.patch_rgb)
    tgt.set_normals(golden["normals"])
    tgt.set_gradients(golden["grad"])
    src = ctx.cloud_from(golden["gn_src_xyz"], golden.gn_src_rgb)
    nn = golden["gn_nn"]
    buf = ctx.alloc(4 * len(nn))
    buf.write(nn)
    jtj, jtr, r2 = np.zeros(36), np.zeros(6), C.c_double()
    ctx.check(ctx.L.gca3d_build_gauss_newton(ctx.h, src.h, tgt.h, buf.ptr, 0.968, jtj.ctypes.data, jtr.ctypes.data,
                                             C.byref(r2)))
    A, b, e = gn_f64(golden["gn_src_xyz"], golden.gn_src_rgb, golden.patch_xyz, golden.patch_rgb, golden["normals"],
                     golden["grad"], nn, 0.968, orc)
    scale = np.abs(A).max()
    assert np.abs(jtj.reshape(6, 6) - A).max() < 1e-5 * scale
    assert np.abs(jtr - b).max() < 1e-5 * np.abs(b).max()
    assert abs(r2.value - e) < 1e-5 * e
    # the reference's FP32 transform_reduce agrees to its own precision
    assert np.abs(golden["gn_jtj"] - A).max() < 1e-3 * scale
    res = ctx.alloc(4 * len(nn))
    ctx.check(ctx.L.gca3d_abs_residual(ctx.h, src.h, tgt.h, buf.ptr, 0.968, res.ptr))
    np.testing.assert_allclose(res.read(np.float32, len(nn)), golden["gn_abs_residual"], rtol=1e-4, atol=1e-6)


def test_build_gauss_newton_rejects_bad_lambda(ctx, golden, N):
    tgt = ctx.cloud_from(golden.patch_xyz, golden.patch_rgb)
    src = ctx.cloud_from(golden["gn_src_xyz"])
    buf = ctx.alloc(4 * 4000)
    jtj, jtr = np.zeros(36), np.zeros(6)
    assert ctx.L.gca3d_build_gauss_newton(ctx.h, src.h, tgt.h, buf.ptr, 1.5, jtj.ctypes.data, jtr.ctypes.data,
                                          None) == N.ERR_INVALID_VALUE
    assert ctx.L.gca3d_build_gauss_newton(ctx.h, src.h, tgt.h, buf.ptr, 0.9, jtj.ctypes.data, jtr.ctypes.data,
                                          None) == N.ERR_INVALID_VALUE  # no normals / gradients


# --------------------------------------------------------------------------- #
# RGB-D frame -> cloud
# --------------------------------------------------------------------------- #
@pytest.fixture(scope="module")
def frames():
    from cuda_3d_gb300 import synth

    return synth.frame_pair(seed=0)


def frame_gpu(ctx, N, depth, bgr, mode, radius=2, ss=3.0, sd=30.0, tmin=0.2, tmax=10.0):
    h, w = depth.shape
    dbuf, cbuf = ctx.alloc(depth.nbytes), ctx.alloc(bgr.nbytes)
    dbuf.write(depth)
    cbuf.write(bgr)
    out = ctx.cloud(h * w)
    di = N.Intrinsics(525.0, 525.0, 319.5, 239.5)
    f = N.Filter(mode, radius, ss, sd)
    ctx.check(ctx.L.gca3d_frame_to_cloud(ctx.h, dbuf.ptr, cbuf.ptr, w, h, C.byref(di), None, None, 0.001, tmin, tmax,
                                         C.byref(f), out.h))
    return out.download()


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_frame_to_cloud_vs_oracle(ctx, N, orc, frames, mode):
    d = frame_gpu(ctx, N, frames.depth0, frames.bgr0, mode)
    ox, oc = orc.make_point_cloud(frames.depth0, frames.bgr0, (525.0, 525.0, 319.5, 239.5), mode=mode, radius=2,
                                  sigma_space=3.0, sigma_depth=30.0, tmin=0.2, tmax=10.0)
    # bit-exact, raster order kept: the filter's exp is evaluated by the same
    # operation sequence on both sides, so even the colour lookups, which sit on
    # pixel boundaries for identity extrinsics, agree
    np.testing.assert_array_equal(d["xyz"], ox)
    np.testing.assert_array_equal(d["rgb"], oc)


@pytest.mark.parametrize("case", ["raw", "adaptive", "fixed", "adaptive_extrinsic", "adaptive_tmin0"])
def test_frame_to_cloud_vs_reference_golden(ctx, N, golden, case):
    """the frame kernel against the reference's own frame helpers
    (cuda_point_cloud_factory.cu:19-187, host build): bit for bit where those use the
    kernel's exp, within the stated ulp bounds where they use the host's expf"""
    di, ci, rot, tr, mode, tmin = golden.frame_case(case)
    depth, bgr = golden["frame_depth"], golden["frame_bgr"]
    h, w = depth.shape
    dbuf, cbuf = ctx.alloc(depth.nbytes), ctx.alloc(bgr.nbytes)
    dbuf.write(depth)
    cbuf.write(bgr)
    out = ctx.cloud(h * w)
    e = N.Extrinsics()
    e.rotation[:] = list(map(float, rot))
    e.translation[:] = list(map(float, tr))
    r, ss, sd = golden.FRAME_FIXED
    f = N.Filter(mode, r, ss, sd)
    ctx.check(ctx.L.gca3d_frame_to_cloud(ctx.h, dbuf.ptr, cbuf.ptr, w, h, C.byref(N.Intrinsics(*di)),
                                         C.byref(N.Intrinsics(*ci)), C.byref(e), 0.001, tmin, 10.0, C.byref(f), out.h))
    d = out.download()
    golden.check_frame(case, d["xyz"], d["rgb"])


def test_frame_tmin_zero_nan_quirk(ctx, N, orc, frames):
    """with tmin = 0 the reference turns isolated zero pixels into NaN points
    (0 / 0 in the filter passes both threshold tests); the build keeps that"""
    d = frame_gpu(ctx, N, frames.depth0, frames.bgr0, 1, tmin=0.0)
    ox, _ = orc.make_point_cloud(frames.depth0, frames.bgr0, (525.0, 525.0, 319.5, 239.5), mode=1, tmin=0.0)
    assert np.isnan(ox).any()
    np.testing.assert_array_equal(d["xyz"], ox)


@pytest.mark.parametrize("w,h", [(1, 1), (33, 5), (65, 9), (129, 3), (2048, 2)])
@pytest.mark.parametrize("mode,radius,sd", [(0, 0, 1.0), (1, 0, 1.0), (2, 0, 30.0), (2, 1, 5.0), (2, 3, 99.0),
                                            (2, 4, 30.0), (2, 5, 300.0), (2, 6, 30.0), (2, 7, 101.0)])
def test_frame_tiles_and_weight_tables_vs_oracle(ctx, N, orc, w, h, mode, radius, sd):
    """ragged tiles, every filter radius, and depth sigmas whose weights end inside the
    range table (5, 30, 99), at its end (101) and beyond it (300)"""
    rng = np.random.default_rng(w * 1000 + h)
    depth = (1500 + 40 * rng.normal(size=(h, w)) + 2000 * (rng.random((h, w)) < 0.3)).astype(np.uint16)
    depth[rng.random((h, w)) < 0.1] = 0
    depth[rng.random((h, w)) < 0.05] = 65535
    bgr = rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
    d = frame_gpu(ctx, N, depth, bgr, mode, radius=radius, sd=sd)
    ox, oc = orc.make_point_cloud(depth, bgr, (525.0, 525.0, 319.5, 239.5), mode=mode, radius=radius,
                                  sigma_space=3.0, sigma_depth=sd, tmin=0.2, tmax=10.0)
    np.testing.assert_array_equal(d["xyz"], ox)
    np.testing.assert_array_equal(d["rgb"], oc)


@pytest.mark.parametrize("w,h", [(64, 11_585), (64, 11_586), (320, 5181), (320, 5182), (65, 20_001)])
def test_tall_frames_vs_oracle(ctx, N, orc, w, h):
    """both forms of the rows' offsets, around the line at which they change (2^27 for the
    height times the row counts, of which there is one per 64 pixels of a row); most pixels
    have no depth"""
    rng = np.random.default_rng(w + h)
    depth = np.where(rng.random((h, w)) < 0.3, rng.integers(1000, 1400, (h, w)), 0).astype(np.uint16)
    depth[h // 3: h // 2] = 0
    bgr = rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
    dbuf, cbuf = ctx.alloc(depth.nbytes), ctx.alloc(bgr.nbytes)
    dbuf.write(depth)
    cbuf.write(bgr)
    cloud = ctx.cloud(h * w)
    intr = (525.0, 525.0, w / 2, h / 2)
    di, f = N.Intrinsics(*intr), N.Filter(0, 0, 3.0, 30.0)
    ctx.check(ctx.L.gca3d_frame_to_cloud(ctx.h, dbuf.ptr, cbuf.ptr, w, h, C.byref(di), None, None, 0.001, 0.2, 10.0,
                                         C.byref(f), cloud.h))
    d = cloud.download()
    ox, oc = orc.make_point_cloud(depth, bgr, intr, mode=0, radius=0, sigma_space=3.0, sigma_depth=30.0, tmin=0.2,
                                  tmax=10.0)
    assert len(ox) > 0.2 * h * w
    np.testing.assert_array_equal(d["xyz"], ox)
    np.testing.assert_array_equal(d["rgb"], oc)


def test_frame_cost_is_linear_in_the_height(ctx, N):
    """a tall frame of 64 x 262,144 pixels against a wide one with as many: alike (the row
    offsets took the tall one eight times as long when every row summed all rows above it)"""
    import time

    def best(w, h):
        d, b = ctx.alloc(2 * w * h), ctx.alloc(3 * w * h)
        d.write(np.full((h, w), 1500, np.uint16))
        b.write(np.zeros((h, w, 3), np.uint8))
        out = ctx.cloud(h * w)
        di, f = N.Intrinsics(525.0, 525.0, w / 2, h / 2), N.Filter(2, 2, 3.0, 30.0)
        times = []
        for _ in range(6):
            t0 = time.perf_counter()
            ctx.check(ctx.L.gca3d_frame_to_cloud(ctx.h, d.ptr, b.ptr, w, h, C.byref(di), None, None, 0.001, 0.2, 10.0,
                                                 C.byref(f), out.h))
            ctx.sync()
            times.append(time.perf_counter() - t0)
        return min(times)

    assert best(64, 262_144) < 4.0 * best(2048, 8192)


# --------------------------------------------------------------------------- #
# radius outlier removal, gather by index, AoS view
# --------------------------------------------------------------------------- #
def _ror(ctx, xyz, rgb, radius, min_nn):
    c = ctx.cloud_from(xyz, rgb)
    out = ctx.cloud(len(xyz))
    ctx.check(ctx.L.gca3d_radius_outlier_removal(ctx.h, c.h, radius, min_nn, out.h))
    return out.download()


def test_radius_outlier_removal_golden(ctx, golden):
    xyz, rgb = golden["cloud_xyz"][:8000], golden["cloud_rgb"][:8000]
    d = _ror(ctx, xyz, rgb, float(golden["ror_radius"]), int(golden["ror_min_nn"]))
    np.testing.assert_array_equal(d["xyz"], golden["ror_xyz"])
    np.testing.assert_array_equal(d["rgb"], golden["ror_rgb"])


@pytest.mark.parametrize("radius,min_nn", [(0.01, 2), (0.02, 8), (0.05, 40)])
def test_radius_outlier_removal_full_size_vs_oracle(ctx, orc, room, radius, min_nn):
    xyz, rgb = room
    d = _ror(ctx, xyz, rgb, radius, min_nn)
    ox, oc = orc.radius_outlier_removal(xyz, rgb, radius, min_nn)
    assert 0 < len(ox) < len(xyz)
    np.testing.assert_array_equal(d["xyz"], ox)
    np.testing.assert_array_equal(d["rgb"], oc)


@pytest.mark.parametrize("extent", [0.3, 3.0, 500.0])
@pytest.mark.parametrize("min_nn", [0, 3, 12])
def test_radius_outlier_removal_row_tables(ctx, extent, min_nn):
    """the direct row table with short and long runs, and the row hash (a set too wide for
    the table), against all distances in FP32"""
    rng = np.random.default_rng(int(extent))
    r, n = 0.01, 4000
    c = (rng.random((250, 3)) * extent).astype(np.float32)
    xyz = (c[rng.integers(0, len(c), n)] + rng.normal(size=(n, 3)) * r * 0.6).astype(np.float32)
    rgb = rng.random((n, 3)).astype(np.float32)
    d2 = np.zeros((n, n), np.float32)
    for k in range(3):
        d = xyz[:, k, None] - xyz[None, :, k]
        d2 += d * d
    keep = (d2 < np.float32(r) * np.float32(r)).sum(1) > min_nn
    assert keep.any() and (min_nn == 0 or not keep.all())
    d = _ror(ctx, xyz, rgb, r, min_nn)
    np.testing.assert_array_equal(d["xyz"], xyz[keep])
    np.testing.assert_array_equal(d["rgb"], rgb[keep])


def test_radius_outlier_removal_invalid(ctx, N, golden):
    c = ctx.cloud_from(golden["cloud_xyz"][:100], golden["cloud_rgb"][:100])
    small = ctx.cloud(10)
    assert ctx.L.gca3d_radius_outlier_removal(ctx.h, c.h, 0.0, 2, c.h) == N.ERR_INVALID_VALUE
    assert ctx.L.gca3d_radius_outlier_removal(ctx.h, c.h, 0.05, 2, small.h) == N.ERR_CAPACITY


def test_cloud_select_and_aos(ctx, N, golden):
    xyz, rgb = golden["cloud_xyz"][:5000], golden["cloud_rgb"][:5000]
    c = ctx.cloud_from(xyz, rgb)
    c.set_normals(golden["normals"][:5000] if len(golden["normals"]) >= 5000 else np.tile([0, 0, 1.0], (5000, 1)))
    idx = np.random.default_rng(0).integers(0, 5000, 777).astype(np.int32)
    out = ctx.cloud(1000)
    ctx.check(ctx.L.gca3d_cloud_select(ctx.h, c.h, idx.ctypes.data, len(idx), out.h))
    d = out.download(normals=True)
    np.testing.assert_array_equal(d["xyz"], xyz[idx])
    np.testing.assert_array_equal(d["rgb"], rgb[idx])
    # an index outside the cloud is reported
    bad = np.array([0, 5000], np.int32)
    assert ctx.L.gca3d_cloud_select(ctx.h, c.h, bad.ctypes.data, 2, out.h) == N.ERR_INVALID_VALUE
    # the 28-byte records of the reference's point_t
    buf = ctx.alloc(28 * 5000)
    nb = ctx.alloc(12 * 5000)
    ctx.check(ctx.L.gca3d_cloud_to_aos(ctx.h, c.h, buf.ptr, nb.ptr))
    raw = buf.read(np.uint8, 28 * 5000).reshape(5000, 28)
    f = raw[:, :24].copy().view(np.float32).reshape(5000, 6)
    np.testing.assert_array_equal(f[:, :3], xyz)
    np.testing.assert_array_equal(f[:, 3:], rgb)
    assert np.all(raw[:, 24] == 1)
