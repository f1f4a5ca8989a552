"""Option values, table shapes and sizes at the edges of what the search entry points accept."""
import numpy as np
import pytest
import torch

import oracle as O
from hashpoint import native, ops, synth

pytestmark = pytest.mark.gpu


def _view(xyz, cam):
    """Device copies and the hash table of a cloud in a view."""
    native.build()
    X, c2w, w2c, K = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (xyz, cam.c2w, cam.w2c, cam.K)]
    sidx, _, table = ops.pts2plane(X, w2c, K, cam.height, cam.width)
    return X, c2w, sidx, table


def _sample(X, c2w, cam, o, sidx, table, **tuning):
    return ops.quick_sampling(X, c2w, cam.fx, cam.fy, cam.cx, cam.cy, cam.width, cam.height, o, sidx, table,
                              tuning=ops.make_tuning(**tuning) if tuning else None)


def _query(X, c2w, cam, o, sidx, table, rays, L=None):
    """quick_query by the product library, or by L."""
    if L is None:
        return ops.quick_query(X, c2w, cam.fx, cam.fy, cam.cx, cam.cy, cam.width, cam.height, o, sidx, table, rays)
    out = torch.empty((len(rays), o.num_point_per_ray), dtype=torch.int32, device="cuda")
    spec = ops.make_camera(c2w=c2w, fx=cam.fx, fy=cam.fy, cx=cam.cx, cy=cam.cy, width=cam.width, height=cam.height)
    rc = L.hp_quick_query_for_nearby_point(X.data_ptr(), len(X), spec, ops.make_options(o), sidx.data_ptr(), len(sidx),
                                           table.data_ptr(), rays.data_ptr(), len(rays), out.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream)
    native.check(rc, "hp_quick_query_for_nearby_point", L)
    return out


@pytest.mark.parametrize("radius", [-0.05, -1e-20, 0.0, float("nan")])
def test_radius_that_keeps_nothing(radius):
    """A candidate is kept when its distance is below the radius: never for one of zero or less."""
    cam = synth.look_at_camera((0.3, 0.2, 4.0), (0, 0, 0), 40, 30, 36.0)
    X, c2w, sidx, table = _view(synth.sphere_cloud(np.random.default_rng(1), 3_000), cam)
    assert (table[:, 1] > 0).any()
    o = synth.Options(kernel_size=3, radius_threshold=radius, num_point_per_ray=16)
    rays = torch.arange(1200, dtype=torch.int32, device="cuda")
    assert (_query(X, c2w, cam, o, sidx, table, rays) == -1).all()
    sp_xyz, pc_idx, sp_t, mask = _sample(X, c2w, cam, o, sidx, table)
    assert not mask.any() and (pc_idx == -1).all() and (sp_t == 0).all() and (sp_xyz == 0).all()


def test_points_a_thousand_away_from_a_sample():
    """The ball query's farthest distance starts at 1e3, so a buffer filled from beyond that replaces slot 0 first."""
    rng = np.random.default_rng(7)
    cam = synth.look_at_camera((0, 0, 0), (1, 0, 0), 32, 24, 20.0)
    z = rng.uniform(2000, 20000, 6000)
    xyz = np.stack([z, rng.uniform(-.8, .8, 6000) * z, rng.uniform(-.6, .6, 6000) * z], 1).astype(np.float32)
    o = synth.Options(kernel_size=3, radius_threshold=3000.0, t_intvl=1000.0, num_sample_points_per_ray=8,
                      num_point_cloud_per_sp=8, sdf2weight_gaussian_alpha=2000.0, sdf2weight_gaussian_gamma=0.3)
    X, c2w, sidx, table = _view(xyz, cam)
    dirs = ops.ray_directions(c2w, cam.fx, cam.fy, cam.cx, cam.cy, 32, 24).cpu().numpy()
    ref = O.quick_sampling(xyz, O.camera_from(cam), o, sidx.cpu().numpy(), table.cpu().numpy(), dirs=dirs)
    assert ref[3].sum() > 3000
    out = _sample(X, c2w, cam, o, sidx, table)
    # the oracle's norm is rounded correctly, the GPU's norm3df within an ulp: a ray may differ only by a decision
    # that close
    bad = ~((out[3].cpu().numpy() == ref[3]).all(-1) & (out[1].cpu().numpy() == ref[1]).all((-1, -2)))
    assert (ref[4].reshape(24, 32)[bad] < 1e-6).all() and bad.sum() <= 7


# (points, image, kernel, radius, row length): cells of 0 to 100 candidates
WINDOWS = [(20_000, (60, 45), 5, 0.03, 256), (30_000, (30, 20), 7, 0.05, 99), (4_000, (9, 7), 31, 0.1, 300),
           (500, (3, 2), 5, 0.5, 64), (2_000, (1, 1), 5, 5.0, 40)]


@pytest.mark.parametrize("n,size,k,radius,cap", WINDOWS)
def test_query_windows_taken_in_rounds(n, size, k, radius, cap):
    """The test library numbers at most 64 candidates at once, as the product does 2^31: the rows are the same."""
    native.build_testing()
    cam = synth.look_at_camera((0.3, 0.2, 4.0), (0, 0, 0), *size, 0.5 * size[0])
    X, c2w, sidx, table = _view(synth.shapes_cloud(np.random.default_rng(n), n), cam)
    o = synth.Options(kernel_size=k, radius_threshold=radius, num_point_per_ray=cap)
    rays = torch.arange(-1, size[0] * size[1] + 1, dtype=torch.int32, device="cuda")
    want = _query(X, c2w, cam, o, sidx, table, rays)
    assert (want >= 0).any()
    assert torch.equal(_query(X, c2w, cam, o, sidx, table, rays, native.testing_lib()), want)


def _sample_by(L, X, c2w, cam, o, sidx, table):
    """quick_sampling by the library L."""
    out = ops.sampling_outputs(cam.height, cam.width, o, "cuda")
    spec = ops.make_camera(c2w=c2w, fx=cam.fx, fy=cam.fy, cx=cam.cx, cy=cam.cy, width=cam.width, height=cam.height)
    ws = torch.empty(L.hp_quick_sampling_workspace_size(len(sidx), cam.height, cam.width), dtype=torch.uint8, device="cuda")
    rc = L.hp_quick_sampling(X.data_ptr(), len(X), spec, ops.make_options(o), sidx.data_ptr(), len(sidx), table.data_ptr(),
                             *[t.data_ptr() for t in out], ws.data_ptr(), len(ws), torch.cuda.current_stream().cuda_stream)
    native.check(rc, "hp_quick_sampling", L)
    return out


def _reversed_buckets(sidx, table):
    """The same buckets, stored last pixel first: rays with two non-empty cells in a window row take the general walk."""
    sidx, h = sidx.cpu().numpy(), table.cpu().numpy().copy()
    out, at = np.full_like(sidx, -1), 0
    for p in np.nonzero(h[:, 1] > 0)[0][::-1]:
        s, c = h[p]
        out[at:at + c] = sidx[s:s + c]
        h[p, 0] = at
        at += c
    return torch.from_numpy(out).cuda(), torch.from_numpy(h).cuda()


def _cloud(kind, n, rng):
    xyz = synth.shapes_cloud(rng, n)
    if kind == "twins":  # every point three times
        xyz = np.repeat(xyz[:n // 3], 3, 0)[rng.permutation(n // 3 * 3)]
    if kind == "lattice":
        xyz = np.round(xyz / 0.004) * 0.004
    return xyz.astype(np.float32)


SHAPED = dict(radius_threshold=0.03)
SLOW = dict(radius_threshold=0.05, sdf2weight_gaussian_gamma=0.05, num_sample_points_per_ray=40, num_point_cloud_per_sp=11)


@pytest.mark.parametrize("kind,n,size,opt", [
    ("shapes", 20_000, (60, 45), SHAPED), ("shapes", 60_000, (40, 31), SHAPED),
    ("shapes", 60_000, (33, 16), dict(kernel_size=2, radius_threshold=0.5)),
    ("shapes", 2_000, (1, 1), dict(radius_threshold=5.0)),
    ("shapes", 3_000, (3, 200), SHAPED), ("shapes", 3_000, (200, 2), dict(kernel_size=4, radius_threshold=0.06)),  # repeated cells
    ("twins", 20_000, (60, 45), SHAPED), ("twins", 60_000, (40, 31), SHAPED), ("twins", 20_000, (61, 40), SLOW),
    ("lattice", 30_000, (97, 61), SHAPED), ("lattice", 90_000, (40, 31), SLOW),
    # mean distances that the quantised sums cannot tell apart, for all rays or for some
    ("shapes", 20_000, (60, 45), dict(SLOW, sdf2weight_gaussian_alpha=0.0005)),
    ("shapes", 20_000, (60, 45), dict(SLOW, sdf2weight_gaussian_alpha=0.005)),
    ("shapes", 9_000, (40, 33), dict(kernel_size=3, radius_threshold=1e-16)),
    ("shapes", 9_000, (40, 33), dict(kernel_size=3, radius_threshold=1e16)),
    ("shapes", 20_000, (60, 45), dict(SHAPED, sdf2weight_gaussian_alpha=0.0)),
    ("shapes", 20_000, (60, 45), dict(SHAPED, sdf2weight_gaussian_alpha=-0.2, sdf2weight_gaussian_gamma=-0.1)),
])
def test_left_rays_by_lists_and_by_the_general_walk(kind, n, size, opt):
    """The test library serves every ray that the fast arithmetic leaves by the general walk, in 64-bit indices, and a table
    in reversed pixel order leaves every ray with two filled cells in a window row: the same bytes three times."""
    native.build_testing()
    T = native.testing_lib()
    cam = synth.look_at_camera((0.3, 0.2, 4.0), (0, 0, 0), *size, 0.5 * max(size))
    X, c2w, sidx, table = _view(_cloud(kind, n, np.random.default_rng(n)), cam)
    sidx[::50] = n + 7  # ids beyond the cloud are skipped
    o = synth.Options(**{"num_point_cloud_per_sp": 8, **opt})
    want = _sample(X, c2w, cam, o, sidx, table)
    turned = _reversed_buckets(sidx, table)
    assert all(torch.equal(a, b) for a, b in zip(_sample(X, c2w, cam, o, *turned), want))
    for s, h in ((sidx, table), turned):
        assert all(torch.equal(a, b) for a, b in zip(_sample_by(T, X, c2w, cam, o, s, h), want))


def test_query_window_beyond_two_to_the_31():
    """961 window cells, all the one bucket of 70 million ids."""
    native.build()
    cam = synth.look_at_camera((0, 0, 4.0), (0, 0, 0), 1, 1, 1.0)
    X = torch.zeros((1, 3), device="cuda")
    sidx = torch.zeros(70_000_000, dtype=torch.int32, device="cuda")
    table = torch.tensor([[0, len(sidx)]], dtype=torch.int32, device="cuda")
    o = synth.Options(kernel_size=31, radius_threshold=1.0, num_point_per_ray=20)
    rows = _query(X, torch.from_numpy(cam.c2w).cuda(), cam, o, sidx, table, torch.zeros(3, dtype=torch.int32, device="cuda"))
    assert (rows == 0).all()


def _time(f, runs=9):
    """Median microseconds of a call on the device."""
    f()
    t = []
    for _ in range(runs):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        f()
        b.record()
        b.synchronize()
        t.append(1e3 * a.elapsed_time(b))
    return sorted(t)[runs // 2]


def test_query_stops_at_a_cells_last_id():
    """A cell gives at most 32 ids: buckets a hundred times as deep cost no more (they did cost that much more)."""
    native.build()
    cam = synth.look_at_camera((0, 0, 4.0), (0, 0, 0), 4, 4, 4.0)
    X, c2w = torch.zeros((1, 3), device="cuda"), torch.from_numpy(cam.c2w).cuda()
    o = synth.Options(kernel_size=5, radius_threshold=5.0, num_point_per_ray=1024)
    rays = torch.arange(16, dtype=torch.int32, device="cuda").repeat(4)

    def call(n):
        sidx = torch.zeros(16 * n, dtype=torch.int32, device="cuda")
        table = torch.stack([torch.arange(16, device="cuda") * n, torch.full((16,), n, device="cuda")], 1).int()
        assert ((_query(X, c2w, cam, o, sidx, table, rays) == 0).sum(1) == 25 * 32).all()
        return _time(lambda: _query(X, c2w, cam, o, sidx, table, rays))

    assert call(100_000) < 4 * call(1_000)


def test_query_short_lists_fill_the_chip():
    """592 rays of 25 buckets of 1,000 ids, none near: on 148 SMs they take little longer than one (with eight rays a warp
    one after another they took eight times as long)."""
    native.build()
    cam = synth.look_at_camera((0, 0, 4.0), (0, 0, 0), 4, 4, 4.0)
    X, c2w = torch.tensor([[50.0, 50.0, 0.0]], device="cuda"), torch.from_numpy(cam.c2w).cuda()
    o = synth.Options(kernel_size=5, radius_threshold=0.1, num_point_per_ray=8)
    sidx = torch.zeros(16_000, dtype=torch.int32, device="cuda")
    table = torch.stack([torch.arange(16, device="cuda") * 1000, torch.full((16,), 1000, device="cuda")], 1).int()

    def call(n):
        rays = torch.full((n,), 5, dtype=torch.int32, device="cuda")
        assert (_query(X, c2w, cam, o, sidx, table, rays) == -1).all()
        return _time(lambda: _query(X, c2w, cam, o, sidx, table, rays))

    assert call(592) < 3 * call(1)


def test_query_long_and_short_lists_agree():
    """Either side of the list length from which a warp serves eight rays: the same rows."""
    cam = synth.look_at_camera((0.3, 0.2, 4.0), (0, 0, 0), 400, 330, 360.0)
    X, c2w, sidx, table = _view(synth.shapes_cloud(np.random.default_rng(3), 60_000), cam)
    o = synth.Options(kernel_size=3, radius_threshold=0.02, num_point_per_ray=12)
    rays = torch.randperm(400 * 330, device="cuda")[:(1 << 17) + 3].int()
    long = _query(X, c2w, cam, o, sidx, table, rays)
    assert (long >= 0).any()
    for a, b in ((0, (1 << 17) - 1), (4, 5), (1 << 17, (1 << 17) + 3)):
        assert torch.equal(_query(X, c2w, cam, o, sidx, table, rays[a:b].contiguous()), long[a:b])


@pytest.mark.parametrize("kind,opt", [("twins", {}), ("lattice", {}), ("shapes", dict(sdf2weight_gaussian_alpha=0.0001))])
def test_ties_cost_little(kind, opt):
    """Equal distances (repeated or lattice points) and close mean distances leave most rays to exact arithmetic: at most
    three times the time of a cloud without them (a walk of its own for each such ray: six times)."""
    cam = synth.look_at_camera((0.3, 0.2, 4.0), (0, 0, 0), 400, 400, 555.0)

    def call(kind, **opt):
        X, c2w, sidx, table = _view(_cloud(kind, 300_000, np.random.default_rng(5)), cam)
        o = synth.Options(radius_threshold=0.016, num_sample_points_per_ray=8, num_point_cloud_per_sp=8, **opt)
        return _time(lambda: _sample(X, c2w, cam, o, sidx, table))

    assert call(kind, **opt) < 3 * call("shapes")


def test_a_window_that_cannot_be_listed_is_not_walked_twice():
    """One pixel of 50,000 points, its bucket in every window cell: the list made from the cells ends once it is full, so the
    ray takes no longer than its general walk, which for one sample passes over all of it once."""
    native.build_testing()
    T = native.testing_lib()
    cam = synth.look_at_camera((0.3, 0.2, 4.0), (0, 0, 0), 1, 1, 0.5)
    X, c2w, sidx, table = _view(synth.shapes_cloud(np.random.default_rng(2), 50_000), cam)
    o = synth.Options(radius_threshold=5.0, num_sample_points_per_ray=1, num_point_cloud_per_sp=8)
    walk = lambda: _sample_by(T, X, c2w, cam, o, sidx, table)
    here = lambda: _sample(X, c2w, cam, o, sidx, table)
    assert all(torch.equal(a, b) for a, b in zip(here(), walk()))
    assert _time(here, 5) < 1.3 * _time(walk, 5)
