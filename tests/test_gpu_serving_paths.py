"""The sampling kernel's paths against one another, bit for bit.

A ray is served by 8 lanes, by a whole warp, or -- where its window's buckets
do not follow one another in the sorted ids, its list overflows or a decision
is too close for the fast arithmetic -- by the general walk.  Storing the same
buckets in reversed pixel order sends every ray with two non-empty cells in a
window row (so not kernel_size 1) to the general walk, so each scene is sampled with both tables and
with heavy windows from "every ray" to "none".
"""
import numpy as np
import pytest
import torch

from hashpoint import native, ops, synth

pytestmark = pytest.mark.gpu


EYE = (0.3, 0.2, 4.0)


def _reversed_buckets(sidx, table):
    """The same buckets, stored last pixel first."""
    sidx, h = sidx.cpu().numpy(), table.cpu().numpy().copy()
    out, at = np.full_like(sidx, -1), 0
    for p in np.nonzero(h[:, 1] > 0)[0][::-1]:
        s, c = h[p]
        out[at:at + c] = sidx[s:s + c]
        h[p, 0] = at
        at += c
    return torch.from_numpy(out).cuda(), torch.from_numpy(h).cuda()


def _scene(kind, n, W, H, rng):
    if kind == "plane":  # a tilted plane and a parallel one behind it: many bins, several samples a ray
        u, v = rng.uniform(-1.2, 1.2, n), rng.uniform(-1.0, 1.0, n)
        z = 0.8 * u + 0.15 * rng.integers(0, 3, n)
        xyz = np.stack([u, v, z], 1).astype(np.float32)
    elif kind == "twins":  # every point three times: equal distances everywhere
        xyz = synth.sphere_cloud(rng, n // 3)
        xyz = np.concatenate([xyz, xyz, xyz])[rng.permutation(3 * len(xyz))]
    elif kind == "pile":  # buckets far above 48 entries
        xyz = synth.sphere_cloud(rng, n, noise=0.05) * 0.3
    elif kind == "rings":  # a ninth point as near to each pixel's ray as the nearest of eight, but for a part in 2^13 or less
        d = np.stack([(np.arange(W * H) % W + 0.5 - W / 2) / (0.9 * W), (np.arange(W * H) // W + 0.5 - H / 2) / (0.9 * W),
                      np.ones(W * H)], 1) @ synth.look_at_camera(EYE, (0, 0, 0), W, H, 0.9 * W).c2w[:3, :3].T.astype(np.float64)
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        a = np.cross(d, [0.3, 0.5, 0.8])
        a /= np.linalg.norm(a, axis=1, keepdims=True)
        rings = n // (W * H)
        phi = rng.uniform(0, 2 * np.pi, (rings, W * H, 1))
        rho = 0.0025 * (1 + 0.05 * np.array([3, 5, 1, 7, 2, 4, 0, 6]))  # the first eight well apart,
        later = rho.min() * (1 + 0.07 * np.arange(rings - 8))  # the later ones next to the least, or apart
        rho = np.concatenate([rho, later])[:, None, None] * np.ones((1, W * H, 1))
        rho[8] *= 1 + np.linspace(0, 2.0 ** -13, W * H)[:, None]
        xyz = (np.asarray(EYE) + 4 * d + rho * (np.cos(phi) * a + np.sin(phi) * np.cross(d, a))).reshape(-1, 3)
    else:
        xyz = synth.shapes_cloud(rng, n)
    cam = synth.look_at_camera(EYE, (0, 0, 0), W, H, 0.9 * W)
    return xyz.astype(np.float32), cam


@pytest.mark.parametrize("kind,n,W,H,opt", [
    ("plane", 30_000, 97, 61, dict(kernel_size=5, radius_threshold=0.05)),
    # slow transmittance: up to S samples a ray, odd S and P
    ("plane", 30_000, 97, 61, dict(kernel_size=4, radius_threshold=0.05, sdf2weight_gaussian_gamma=0.05,
                                   num_sample_points_per_ray=7, num_point_cloud_per_sp=3)),
    ("plane", 9_000, 40, 33, dict(kernel_size=3, radius_threshold=0.1, sdf2weight_gaussian_gamma=0.2, t_intvl=0.003,
                                  num_sample_points_per_ray=5, num_point_cloud_per_sp=12)),
    # mean distances that the quantised sums cannot tell apart, and ones they can
    ("plane", 9_000, 40, 33, dict(kernel_size=3, radius_threshold=0.1, sdf2weight_gaussian_alpha=0.0005)),
    ("plane", 9_000, 40, 33, dict(kernel_size=3, radius_threshold=0.1, sdf2weight_gaussian_alpha=0.02)),
    ("twins", 20_000, 65, 49, dict(kernel_size=5, radius_threshold=0.04, num_point_cloud_per_sp=8)),
    # distances around the closeness that sends a ray to the general walk
    ("rings", 9 * 200 * 150, 200, 150, dict(kernel_size=2, radius_threshold=0.005)),
    ("rings", 11 * 200 * 150, 200, 150, dict(kernel_size=2, radius_threshold=0.005)),
    ("pile", 60_000, 40, 31, dict(kernel_size=5, radius_threshold=0.03, num_point_cloud_per_sp=8)),
    ("pile", 60_000, 33, 16, dict(kernel_size=2, radius_threshold=0.5, num_point_cloud_per_sp=8)),
    ("shapes", 40_000, 160, 120, dict(kernel_size=1, radius_threshold=0.02, num_point_cloud_per_sp=4)),
    ("shapes", 3, 5, 1, dict(kernel_size=5, radius_threshold=2.0, num_point_cloud_per_sp=1)),
])
def test_paths_agree(kind, n, W, H, opt):
    native.build()
    xyz, cam = _scene(kind, n, W, H, np.random.default_rng(n + W))
    o = synth.Options(**{"num_point_cloud_per_sp": 8, **opt})
    X, c2w, w2c, K = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (xyz, cam.c2w, cam.w2c, cam.K)]
    sidx, _, table = ops.pts2plane(X, w2c, K, H, W)

    def run(ids, h, **tuning):
        out = ops.quick_sampling(X, c2w, cam.fx, cam.fy, cam.cx, cam.cy, W, H, o, ids, h,
                                 tuning=ops.make_tuning(**tuning))
        return [t.cpu().numpy().view(np.uint8) for t in out]

    want = run(*_reversed_buckets(sidx, table))
    for heavy in (0, 1, 40, 4096):
        for stage in (3, 4):
            for a, b in zip(run(sidx, table, heavy_window=heavy, stage_config=stage), want):
                assert np.array_equal(a, b), (heavy, stage)


@pytest.mark.parametrize("kind,n,W,H,k,radius,cap,rays", [
    ("shapes", 20_000, 120, 90, 5, 0.02, 256, 3_001),
    ("pile", 60_000, 40, 31, 5, 0.03, 256, 1_240),   # buckets above the 32 ids a cell gives, rows that overflow
    ("pile", 60_000, 40, 31, 7, 0.03, 30, 333),      # more than 32 window cells, an odd row length
    ("plane", 9_000, 40, 33, 31, 0.3, 101, 100),
    ("plane", 9_000, 40, 33, 1, 0.1, 7, 9),
])
def test_listed_ray_query_vs_oracle(kind, n, W, H, k, radius, cap, rays):
    import oracle as O
    native.build()
    rng = np.random.default_rng(n + k)
    xyz, cam = _scene(kind, n, W, H, rng)
    o = synth.Options(kernel_size=k, radius_threshold=radius, num_point_per_ray=cap)
    X, c2w, w2c, K = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (xyz, cam.c2w, cam.w2c, cam.K)]
    sidx, _, table = ops.pts2plane(X, w2c, K, H, W)
    ids = rng.integers(-2, W * H + 2, rays).astype(np.int32)  # rays off the image give empty rows
    out = ops.quick_query(X, c2w, cam.fx, cam.fy, cam.cx, cam.cy, W, H, o, sidx, table, torch.from_numpy(ids).cuda())
    dirs = ops.ray_directions(c2w, cam.fx, cam.fy, cam.cx, cam.cy, W, H)
    want, _, _ = O.quick_query(xyz, O.camera_from(cam), o, sidx.cpu().numpy(), table.cpu().numpy(), ids,
                               dirs=dirs.cpu().numpy())
    diff = np.nonzero((out.cpu().numpy() != want).any(1))[0]
    # the oracle's norm is rounded correctly, the GPU's norm3df within an ulp: a row may differ only by a point
    # whose distance is that close to the radius
    _, _, margin = O.quick_query(xyz, O.camera_from(cam), o, sidx.cpu().numpy(), table.cpu().numpy(), ids,
                                 dirs=dirs.cpu().numpy())
    assert np.all(margin[diff] < 1e-6) and len(diff) <= max(1, rays // 100)


@pytest.mark.parametrize("rays,S", [(1, 1), (1, 3), (3, 5), (257, 4), (255, 7), (1025, 8), (400, 16), (33, 31)])
@pytest.mark.parametrize("off", [0, 1])
def test_clamp_t_any_shape(rays, S, off):
    native.build()
    g = torch.Generator(device="cuda").manual_seed(rays * 37 + S)
    buf = torch.empty(rays * S + off, device="cuda")
    t = buf[off:].view(rays, S)
    t.copy_(torch.cumsum(torch.rand((rays, S), device="cuda", generator=g) * 0.02 - 0.002, 1))
    d = torch.cat([t[:, 1:] - t[:, :-1], torch.full_like(t[:, :1], 0.004)], 1)
    m = ((d < 1e-8) | (d > 2 * torch.tensor(0.004, device="cuda"))).float()
    assert torch.equal(ops.clamp_t(t, 0.004), d * (1 - m) + m * 0.004)


# a tile is 4096 entries; 4096 tiles are the most whose counts each block adds up itself
@pytest.mark.parametrize("n", [1, 3, 511, 4096, 4099, 300_001, 4096 * 4096, 4096 * 4096 + 5])
@pytest.mark.parametrize("shift", [0, 1, 4])
def test_mask_scan_any_size(n, shift):
    """Byte-exact exclusive scan: aligned and unaligned masks, any nonzero byte set, either side of the tile limit."""
    g = torch.Generator(device="cuda").manual_seed(n + shift)
    m = torch.randint(0, 5, (n + shift,), device="cuda", generator=g, dtype=torch.uint8)[shift:]
    offsets, count = ops.mask_scan(m)
    incl = (m != 0).cumsum(0)
    assert torch.equal(offsets.long(), incl - (m != 0).long()) and int(count) == int(incl[-1])


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("rays,S,P,F", [(1, 1, 1, 8), (43, 3, 3, 32), (127, 1, 8, 32), (129, 8, 8, 32), (60, 5, 11, 40),
                                        (33, 4, 17, 64), (300, 2, 40, 8)])
def test_feature_gather_paths_agree(rays, S, P, F, half):
    """Rows a multiple of 16 bytes take the wide gather; the same rows from an unaligned base take the general one."""
    rng = np.random.default_rng(rays * 100 + P)
    n, dev = 500, "cuda"
    T = lambda *s: torch.from_numpy(rng.standard_normal(s).astype(np.float32)).to(dev)
    xyz, rgb, dir_, sp = T(n, 3), T(n, 3), T(n, 3), T(rays, S, 3)
    feat = T(n, F).to(torch.float16 if half else torch.float32)
    odd = torch.empty(n * F + 1, dtype=feat.dtype, device=dev)[1:].view(n, F)
    odd.copy_(feat)
    ids = torch.from_numpy(rng.integers(-1, n, (rays, S, P)).astype(np.int32)).to(dev)
    mask = torch.from_numpy(rng.random((rays, S)) < 0.4).to(dev)
    mask[-1, -1] = True
    uv = torch.from_numpy(rng.integers(0, 90, (rays, 2)).astype(np.int32)).to(dev)
    for ray_uv in (None, uv):
        call = lambda f: ops.feature_query(xyz, rgb, dir_, f, sp, ids, mask, T_c2w, 80.0, 81.0, 20.0, 21.0, 37, ray_uv)
        T_c2w = torch.eye(4, device=dev) + 0.1 * torch.arange(16, device=dev, dtype=torch.float32).view(4, 4)
        wide, general = call(feat), call(odd)
        assert all(torch.equal(a, b) for a, b in zip(wide, general))
        assert torch.equal(wide[4], sp[mask])
        sel = ids[mask].long()
        want = torch.where((sel >= 0)[..., None], feat.float()[sel.clamp(min=0)], torch.zeros((), device=dev))
        assert torch.equal(wide[3], want) and torch.equal(wide[5], sel >= 0)


@pytest.mark.parametrize("M", [128 * 148, 128 * 148 + 1, 2 * 128 * 148 + 5])
def test_aggregator_tiles_agree(M):
    """CTAs that serve several tiles one after another give what they give for one tile each, bit for bit."""
    g = torch.Generator(device="cuda").manual_seed(M)
    R = lambda *s: torch.randn(*s, device="cuda", generator=g)
    layers = [(R(o, i) / i ** 0.5, 0.1 * R(o)) for _, o, i in ops.AGG_LAYERS]
    packed = ops.aggregator_pack([w for w, _ in layers], [b for _, b in layers])
    P = 2
    sp, rays = R(M, 3), R(M, 3)
    ins = [sp[:, None] + 0.01 * R(M, P, 3), R(M, P, 3), R(M, P, 3), R(M, P, 32), sp, R(M, P) > -0.5]
    call = lambda a, b: ops.aggregator_forward(packed, *[x[a:b].contiguous() for x in ins],
                                               torch.ones((b - a, 1), dtype=torch.bool, device="cuda"),
                                               rays[a:b].contiguous(), check_status=True)
    alpha, color = call(0, M)
    step = 128 * 64
    parts = [call(a, min(M, a + step)) for a in range(0, M, step)]
    assert torch.equal(alpha, torch.cat([p[0] for p in parts])) and torch.equal(color, torch.cat([p[1] for p in parts]))
    assert torch.isfinite(color).all() and color.std() > 0
