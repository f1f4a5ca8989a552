"""The work that users of this framework have it do, as cases whose time and outputs can be measured.

A case is a dict of plain values; `prepare` makes what a user's program holds before the call (clouds and cameras on the
GPU, weights, a batch's renderer), `run` is one pass through the public entry points and `exact` the same outputs in
64 bits by plain torch.  Clouds and cameras are those of `hashpoint.synth` (the workloads of the benchmark and the tests).

The search and sampling outputs have no value in 64 bits to be held against: bucket order, the kept points, the depth
bins and the emitted samples are decisions that 32-bit arithmetic takes, and one decision taken otherwise moves all that
follows.  They are compared as they are.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hashpoint-code_b200"))

from epcq import epcq  # noqa: E402
from hashpoint import batch, synth  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # one view of a few thousand points on a small image, as an interactive preview or a unit of a test asks for:
        # launches and host calls are most of it
        view("view-tiny", "sphere", 4_000, 48, 40, kernel=3, radius=0.05),
        # a single object at 400 x 400: 100k points on a sphere, 3 x 3 window
        view("view-sphere", "sphere", 100_000, 400, 400, kernel=3, radius=0.01),
        # the headline workload: one of its views of 1M points on boxes and ellipsoids at 800 x 800, 5 x 5 window
        view("view-shapes", "shapes", 1_000_000, 800, 800),
        # very uneven density at 1600 x 1200: 3M clustered points, 16 samples a ray
        view("view-clusters", "clusters", 3_000_000, 1600, 1200, radius=0.005, samples=16),
        # a large scene asked for at a small resolution, as the serving workload does: hundreds of candidates a ray
        view("view-dense", "shapes", 4_000_000, 512, 512),
        # the render options' defaults (16 samples, 4 points each, radius 0.016) on an image that is no multiple of a
        # tile, buckets ordered by depth
        view("view-sorted-ragged", "shapes", 333_333, 763, 509, radius=0.016, samples=16, per_sample=4, sort=True),
        # many views of several clouds of uneven sizes and resolutions in one call
        {"name": "batch-mixed", "kind": "batch", "clouds": 4, "views": 10, "points_lo": 50_000, "points_hi": 1_500_000},
        # the ids near listed pixel rays, as the point-ray search benchmark asks for them
        {"name": "query-rays", "kind": "query", "points": 1_000_000, "width": 800, "height": 800, "rays": 65_536,
         "kernel": 5, "radius": 0.008, "cap": 256},
        # the point attributes of a view's samples (16-bit features of the headline workload)
        {"name": "feature-query", "kind": "features", "points": 1_000_000, "width": 800, "height": 800, "samples": 8,
         "per_sample": 8, "half": True},
        # the per-point MLP over a quarter of a view's samples (a view is rendered in chunks of rays)
        {"name": "aggregate", "kind": "aggregate", "samples": 143_000, "slots": 8, "per_sample": 8, "rays": 160_000},
        # compositing a view's samples
        {"name": "render", "kind": "render", "rays": 640_000, "slots": 8, "white": True},
        # a whole frame: search, gather, MLP and compositing of one 400 x 400 view
        {"name": "frame", "kind": "frame", "cloud": "shapes", "points": 300_000, "width": 400, "height": 400},
    ]


def view(name, cloud, points, width, height, kernel=5, radius=0.008, samples=8, per_sample=8, sort=False):
    return {"name": name, "kind": "view", "cloud": cloud, "points": points, "width": width, "height": height,
            "kernel": kernel, "radius": radius, "samples": samples, "per_sample": per_sample, "sort": sort}


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["view", "view", "view", "view", "batch", "query", "features", "aggregate", "render", "frame"])
    if kind == "view":
        cloud = rng.choice(["sphere", "shapes", "shapes", "clusters"])
        top = {"sphere": 400_000, "shapes": 3_000_000, "clusters": 3_000_000}[cloud]
        width = log(48, 1600)
        c = view("", cloud, log(3_000, top), width, min(1200, max(40, int(width * rng.uniform(0.6, 1.1)))),
                 kernel=rng.choice([1, 2, 3, 3, 4, 5, 5, 5]), radius=rng.choice([0.004, 0.005, 0.008, 0.01, 0.016]),
                 samples=rng.choice([4, 5, 8, 8, 16]), per_sample=rng.choice([4, 8, 8, 12]), sort=rng.random() < 0.25)
        del c["name"]
        return c
    if kind == "batch":
        lo = log(20_000, 200_000)
        return {"kind": kind, "clouds": rng.randint(1, 4), "views": rng.randint(2, 9), "points_lo": lo,
                "points_hi": lo + log(50_000, 1_200_000)}
    if kind == "query":
        width = log(200, 1000)
        return {"kind": kind, "points": log(30_000, 1_000_000), "width": width, "height": int(width * rng.uniform(0.6, 1.0)),
                "rays": log(500, 65_000), "kernel": rng.choice([1, 3, 5, 7]), "radius": rng.choice([0.005, 0.008, 0.016]),
                "cap": rng.choice([32, 100, 256])}
    if kind == "features":
        width = log(80, 790)
        return {"kind": kind, "points": log(20_000, 1_000_000), "width": width, "height": int(width * rng.uniform(0.6, 1.0)),
                "samples": rng.choice([4, 8, 16]), "per_sample": rng.choice([4, 8, 8]), "half": rng.random() < 0.5}
    if kind == "aggregate":
        m = log(300, 140_000)
        return {"kind": kind, "samples": m, "slots": rng.choice([8, 16]), "per_sample": rng.choice([4, 8, 8]),
                "rays": int(m * rng.uniform(0.4, 1.4)) + 64}
    if kind == "render":
        return {"kind": kind, "rays": log(1_000, 639_999), "slots": rng.choice([4, 7, 8, 8, 16]), "white": rng.random() < 0.5}
    width = log(60, 400)
    return {"kind": kind, "cloud": rng.choice(["sphere", "shapes"]), "points": log(10_000, 300_000), "width": width,
            "height": int(width * rng.uniform(0.6, 1.0))}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def cloud_and_camera(rng, c):
    """A cloud and a camera of the named workload, the focal length scaled to the image."""
    W, H = c["width"], c["height"]
    if c["cloud"] == "sphere":
        return synth.sphere_cloud(rng, c["points"]), synth.orbit_cameras(rng, 1, 4.0, W, H, 555.0 * W / 400)[0]
    if c["cloud"] == "shapes":
        return synth.shapes_cloud(rng, c["points"]), synth.orbit_cameras(rng, 1, 4.0, W, H, 1111.0 * W / 800)[0]
    cam = synth.orbit_cameras(rng, 1, None, W, H, 2890.0 * W / 1600, elev_deg=(20.0, 80.0), radius_range=(2.5, 3.5))[0]
    return synth.clusters_cloud(rng, c["points"]), cam


def on_gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def camera_spec(cam):
    return epcq.CameraSpec(on_gpu(cam.c2w), on_gpu(cam.w2c), on_gpu(cam.K), cam.fx, cam.fy, cam.cx, cam.cy, cam.width,
                           cam.height)


def generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def attributes(npnt, seed, half):
    """Colours, directions and 32-wide features of a cloud's points, as a checkpoint brings them."""
    g, n = generator(seed), npnt.xyz_data.shape[0]
    npnt.rgb_data.data = torch.rand((n, 3), device=DEV, generator=g)
    npnt.dir_data.data = torch.nn.functional.normalize(torch.randn((n, 3), device=DEV, generator=g), dim=-1)
    feat = torch.randn((n, 32), device=DEV, generator=g).half()  # 16-bit values, held in 16 or 32 bits
    npnt.feat_data.data = feat if half else feat.float()


def trained_aggregator(seed):
    """An Aggregator whose biases are not all zero, as training leaves them."""
    torch.manual_seed(int(seed))
    agg = epcq.Aggregator()
    with torch.no_grad():
        for p in agg.parameters():
            if p.dim() == 1:
                p.normal_(0.0, 0.05)
    return agg.to(DEV)


def view_samples(seed, c):
    """A view's sample arrays, made by torch alone: a ray's samples lie near the points of its pixel and the pixels
    after it, so that neighbouring rays share points as in a real view, and three rays in ten hold one to five samples."""
    rng = np.random.default_rng(seed)
    xyz, cam = cloud_and_camera(rng, dict(c, cloud="shapes"))
    X, H, W, S, P = on_gpu(xyz), cam.height, cam.width, c["samples"], c["per_sample"]
    g = generator(seed)
    p = X.double() @ on_gpu(cam.w2c).double()[:3, :3].t() + on_gpu(cam.w2c).double()[:3, 3]
    u = (p[:, 0] / p[:, 2] * cam.fx + cam.cx).long().clamp(0, W - 1)
    v = (p[:, 1] / p[:, 2] * cam.fy + cam.cy).long().clamp(0, H - 1)
    pix, order = torch.sort(v * W + u)
    first = torch.searchsorted(pix, torch.arange(H * W, device=DEV))
    count = torch.searchsorted(pix, torch.arange(H * W, device=DEV), right=True) - first
    n = len(xyz)
    slot = torch.arange(S, device=DEV)
    hit = torch.sort((count == 0).int(), stable=True).indices[:H * W * 3 // 10]  # rays over points first
    emitted = torch.zeros(H * W, dtype=torch.long, device=DEV)
    emitted[hit] = (torch.arange(len(hit), device=DEV) % min(5, S) + 1)[torch.randperm(len(hit), device=DEV, generator=g)]
    mask = slot[None, :] < emitted[:, None]
    at = (first[:, None, None] + slot[None, :, None] + torch.arange(P, device=DEV)[None, None, :]).clamp(0, n - 1)
    found = torch.randint(1, P + 4, (H * W, S, 1), device=DEV, generator=g)  # most samples find all of their points
    ids = torch.where((torch.arange(P, device=DEV) < found) & mask[..., None], order[at], -1)
    near = X[order[at[..., 0]]] + 0.002 * torch.randn((H * W, S, 3), device=DEV, generator=g)
    return (X, cam, torch.where(mask[..., None], near, 0.0).view(H, W, S, 3).contiguous(),
            ids.to(torch.int32).view(H, W, S, P).contiguous(), mask.view(H, W, S).contiguous())


def pair_inputs(seed, c):
    """What FeatureQuery hands to the Aggregator: zeros where a sample found no further point."""
    g, M, P, S, R = generator(seed), c["samples"], c["per_sample"], c["slots"], c["rays"]

    def rn(*s):
        return torch.randn(s, device=DEV, generator=g)

    sp = rn(M, 3)
    found = torch.randint(1, P + 4, (M, 1), device=DEV, generator=g)
    valid = torch.arange(P, device=DEV) < found
    z = valid[..., None]
    xyz = torch.where(z, sp[:, None, :] + 0.004 * rn(M, P, 3), 0.0)
    rgb = torch.where(z, torch.rand((M, P, 3), device=DEV, generator=g), 0.0)
    dr = torch.where(z, torch.nn.functional.normalize(rn(M, P, 3), dim=-1), 0.0)
    feat = torch.where(z, rn(M, P, 32).half().float(), 0.0)
    rays = rn(M, 3)
    mask = torch.zeros(R * S, dtype=torch.bool, device=DEV)
    mask[torch.randperm(R * S, device=DEV, generator=g)[:M]] = True
    return xyz, rgb, dr, feat, sp, valid, mask.view(R, S), rays


def ray_samples(seed, c):
    g, R, S = generator(seed), c["rays"], c["slots"]
    t = 3.0 + torch.cumsum((torch.randint(0, 40, (R, S), device=DEV, generator=g) + 0.5) * 0.001, 1)
    n = torch.randint(0, S + 1, (R, 1), device=DEV, generator=g)
    on = torch.arange(S, device=DEV) < n
    sigma = torch.where(on, 200.0 * torch.rand((R, S), device=DEV, generator=g) ** 2, 0.0)
    rgb = torch.where(on[..., None], torch.rand((R, S, 3), device=DEV, generator=g), 0.0)
    return torch.where(on, t, 0.0), sigma, rgb


def options(c):
    return epcq.RenderOptions(kernel_size=c["kernel"], radius_threshold=c["radius"],
                              num_sample_points_per_ray=c.get("samples", 8), num_point_cloud_per_sp=c.get("per_sample", 8),
                              num_point_per_ray=c.get("cap", 256))


BATCH = {"kernel": 5, "radius": 0.008, "samples": 8, "per_sample": 8}
FRAME = {"kernel": 5, "radius": 0.016, "samples": 8, "per_sample": 8}


def prepare(case, seed):
    c, kind = case, case["kind"]
    rng = np.random.default_rng(seed)
    s = {"kind": kind, "case": c}
    if kind == "view":
        xyz, cam = cloud_and_camera(rng, c)
        s.update(points=epcq.NeuralPoints(pc_type="pc", points=on_gpu(xyz)), cam=camera_spec(cam), opt=options(c))
    elif kind == "batch":
        sizes = [int(n) for n in np.geomspace(c["points_lo"], c["points_hi"], c["clouds"])]
        clouds = [on_gpu(synth.shapes_cloud(rng, n)) for n in sizes]
        views = []
        for i in range(c["views"]):
            W, H = synth.MIXED_RESOLUTIONS[(i + i // 4) % 4]
            views.append((i % c["clouds"], synth.orbit_cameras(rng, 1, 4.0, W, H, 1111.0 * W / 800)[0]))
        s.update(renderer=batch.BatchRenderer(clouds, views, options(BATCH), device=DEV))
    elif kind == "query":
        xyz, cam = cloud_and_camera(rng, dict(c, cloud="shapes"))
        points, spec, opt = epcq.NeuralPoints(pc_type="pc", points=on_gpu(xyz)), camera_spec(cam), options(c)
        idx, _, table = points.pts2plane(spec, opt)
        rays = torch.randperm(cam.width * cam.height, device=DEV, generator=generator(seed))[:c["rays"]].to(torch.int32)
        s.update(points=points, cam=spec, opt=opt, idx=idx, table=table, rays=rays)
    elif kind == "features":
        X, cam, sp_xyz, pc_idx, mask = view_samples(seed, c)
        points = epcq.NeuralPoints(pc_type="pc", points=X)
        attributes(points, seed, c["half"])
        s.update(points=points, cam=camera_spec(cam), query=epcq.FeatureQuery(), args=(sp_xyz, pc_idx, mask))
    elif kind == "aggregate":
        s.update(agg=trained_aggregator(seed), args=pair_inputs(seed, c))
    elif kind == "render":
        s.update(args=ray_samples(seed, c))
    else:
        xyz, cam = cloud_and_camera(rng, c)
        points = epcq.NeuralPoints(pc_type="pc", points=on_gpu(xyz))
        attributes(points, seed, True)
        s.update(points=points, cam=camera_spec(cam), opt=options(FRAME), query=epcq.FeatureQuery(),
                 agg=trained_aggregator(seed))
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "view":
        table = s["points"].pts2plane(s["cam"], s["opt"], sort=s["case"]["sort"])
        return table + s["points"].render_image_hashtable_topk(s["cam"], s["opt"], *table)
    if kind == "batch":
        r = s["renderer"]
        r.run()
        return [r.outputs(i) for i in range(len(r.views))]
    if kind == "query":
        return epcq._C.quick_query_for_nearby_point(s["points"]._to_cpp(), s["cam"]._to_cpp(), s["opt"]._to_cpp(), s["idx"],
                                                    s["table"], s["rays"])
    if kind == "features":
        return s["query"](s["points"], *s["args"], s["cam"])
    if kind == "aggregate":
        with torch.no_grad():
            return s["agg"](*s["args"])
    if kind == "render":
        t, sigma, rgb = s["args"]
        gaps = epcq.clamp_t(t, 0.004)
        return gaps, epcq.render(gaps, sigma, rgb, s["case"]["white"])
    points, cam, opt = s["points"], s["cam"], s["opt"]
    with torch.no_grad():
        table = points.pts2plane(cam, opt)
        sp_xyz, pc_idx, sp_t, mask = points.render_image_hashtable_topk(cam, opt, *table)
        near = s["query"](points, sp_xyz, pc_idx, mask, cam)
        sigma, rgb = s["agg"](*near[:6], mask, near[6])
        color = epcq.render(epcq.clamp_t(sp_t.view(sigma.shape), 0.004), sigma, rgb, True)
    return sp_t, pc_idx, mask, sigma, rgb, color


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
PAIR_FLOPS = 2 * (284 + 256 + 263 + 256) * 256 + 2 * 256  # block1, block3 and the alpha branch of one pair
COLOR_FLOPS = 2 * (280 + 128 + 128 + 3) * 128


def view_work(n, W, H, k, S, P):
    # points read once; sorted ids and depths, the hash table and the samples written once; each point projected and
    # held against the rays of its window
    return {"bytes": n * 12 + n * 8 + W * H * 8 + W * H * S * (12 + 4 + 1 + 4 * P), "flops": n * (36 + 25 * k * k)}


def work(case):
    c, kind = case, case["kind"]
    if kind == "view":
        return view_work(c["points"], c["width"], c["height"], c["kernel"], c["samples"], c["per_sample"])
    if kind == "batch":
        n = float(np.mean(np.geomspace(c["points_lo"], c["points_hi"], c["clouds"])))
        px = sum(w * h for w, h in synth.MIXED_RESOLUTIONS) / len(synth.MIXED_RESOLUTIONS)
        w = view_work(n, 1, px, 5, 8, 8)
        return {k: v * c["views"] for k, v in w.items()}
    if kind == "query":  # the window's cells, ids and points of each ray, its row of ids
        seen = c["kernel"] ** 2 * 1.4
        return {"bytes": c["rays"] * (4 + c["kernel"] ** 2 * 8 + seen * 16 + c["cap"] * 4), "flops": c["rays"] * seen * 25}
    if kind == "features":
        slots, m = c["width"] * c["height"] * c["samples"], c["width"] * c["height"] * 0.15 * (min(5, c["samples"]) + 1)
        row = c["per_sample"] * (37 + 4 * 32) + 24
        return {"bytes": slots + m * (12 + 4 * c["per_sample"]) + c["points"] * (36 + 32 * (2 if c["half"] else 4)) + m * row,
                "flops": 0}
    if kind == "aggregate":
        m, p = c["samples"], c["per_sample"]
        return {"bytes": m * (p * (37 + 128) + 24) + c["rays"] * c["slots"] * 17,
                "flops": m * (min(p, 0.5 * (p + 3)) * PAIR_FLOPS + COLOR_FLOPS)}
    if kind == "render":
        return {"bytes": c["rays"] * (c["slots"] * (4 + 4 + 4 + 12) + 12), "flops": c["rays"] * c["slots"] * 20}
    px, o = c["width"] * c["height"], FRAME
    w = view_work(c["points"], c["width"], c["height"], o["kernel"], o["samples"], o["per_sample"])
    m = px * 0.8  # samples: a little under one a ray
    return {"bytes": w["bytes"] + m * 8 * 165 * 2 + px * (8 * 40 + 12), "flops": w["flops"] + m * (6 * PAIR_FLOPS + COLOR_FLOPS)}


# ---------------------------------------------------------------------------
# the same in 64 bits, by plain torch
# ---------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "features":
        return exact_features(case, seed)
    if kind == "aggregate":
        return exact_aggregate(case, seed)
    if kind == "render":
        return exact_render(case, seed)
    return None  # search and sampling: see the file's head


def exact_features(c, seed):
    s = prepare(c, seed)
    points, cam, (sp_xyz, pc_idx, mask) = s["points"], s["cam"], s["args"]
    S = mask.shape[-1]
    at = mask.view(-1).nonzero().view(-1)
    ids = pc_idx.view(-1, pc_idx.shape[-1])[at].long()
    valid = ids >= 0
    rows = [torch.where(valid[..., None], t.data[ids.clamp(min=0)].double(), 0.0)
            for t in (points.xyz_data, points.rgb_data, points.dir_data, points.feat_data)]
    pixel = at // S
    d = torch.stack([(pixel % cam.width - cam.cx) / cam.fx, (pixel // cam.width - cam.cy) / cam.fy,
                     torch.ones_like(pixel, dtype=torch.float64)], -1)
    return (*rows, sp_xyz.view(-1, 3)[at].double(), None, d.double() @ cam.c2w.double()[:3, :3].t())


def encoded(x, freqs):
    a = (x[..., None] * 2.0 ** torch.arange(freqs, dtype=torch.float64, device=x.device)).flatten(-2)
    return torch.stack([torch.sin(a), torch.cos(a)], -1).flatten(-2)


def exact_aggregate(c, seed):
    s = prepare(c, seed)
    xyz, rgb, dr, feat, sp, valid, mask, rays = [t.double() if t.is_floating_point() else t for t in s["args"]]
    prm = {k: v.detach().double() for k, v in s["agg"].state_dict().items()}

    def linear(name, x):
        return x @ prm[name + ".weight"].t() + prm[name + ".bias"]

    def act(x):
        return torch.where(x > 0, x, 0.01 * x)

    alphas = torch.zeros(mask.shape, dtype=torch.float64, device=DEV)
    colors = torch.zeros((*mask.shape, 3), dtype=torch.float64, device=DEV)
    a_out, c_out = [], []
    for i in range(0, len(sp), 16384):
        j = slice(i, i + 16384)
        x, p, ray = xyz[j], sp[j][:, None, :], rays[j][:, None, :]
        h = torch.cat([feat[j], encoded(feat[j], 3), encoded(torch.cat([x - p, x * x - p * p], -1), 5)], -1)
        h = act(linear("block1.2", act(linear("block1.0", h))))
        h = torch.cat([h, rgb[j], dr[j] - ray, (dr[j] * ray).sum(-1, keepdim=True)], -1)
        h = act(linear("block3.2", act(linear("block3.0", h))))
        w = valid[j].double() / (torch.linalg.norm(x - p, dim=-1) + 1e-6)
        w = w / (w.sum(-1, keepdim=True) + 1e-6)
        a_out.append((torch.nn.functional.softplus(linear("alpha_branch.0", h)[..., 0] - 1) * w).sum(-1))
        h = torch.cat([(h * w[..., None]).sum(1), encoded(rays[j], 4)], -1)
        for k in (0, 2, 4):
            h = act(linear("color_branch.%d" % k, h))
        c_out.append(torch.sigmoid(linear("color_branch.6", h)) * 1.002 - 0.001)
    alphas[mask], colors[mask] = torch.cat(a_out), torch.cat(c_out)
    return alphas, colors


def exact_render(c, seed):
    t, sigma, rgb = [x.double() for x in ray_samples(seed, c)]
    gap = torch.cat([t[:, 1:] - t[:, :-1], torch.full_like(t[:, :1], 0.004)], 1)
    gap = torch.where((gap < 1e-8) | (gap > 0.008), torch.full_like(gap, 0.004), gap)
    opacity = 1 - torch.exp(-sigma * gap)
    through = torch.cumprod(torch.cat([torch.ones_like(t[:, :1]), 1 - opacity + 1e-10], 1), 1)
    color = ((opacity * through[:, :-1])[..., None] * rgb).sum(1)
    return gap, color + through[:, -2:-1] * float(c["white"])
