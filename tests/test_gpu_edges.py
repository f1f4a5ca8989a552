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


@pytest.mark.parametrize("radius", [-0.05, -1e-20, 0.0, float("nan")])
def test_radius_that_keeps_nothing(radius):
    """A candidate is kept when its distance is below the radius: never for one of zero or less."""
    cam = synth.look_at_camera((0.3, 0.2, 4.0), (0, 0, 0), 40, 30, 36.0)
    X, c2w, sidx, table = _view(synth.sphere_cloud(np.random.default_rng(1), 3_000), cam)
    assert (table[:, 1] > 0).any()
    o = synth.Options(kernel_size=3, radius_threshold=radius, num_point_per_ray=16)
    rays = torch.arange(1200, dtype=torch.int32, device="cuda")
    rows = ops.quick_query(X, c2w, cam.fx, cam.fy, cam.cx, cam.cy, 40, 30, o, sidx, table, rays)
    assert (rows == -1).all()
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
