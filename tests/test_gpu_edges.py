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
