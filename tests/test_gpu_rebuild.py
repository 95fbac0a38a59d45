"""Builds that reuse the context's arrays and workspace: a scene that grows
and is built again casts like the same scene built once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (icosphere level, meshes, instances) added before each build: one triangle
# mesh up to blocks of several MB, instances with shared meshes
STEPS = [[(0, 1, 1), (1, 3, 5), (2, 0, 40)], [(5, 2, 3), (0, 300, 300), (6, 4, 4)], [(7, 1, 2), (1, 1, 1)]]


def _mesh(level, k):
    from mray_gb300 import scenes
    if level == 0 and k % 2:                       # a single triangle
        return np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32) + k % 7, np.array([[0, 1, 2]], np.uint32)
    pos, idx = scenes.icosphere(level, 1.0 + 0.1 * (k % 5), 0.05, 4.0, k)
    return pos, idx


def _add(acc, meshes, instances, level, base):
    from mray_gb300 import scenes
    ids = []
    for k in range(meshes):
        pos, idx = _mesh(level, k)
        ids.append(acc.upload_mesh(pos, idx, prim_key_base=base))
        base += idx.shape[0]
    m = scenes.instance_field(instances, level + 1, box=30.0)
    last = ids[-1] if ids else 0
    for i in range(instances):
        acc.add_instance(ids[i % len(ids)] if ids else last, m[i], trans_key=i, accel_key=level)
    return base


def _cast(acc):
    import torch
    from mray_gb300 import scenes
    rays = torch.from_numpy(scenes.primary_rays(96, 64, seed=1, eye=(0.0, 0.0, -60.0))).cuda()
    hits = torch.full((rays.shape[0], 4), -1, dtype=torch.int32, device="cuda")
    meta = torch.zeros((rays.shape[0], 2), device="cuda")
    acc.cast_rays(rays, hits, meta)
    acc.sync_status()
    return rays.cpu().numpy().view(np.uint32), hits.cpu().numpy(), meta.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("steps", STEPS)
@pytest.mark.parametrize("watertight", [False, True])
def test_rebuilt_scene_casts_like_a_new_one(steps, watertight):
    from mray_gb300 import Accelerator
    acc = Accelerator(0, watertight=watertight)
    base = 0
    for n in range(len(steps)):
        level, meshes, instances = steps[n]
        base = _add(acc, meshes, instances, level, base)
        for again in range(2):
            acc.construct()
            got = _cast(acc)
        fresh = Accelerator(0, watertight=watertight)
        b = 0
        for level, meshes, instances in steps[:n + 1]:
            b = _add(fresh, meshes, instances, level, b)
        fresh.construct()
        want = _cast(fresh)
        assert (want[1][:, 0] != -1).any()
        for x, y in zip(got, want):
            np.testing.assert_array_equal(x, y)
        np.testing.assert_array_equal(acc.scene_aabb(), fresh.scene_aabb())
        assert acc.stats()["blasNodes"] == fresh.stats()["blasNodes"]
        fresh.close()
    acc.close()
