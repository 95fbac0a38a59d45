"""The collapse to 8-wide nodes, every way of choosing children, on trees where
its order of children and slots is least clear: equal boxes, one axis, few
triangles, chains; against the CPU oracle."""
import numpy as np
import pytest

from mray_gb300 import scenes
from parity_util import MISS, build_pair, gpu_closest, tri_retest

pytestmark = pytest.mark.gpu


def _mesh(shape):
    rng = np.random.default_rng(7)
    if shape == "equal":            # 300 triangles of 3 kinds, all boxes alike
        pos = np.tile(np.eye(3), (300, 1))
    elif shape == "line":           # centroids on one axis
        pos = np.zeros((700, 3, 3))
        pos[:, :, 0] = np.arange(700)[:, None] * 0.004
        pos[:, 1, 1] = pos[:, 2, 2] = 0.4
    elif shape == "chain":          # sizes over six orders: a tree as deep as it gets
        s = np.geomspace(1e-6, 1.0, 120)[:, None, None]
        pos = s * (1.0 + 0.5 * rng.uniform(-1, 1, (120, 3, 3)))
    else:                           # a soup of so many triangles
        pos = rng.uniform(-1, 1, (int(shape), 1, 3)) + rng.uniform(-0.3, 0.3, (int(shape), 3, 3))
    pos = pos.reshape(-1, 3).astype(np.float32)
    return pos, np.arange(pos.shape[0], dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("mode", ["sah-blas", "sah", "sah-large", "greedy"])
@pytest.mark.parametrize("shape", ["equal", "line", "chain", "1", "2", "7", "8", "9", "65", "2100"])
def test_collapse_keeps_every_triangle(cuda_lib, built_libs, monkeypatch, mode, shape):
    monkeypatch.setenv("MRG_BVH_COLLAPSE", mode)
    pos, idx = _mesh(shape)
    acc, S = build_pair(pos, idx, scenes.instance_field(11, 3, box=2.5, jitter=0.3))
    assert acc.stats()["blasTriangles"] == idx.shape[0]
    rays = scenes.primary_rays(120, 90, 4, eye=(0, 0, -9), tan_half_fov=0.5)
    rng = np.random.default_rng(2)
    rays[::2, 0:3] = rng.uniform(-3, 3, rays[::2, 0:3].shape)      # origins among the instances
    grays, ghits, gmeta = gpu_closest(acc, rays, pre_hits=np.full((rays.shape[0], 4), MISS, np.uint32))
    orays, _, _, oinst = S.cast_closest(rays)
    # equal triangles tie by the dozen, so any that is hit at the oracle's t will do
    hit = ghits[:, 0] != MISS
    if shape == "chain":            # the reference's walk loses rays in a binary tree this deep
        assert hit[oinst != MISS].all() and (grays[:, 7] <= orays[:, 7]).all()
    else:
        np.testing.assert_array_equal(hit, oinst != MISS)
        np.testing.assert_array_equal(grays[:, 7].view(np.uint32), orays[:, 7].view(np.uint32))
    retest = tri_retest(S, rays, pos, idx)
    assert all(retest(int(k), ghits[k], gmeta[k], grays[k, 7]) for k in np.flatnonzero(hit))
    assert len(shape) < 4 or hit.any()
    acc.close()
