"""Small casts spread their rays over the warps, large ones fill them: both leave
the same bytes, ties between equal triangles and instances included."""
import numpy as np
import pytest

from mray_gb300 import Accelerator, scenes

pytestmark = pytest.mark.gpu

LARGE = 600000         # above every limit of the small form


def _soup(n, seed):
    """n triangles in a unit cube, every third one listed again at the end."""
    rng = np.random.default_rng(seed)
    pos = (rng.uniform(-1, 1, (n, 1, 3)) + rng.uniform(-0.3, 0.3, (n, 3, 3))).reshape(-1, 3).astype(np.float32)
    idx = np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    return pos, np.concatenate([idx, idx[::3]])


@pytest.mark.parametrize("watertight", [False, True])
@pytest.mark.parametrize("tris,ninst", [(1, 1), (7, 3), (900, 20), (20000, 40)])
def test_small_casts_equal_large_ones(tris, ninst, watertight):
    import torch
    acc = Accelerator(0, watertight=watertight)
    mesh = acc.upload_mesh(*_soup(tris, tris))
    m = scenes.instance_field(ninst, 5, box=3.0, jitter=0.3)
    m = np.concatenate([m, m[:(ninst + 1) // 2]])                # every other instance twice
    for i in range(m.shape[0]):
        acc.add_instance(mesh, m[i], trans_key=i, accel_key=i)
    acc.construct()
    rays = scenes.primary_rays(800, 750, 2, eye=(0, 0, -9), tan_half_fov=0.5)[:LARGE]
    rng = np.random.default_rng(8)
    rays[::3, 0:3] = rng.uniform(-4, 4, rays[::3, 0:3].shape)    # origins inside the field
    rays[::7, 4:7] = np.eye(3)[rng.integers(0, 3, rays[::7].shape[0])] * rng.choice([-1.0, 1.0], (rays[::7].shape[0], 1))
    rays = torch.from_numpy(np.ascontiguousarray(rays.astype(np.float32))).cuda()

    def cast(part, order=None):
        r, n = part.clone(), part.shape[0]
        hits = torch.full((n, 4), -1, dtype=torch.int32, device="cuda")
        meta = torch.zeros((n, 2), dtype=torch.float32, device="cuda")
        bits = torch.zeros((n + 31) // 32, dtype=torch.int32, device="cuda")
        acc.cast_visibility_rays(bits, part, order)
        acc.cast_rays(r, hits, meta, order)
        vis = (bits.cpu().numpy().view(np.uint32)[np.arange(n) >> 5] >> (np.arange(n) & 31)) & 1
        return [r.cpu().numpy(), hits.cpu().numpy(), meta.cpu().numpy(), vis]

    want = cast(rays)
    assert tris < 100 or (want[1][:, 0] != -1).sum() > 1000
    at = 0
    for n in (1, 3, 31, 32, 33, 2127, 2129, 30000, 34047, 34049, 136193, 250000):
        for a, b in zip(cast(rays[at:at + n]), want):
            np.testing.assert_array_equal(a.view(np.uint32), b[at:at + n].view(np.uint32))
        at += n
    # listed rays only: the others keep what they held
    order = torch.randperm(LARGE, device="cuda")[:1003].to(torch.int32)
    got, listed = cast(rays, order), order.cpu().numpy()
    for k in range(3):
        np.testing.assert_array_equal(got[k][listed].view(np.uint32), want[k][listed].view(np.uint32))
    np.testing.assert_array_equal(got[3][listed], want[3][listed])
    rest = np.setdiff1d(np.arange(LARGE), listed)
    assert (got[1][rest] == -1).all() and (got[3][rest] == 0).all()
    acc.close()
