"""Radiance-cache kernels at the edges of their tiles (16 samples a warp, 32
warps a block, partial rounds of blocks) against single samples: a sample's
answer does not depend on its place in a batch."""
import numpy as np
import pytest
import torch

from mray_gb300.cache import RadianceCache
from oracle import nrc

pytestmark = pytest.mark.gpu
AABB = (-2.0, -2.0, -2.0, 2.0, 2.0, 2.0)


def _cache(levels, log2):
    c = RadianceCache(levels=levels, log2_table_size=log2, aabb=AABB, max_batch=4096, seed=3)
    rng = np.random.default_rng(levels)
    c.set_params(rng.uniform(-0.25, 0.25, nrc.WEIGHTS).astype(np.float32),
                 rng.uniform(-0.6, 0.6, c.table_size).astype(np.float16).astype(np.float32))
    return c


def _inputs(n, seed):
    rng = np.random.default_rng(seed)
    x = np.zeros((n, 16), np.float32)
    x[:, 0:3] = rng.random((n, 3)) * 4.4 - 2.2            # some outside the box: clamped
    x[:, 3] = rng.random(n)
    d = rng.standard_normal((n, 3))
    x[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    x[:, 8:11] = x[:, [6, 4, 5]]
    x[:, 12:15] = rng.random((n, 3))
    return torch.from_numpy(x).cuda()


# an odd level count leaves one lane of a pair without a level
@pytest.mark.parametrize("levels,log2", [(16, 14), (7, 10), (1, 8)])
def test_query_batches_agree(levels, log2):
    c = _cache(levels, log2)
    x = _inputs((1 << 17) + 33, 1)
    whole = c.query(x)                                     # a full round and a partial one
    # 152 blocks of 32 warps hold 77,824 samples
    for n in (1, 15, 16, 17, 63, 64, 65, 1000, 77823, 77825, 98304, 98305, 1 << 17):
        assert torch.equal(c.query(x[:n].contiguous()), whole[:n]), n
    assert torch.equal(c.query(x[-40:].contiguous()), whole[-40:])
    c.close()


@pytest.mark.parametrize("levels,n", [(16, 1), (16, 17), (7, 65), (1, 130), (16, 1000)])
def test_gradients_of_ragged_batches(levels, n):
    log2 = 10
    c = _cache(levels, log2)
    w, t = c.get_params()
    x = _inputs(n, 2)
    tgt = torch.rand((n, 4), device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    _, gw, gt = c.gradients(x, tgt)
    _, gwr, gtr = nrc.CacheRef(levels, log2, 16, 2048, AABB).gradients(x.cpu().numpy(), tgt.cpu().numpy(), w, t,
                                                                      bf16=True)
    # the bar of the larger batches (tests/test_gpu_cache.py)
    assert np.linalg.norm(gw - gwr) <= 2e-2 * np.linalg.norm(gwr)
    assert np.linalg.norm(gt - gtr.ravel()[:gt.size]) <= 2e-2 * np.linalg.norm(gtr)
    c.close()
