"""Guided path tracing where its kernels change course, against the oracle:
a table past its entry limit (draws without a slot), and cells that take more
records a bounce than a warp's window, than one warp's chain (1,024), and many
times that."""
import numpy as np
import pytest

import oracle
from mray_gb300 import scenes
from mray_gb300.pt import PathTracer, load_box_scene
from test_gpu_guided import _check_grids, _check_images

pytestmark = pytest.mark.gpu


def _both(w, h, spp, per_pass, depth, seed=5, **guide):
    cam = scenes.box_camera()
    pt = PathTracer(0)
    S = oracle.PtScene(load_box_scene(pt, 0))
    pt.guide_create(**guide)
    G = S.guide(**guide)
    g = pt.render_guided(PathTracer.params(w, h, spp, cam, max_depth=depth, rr_start=2, seed=seed,
                                           samples_per_pass=per_pass))
    o = S.render_guided(S.params(w, h, spp, cam, max_depth=depth, rr_start=2, seed=seed), G, per_pass)
    out = g.cpu().numpy(), o, pt.guide_read(), G.read(), pt.guide_stats()
    pt.close()
    return out


# one path at a time: the order of insertions, and so which of them still find
# room, is the oracle's (at the vertex that reaches the limit a code drawn
# again keeps the slot of its first draw here, where the oracle asks the full
# table once more: these sizes do not meet it)
@pytest.mark.parametrize("limit,spp", [(1, 8), (8, 48), (200, 96)])
def test_past_the_entry_limit(limit, spp):
    g, o, gs, os_, (used, size) = _both(1, 1, spp, 1, 6, entry_limit=limit)
    assert used == (gs[0] != np.uint64(0xFFFFFFFFFFFFFFFF)).sum()
    _check_images(g, o)
    if limit == 1:                              # a table of one slot: room for none
        assert used == 0 and (os_[0] == gs[0]).all()
        return
    _check_grids(gs, os_)
    if limit == 8:
        assert used >= int(0.6 * size)          # the limit was reached


@pytest.mark.parametrize("w,h,spp,depth", [(16, 16, 4, 4), (64, 64, 8, 3), (160, 128, 8, 3)])
def test_runs_of_many_records(w, h, spp, depth):
    g, o, gs, os_, _ = _both(w, h, spp, spp, depth, max_level_offset=8)
    _check_images(g, o)
    _check_grids(gs, os_)
