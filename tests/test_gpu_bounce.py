"""The bounce loop's work groups: grouping the paths before shading changes no
image, at sizes around the grouping kernel's tiles (2048 paths) and warps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _render(pt, guided, **kw):
    from mray_gb300 import scenes
    from mray_gb300.pt import PathTracer
    p = PathTracer.params(camera=scenes.box_camera(), rr_start=2, seed=9, **kw)
    if guided:
        pt.guide_clear()
        return pt.render_guided(p).cpu().numpy()
    return pt.render(p).cpu().numpy()


@pytest.mark.parametrize("scene", ["box_scene_mixed", "sky_scene"])
@pytest.mark.parametrize("w,h,spp,depth", [(1, 1, 1, 1), (31, 1, 1, 3), (64, 32, 1, 4), (683, 3, 1, 4), (61, 47, 5, 6),
                                           (512, 513, 1, 3)])
def test_grouping_is_invisible(scene, w, h, spp, depth):
    from mray_gb300 import scenes
    from mray_gb300.pt import PathTracer, load_box_scene
    pt = PathTracer(0)
    load_box_scene(pt, getattr(scenes, scene)(3))
    if scene == "sky_scene":
        pt.set_env(scenes.sky_map(32, 16, seed=1))
    pt.guide_create(entry_limit=20000)
    for guided in (False, True):
        a, b, c = (_render(pt, guided, width=w, height=h, spp=spp, max_depth=depth, partition=k)
                   for k in (False, True, "auto"))
        np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(a, c)
    pt.close()
