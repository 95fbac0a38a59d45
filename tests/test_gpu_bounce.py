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


# passes that do not divide the samples, automatic passes on either side of the
# split into two (2^19 paths), spectral and ZSobol numbers
@pytest.mark.parametrize("w,h,spp,sampler", [(37, 29, 7, "independent"), (64, 33, 13, "zsobol-owen"),
                                             (256, 227, 9, "independent"), (256, 228, 9, "pcg32")])
def test_passes_are_invisible(w, h, spp, sampler):
    from mray_gb300 import scenes
    from mray_gb300.pt import PathTracer, load_box_scene
    pt = PathTracer(0)
    load_box_scene(pt, scenes.box_scene_mixed(2))
    want = None
    for per_pass in (spp, 0, 1, 2, 4, spp - 1):
        p = PathTracer.params(w, h, spp, scenes.box_camera(), max_depth=4, rr_start=2, seed=5, sampler=sampler,
                              samples_per_pass=per_pass, sample_start=3)
        img = pt.render(p).cpu().numpy()
        want = img if want is None else want
        np.testing.assert_array_equal(img, want)
    assert (want[..., 3] == spp).all()
    pt.close()
