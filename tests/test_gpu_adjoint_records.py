"""The adjoint's vertex records against its replay of each pass
(MRG_PT_ADJOINT=replay): the same terms, summed in another order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tracer(tex):
    from mray_gb300 import scenes
    from mray_gb300.pt import PathTracer
    pt = PathTracer(0)
    sphere = None
    for s in scenes.adjoint_scene(None, n_theta=16, n_phi=32):
        inst = pt.add_surface(s["pos"], s["idx"], s["m34"], cull=s.get("cull", True), uv=s.get("uv"))
        if s["kind"] == "light":
            pt.set_area_light(inst, s["radiance"])
        else:
            pt.set_lambert(inst, s["albedo"])
        if "uv" in s:
            sphere = inst
    tid = pt.add_texture(tex)
    pt.set_albedo_texture(sphere, tid)
    pt.build()
    return pt, tid


# one pass and several (two pipelines), odd sizes, a one-texel texture, depth 1
# (every record is a path's last vertex), a gradient that is only 4-byte aligned
@pytest.mark.parametrize("w,h,spp,per_pass,depth,size,offset", [
    (33, 17, 1, 1, 1, 8, 0), (64, 48, 6, 2, 5, 1, 0), (127, 65, 4, 4, 6, 33, 0), (64, 64, 5, 1, 12, 16, 1)])
def test_records_equal_replay(monkeypatch, w, h, spp, per_pass, depth, size, offset):
    import torch
    from mray_gb300 import scenes
    from mray_gb300.pt import PathTracer
    tex = torch.from_numpy(scenes.value_noise_texture(64, seed=2, dtype=np.float32)[:size, :size].copy()).cuda()
    pt, tid = _tracer(tex)
    p = PathTracer.params(w, h, spp, scenes.box_camera(), max_depth=depth, rr_start=3, seed=4, samples_per_pass=per_pass)
    delta = torch.full((h, w, 4), 1e-3, device="cuda")
    got = {}
    for mode in ("record", "replay"):
        monkeypatch.setenv("MRG_PT_ADJOINT", mode)
        block = torch.zeros(size * size * 4 + 4, device="cuda")
        grad = block[offset:offset + size * size * 4].view(size, size, 4)
        em = torch.zeros((pt.n_instances, 4), device="cuda")
        img = torch.zeros((h, w, 4), device="cuda")
        pt.adjoint(p, tid, delta, grad=grad, image=img, grad_emission=em)
        only = torch.zeros((pt.n_instances, 4), device="cuda")
        pt.adjoint(p, None, delta, grad_emission=only)
        got[mode] = [x.cpu().numpy() for x in (grad, img, em, only)]
        assert (block[:offset] == 0).all() and (block[offset + size * size * 4:] == 0).all()
    pt.close()
    (ga, ia, ea, oa), (gb, ib, eb, ob) = got["record"], got["replay"]
    np.testing.assert_array_equal(ia, ib)
    # every term is positive: m float32 additions in any order stay within
    # m * 2^-24 of the exact sum on either side; m is at most 4 reads a vertex
    # of every path, spread over the texels (one texel takes all of its reads)
    assert (ga > 0).any() or depth == 1
    m = max(8.0, 4.0 * w * h * spp * depth / (size * size))
    assert np.abs(ga - gb).max() <= m * 2.0 ** -23 * max(gb.max(), 1e-30)
    # FP64 sums of a thread's runs of float32 terms (runs as long as its trips)
    np.testing.assert_allclose(ea, eb, rtol=1e-5, atol=1e-9)
    np.testing.assert_allclose(oa, eb, rtol=1e-5, atol=1e-9)
