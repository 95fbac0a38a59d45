"""Shading takes more blocks an SM from 2^20 paths a pass on, and appends to its
lists by block: the split into passes changes neither image nor gradients."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


@pytest.mark.parametrize("spectral", [False, True])
def test_large_passes_render_the_same(spectral):
    from mray_gb300 import scenes
    from mray_gb300 import spectral as sp
    from mray_gb300.pt import PathTracer, load_box_scene
    pt = PathTracer(0)
    load_box_scene(pt, scenes.box_scene_mixed(3))
    if spectral:
        res, lut = sp.read_mrspectra(os.path.join(GOLDEN, "REC_709_r32.mrspectra"))
        pt.set_spectral(res, lut, sp.load_tables(os.path.join(GOLDEN, "spectral_rec709.npz")))
    w, h, spp = 331, 397, 9                       # 131,407 paths a sample
    img = {}
    for per_pass in (1, 7, 8, 9):                 # 8 samples are the first pass over 2^20
        p = PathTracer.params(w, h, spp, scenes.box_camera(), max_depth=5, rr_start=2, seed=11, samples_per_pass=per_pass)
        img[per_pass] = pt.render(p).cpu().numpy()
    for per_pass in (7, 8, 9):
        np.testing.assert_array_equal(img[per_pass], img[1])
    pt.close()


def test_large_passes_have_the_same_gradients():
    import torch
    from mray_gb300 import scenes
    from mray_gb300.pt import PathTracer
    from test_gpu_adjoint_records import _tracer
    size, w, h, spp, depth = 16, 331, 397, 9, 4
    tex = torch.from_numpy(scenes.value_noise_texture(64, seed=2, dtype=np.float32)[:size, :size].copy()).cuda()
    pt, tid = _tracer(tex)
    delta = torch.full((h, w, 4), 1e-3, device="cuda")
    out = {}
    for per_pass in (1, 9):
        p = PathTracer.params(w, h, spp, scenes.box_camera(), max_depth=depth, rr_start=3, seed=4, samples_per_pass=per_pass)
        grad = torch.zeros((size, size, 4), device="cuda")
        em, img = torch.zeros((pt.n_instances, 4), device="cuda"), torch.zeros((h, w, 4), device="cuda")
        pt.adjoint(p, tid, delta, grad=grad, image=img, grad_emission=em)
        out[per_pass] = [x.cpu().numpy() for x in (grad, img, em)]
    pt.close()
    (ga, ia, ea), (gb, ib, eb) = out[1], out[9]
    np.testing.assert_array_equal(ia, ib)
    # terms of one sign, m of them on a texel at most: either side's rounding is within m * 2^-24
    assert (ga > 0).any()
    m = 4.0 * w * h * spp * depth / (size * size)
    assert np.abs(ga - gb).max() <= m * 2.0 ** -23 * gb.max()
    # FP64 sums of runs of float32 terms, as many as a thread's trips
    np.testing.assert_allclose(ea, eb, rtol=1e-5, atol=1e-9)
