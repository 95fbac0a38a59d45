"""Performance cases: the calls a renderer makes into this package, through its
public classes (``Accelerator``, ``PathTracer``, ``RadianceCache``).

Every case is a dict of plain values; ``prepare`` makes the scene, rays or
samples of one seed on the GPU, ``run`` makes one pass over them.  Kinds:

- ``closest`` / ``shadow``: closest-hit and any-hit casts of device ray buffers,
  half of the closest-hit rays from a camera and half diffuse bounces off what
  those hit (a wavefront's mix), shadow rays from the hits to a point light;
- ``rebuild``: the accelerator built again over a changed scene and the first
  small cast on it;
- ``render`` / ``guided``: frames of the plain and the guided path tracer;
- ``adjoint``: gradients by an albedo texture and by the area-light emission;
- ``query`` / ``train``: the radiance cache's inference and optimisation steps.
"""
import functools
import math
import os

import numpy as np
import torch

from mray_gb300 import scenes, spectral
from mray_gb300.accel import Accelerator
from mray_gb300.cache import WEIGHTS, RadianceCache
from mray_gb300.pt import PathTracer, load_box_scene

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), os.pardir, "tests", "golden")
DEV = "cuda:0"
FAR = 1000.0                  # tMax of the cast rays: beyond every scene here
SKY = (512, 256)              # texels of the skysphere map
NOISE_TEXTURE = 1024          # texels a side of the production scene's textures
CACHE_BOX = (-2.0, -2.0, -2.0, 2.0, 2.0, 2.0)


def listed():
    return [
        # A picking or probe query of an editor or a game: a few hundred rays, the
        # answer wanted at once.  All latency.
        {"name": "closest_probe", "kind": "closest", "level": 5, "instances": 1, "rays": 1000, "watertight": False},
        # The wavefront of a 1080p frame on the instanced 1.31M-triangle stress scene:
        # primaries and one diffuse bounce each.
        {"name": "closest_wavefront", "kind": "closest", "level": 8, "instances": 64, "rays": 3949977,
         "watertight": False},
        # The shadow rays of one wavefront on a mid-size scene.
        {"name": "shadow_wavefront", "kind": "shadow", "level": 6, "instances": 27, "rays": 1048575,
         "watertight": False},
        # An edited scene of many small meshes: full rebuild and the first cast.
        {"name": "rebuild_scene", "kind": "rebuild", "level": 2, "meshes": 509, "instances": 509, "rays": 65536},
        # An interactive preview: a thumbnail at one sample per pixel.
        {"name": "render_preview", "kind": "render", "scene": "mixed", "width": 160, "height": 90, "spp": 1, "depth": 5,
         "sampler": "independent", "spectral": False},
        # The box scene at its usual size.
        {"name": "render_box", "kind": "render", "scene": "box", "width": 256, "height": 256, "spp": 16, "depth": 8,
         "sampler": "independent", "spectral": False},
        # Textured materials under the stratified sampler, an odd size.
        {"name": "render_zsobol", "kind": "render", "scene": "textured", "width": 333, "height": 251, "spp": 8,
         "depth": 6, "sampler": "zsobol-owen", "spectral": False},
        # The spectral production scene at 1080p: 509 surfaces, every material, sky and area lights.
        {"name": "render_production", "kind": "render", "scene": "production", "width": 1920, "height": 1080, "spp": 4,
         "depth": 12, "sampler": "independent", "spectral": True},
        # One optimisation step's gradients of a differentiable render.
        {"name": "adjoint_texture", "kind": "adjoint", "texture": 512, "width": 512, "height": 512, "spp": 32,
         "depth": 6},
        # A guided frame from an empty grid: learning while it renders.
        {"name": "guided_box", "kind": "guided", "scene": "box", "width": 256, "height": 256, "spp": 16, "depth": 8},
        # The radiance cache answering one 1080p frame's path ends.
        {"name": "cache_query", "kind": "query", "levels": 16, "log2_table": 19, "samples": 2073600},
        # The cache's online training: a burst of steps, then its parameters read back.
        {"name": "cache_train", "kind": "train", "levels": 16, "log2_table": 19, "samples": 65536, "steps": 8},
    ]


def _spread(rng, lo, hi):
    """A whole number spread over [lo, hi] by its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["closest", "closest", "shadow", "rebuild", "render", "render", "render", "adjoint", "guided",
                       "query", "train"])
    c = {"kind": kind}
    if kind in ("closest", "shadow"):
        c.update(level=rng.randint(2, 8), instances=_spread(rng, 1, 128), rays=_spread(rng, 200, 3900000),
                 watertight=rng.random() < 0.25)
    elif kind == "rebuild":
        level = rng.randint(1, 8)
        meshes = _spread(rng, 1, max(1, min(600, 1400000 // (20 * 4 ** level))))
        c.update(level=level, meshes=meshes, instances=meshes + rng.randint(0, 64), rays=_spread(rng, 1000, 100000))
    elif kind == "render":
        scene = rng.choice(["box", "mixed", "textured", "sky", "production"])
        c.update(scene=scene, width=_spread(rng, 48, 1920), height=_spread(rng, 32, 1080))
        c.update(spp=max(1, min(16, _spread(rng, 1, 16), 8000000 // (c["width"] * c["height"]))), depth=rng.randint(3, 12),
                 sampler=rng.choice(["independent", "independent", "zsobol", "zsobol-owen", "pcg32"]),
                 spectral=rng.random() < 0.4)
    elif kind == "adjoint":
        c.update(texture=_spread(rng, 32, 1024), width=_spread(rng, 64, 512), height=_spread(rng, 64, 512),
                 spp=_spread(rng, 1, 32), depth=rng.randint(2, 6))
    elif kind == "guided":
        c.update(scene=rng.choice(["box", "mixed", "textured"]), width=_spread(rng, 64, 512),
                 height=_spread(rng, 64, 512), spp=_spread(rng, 1, 16), depth=rng.randint(3, 8))
    elif kind == "query":
        c.update(levels=rng.choice([8, 12, 16]), log2_table=rng.randint(14, 19), samples=_spread(rng, 1000, 2073600))
    else:
        c.update(levels=rng.choice([8, 12, 16]), log2_table=rng.randint(14, 19), samples=_spread(rng, 1000, 65536),
                 steps=rng.randint(1, 8))
    return c


# ---------------------------------------------------------------------------
# Scene assets that do not depend on the seed
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _icosphere(level, radius, noise):
    return scenes.icosphere(level, radius, noise, scenes.STRESS_NOISE_FREQ, 0)


@functools.lru_cache(maxsize=None)
def _sky():
    return scenes.sky_map(SKY[0], SKY[1], seed=0)


@functools.lru_cache(maxsize=None)
def _noise(size, seed, f32=False):
    return scenes.value_noise_texture(size, seed, dtype=np.float32 if f32 else np.uint8)


@functools.lru_cache(maxsize=None)
def _uv_sphere():
    return scenes.uv_sphere(128, 256, 0.15, noise=0.03, seed=0)


@functools.lru_cache(maxsize=None)
def _spectral():
    res, lut = spectral.read_mrspectra(os.path.join(GOLDEN, "REC_709_r32.mrspectra"))
    return res, lut, spectral.load_tables(os.path.join(GOLDEN, "spectral_rec709.npz"))


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed & 0x7FFFFFFF)


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


# ---------------------------------------------------------------------------
# Casts
# ---------------------------------------------------------------------------
def _field(case, seed):
    """Mesh and transforms of the instance field (rotations whose inverse every
    mode of the accelerator gets right)."""
    pos, idx = _icosphere(case["level"], scenes.STRESS_RADIUS, scenes.STRESS_NOISE_AMP)
    return pos, idx, scenes.instance_field(case["instances"], seed & 0xFFFF)


def _camera_rays(n, seed, box):
    """n jittered camera rays, row by row, looking at the scene's box."""
    lo, hi = np.asarray(box[:3], np.float64), np.asarray(box[3:], np.float64)
    mid, size = 0.5 * (lo + hi), float((hi - lo).max())
    w = max(1, int(math.sqrt(n * 16.0 / 9.0)))
    h = -(-n // w)
    eye = (mid[0], mid[1], mid[2] - 1.4 * size)
    rays = scenes.primary_rays(w, h, seed=seed & 0xFFFF, eye=eye, target=tuple(mid))[:n]
    rays[:, 7] = FAR
    return _cuda(rays)


def _surface_points(acc, rays, pos, idx, m34):
    """World points and unit normals (towards the ray) where `rays` hit."""
    n = rays.shape[0]
    work = rays.clone()
    hits = torch.full((n, 4), -1, dtype=torch.int32, device=DEV)
    meta = torch.zeros((n, 2), dtype=torch.float32, device=DEV)
    acc.cast_rays(work, hits, meta)
    got = (hits[:, 0] != -1).nonzero().flatten()
    r, h = work[got].double(), hits[got]
    m = _cuda(m34).double().reshape(-1, 3, 4)[h[:, 2].long()]
    tri = _cuda(pos).double()[_cuda(idx.astype(np.int64))[h[:, 0].long()]]
    nl = torch.linalg.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
    nw = torch.einsum("nij,nj->ni", m[:, :, :3], nl)
    nw = nw / nw.norm(dim=1, keepdim=True)
    nw = torch.where(((nw * r[:, 4:7]).sum(1, keepdim=True) > 0.0), -nw, nw)
    return r[:, 0:3] + r[:, 4:7] * r[:, 7:8], nw


def _prepare_cast(case, seed):
    pos, idx, m34 = _field(case, seed)
    acc = Accelerator(0, watertight=case["watertight"])
    mesh = acc.upload_mesh(pos, idx)
    for i in range(m34.shape[0]):
        acc.add_instance(mesh, m34[i], trans_key=i, accel_key=i)
    acc.construct()
    n, gen = case["rays"], _generator(seed)
    box = acc.scene_aabb()
    shadow = case["kind"] == "shadow"
    first = _camera_rays(n if shadow else (n + 1) // 2, seed, box)
    pts, nrm = _surface_points(acc, first, pos, idx, m34)
    if pts.shape[0] == 0:
        pts, nrm = first[:1, 0:3].double(), -first[:1, 4:7].double()
    k = torch.arange(n if shadow else n - first.shape[0], device=DEV) % pts.shape[0]
    rest = torch.zeros((k.numel(), 8), dtype=torch.float32, device=DEV)
    org = pts[k] + 2e-3 * nrm[k]
    if shadow:
        light = torch.tensor([0.5 * (box[0] + box[3]), box[4] + 0.3 * (box[4] - box[1]) + 5.0, box[2] - 5.0], device=DEV,
                             dtype=torch.float64)
        d = light + torch.rand((k.numel(), 3), generator=gen, device=DEV, dtype=torch.float64) - org
        rest[:, 7] = d.norm(dim=1) * 0.999
    else:
        d = torch.randn((k.numel(), 3), generator=gen, device=DEV, dtype=torch.float64)
        d = d / d.norm(dim=1, keepdim=True) + nrm[k] * 1.001
        rest[:, 7] = FAR
    rest[:, 0:3] = org
    rest[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    rest[:, 3] = 1e-4
    rays = rest if shadow else torch.cat([first, rest])
    state = {"acc": acc, "rays": rays.contiguous()}
    if shadow:
        state["bits"] = torch.zeros((n + 31) // 32, dtype=torch.int32, device=DEV)
    else:
        state["hits"] = torch.full((n, 4), -1, dtype=torch.int32, device=DEV)
        state["meta"] = torch.zeros((n, 2), dtype=torch.float32, device=DEV)
    return state


def _run_closest(s):
    s["rays"][:, 7].fill_(FAR)              # a cast shortens tMax to the hit
    s["acc"].cast_rays(s["rays"], s["hits"], s["meta"])
    return {"rays": s["rays"], "hits": s["hits"], "meta": s["meta"]}


def _run_shadow(s):
    s["acc"].cast_visibility_rays(s["bits"], s["rays"])
    return {"visible": s["bits"]}


def _exact_closest(case, seed):
    """Every ray against every triangle in 64 bits (rays moved into each instance's space)."""
    pos, idx, m34 = _field(case, seed)
    if case["rays"] * idx.shape[0] * m34.shape[0] > 6e9:
        return None
    rays = _prepare_cast(case, seed)["rays"]
    out = rays.double()
    meta = torch.zeros((rays.shape[0], 2), dtype=torch.float64, device=DEV)
    tri = _cuda(pos).double()[_cuda(idx.astype(np.int64))]
    v0, e0, e1 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    nrm = torch.linalg.cross(e0, e1)
    step = max(1, 20000000 // idx.shape[0])
    for i in range(m34.shape[0]):
        m = _cuda(m34[i]).double().reshape(3, 4)
        inv = torch.linalg.inv(m[:, :3])
        for b in range(0, rays.shape[0], step):
            o = (out[b:b + step, 0:3] - m[:, 3]) @ inv.T
            d = out[b:b + step, 4:7] @ inv.T
            # Cramer: t, u, v of o + t d = v0 + u e0 + v e1 (front faces only)
            det = -(d @ nrm.T)
            c = torch.linalg.cross(o, d)
            t = (o @ nrm.T - (v0 * nrm).sum(1)) / det
            u = (c @ e1.T - d @ torch.linalg.cross(e1, v0).T) / det
            v = (d @ torch.linalg.cross(e0, v0).T - c @ e0.T) / det
            ok = (det > 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= out[b:b + step, 3:4]) & (t < out[b:b + step, 7:8])
            t = torch.where(ok, t, torch.full_like(t, float("inf")))
            best, at = t.min(dim=1)
            hit = torch.isfinite(best)
            uu, vv = (x.gather(1, at[:, None])[:, 0] for x in (u, v))
            out[b:b + step, 7] = torch.where(hit, best, out[b:b + step, 7])
            meta[b:b + step] = torch.where(hit[:, None], torch.stack([1.0 - uu - vv, uu], 1), meta[b:b + step])
    return {"rays": out, "hits": None, "meta": meta}


# ---------------------------------------------------------------------------
# Rebuild
# ---------------------------------------------------------------------------
def _prepare_rebuild(case, seed):
    rng = np.random.default_rng(seed)
    pos, idx = _icosphere(case["level"], 1.0, 0.0)
    m34 = scenes.instance_field(case["instances"], seed & 0xFFFF)
    acc = Accelerator(0)
    for k in range(case["meshes"]):
        # every mesh its own shape
        acc.upload_mesh(pos * rng.uniform(0.5, 4.0, 3).astype(np.float32) +
                        rng.normal(0.0, 0.01, pos.shape).astype(np.float32), idx, prim_key_base=k * idx.shape[0])
    for i in range(case["instances"]):
        acc.add_instance(i % case["meshes"], m34[i], trans_key=i, accel_key=i)
    n = case["rays"]
    return {"acc": acc, "rays": _camera_rays(n, seed, (-50.0, -50.0, -50.0, 50.0, 50.0, 50.0)),
            "hits": torch.full((n, 4), -1, dtype=torch.int32, device=DEV),
            "meta": torch.zeros((n, 2), dtype=torch.float32, device=DEV)}


def _run_rebuild(s):
    s["acc"].construct()
    return dict(_run_closest(s), box=s["acc"].scene_aabb())


# ---------------------------------------------------------------------------
# Path tracing
# ---------------------------------------------------------------------------
def _scene(case, seed):
    """Surfaces and camera of a path-traced scene."""
    name, cam = case["scene"], scenes.box_camera()
    s = seed & 0xFFFF
    if name == "box":
        return scenes.box_scene(s), cam
    if name == "mixed":
        return scenes.box_scene_mixed(s), cam
    if name == "sky":
        return scenes.sky_scene(s), cam
    if name == "textured":
        surf = scenes.box_scene(s)
        for k, t in ((0, 0), (2, 1), (3, 0)):
            surf[k].update(uv=scenes.quad_uv() * 2.0, texture=_noise(256, t))
        return scenes.mipmapped(surf), cam
    surf, cam = scenes.c2_scene(s, texture_size=16)
    for k, x in enumerate(surf):
        if x.get("texture") is not None:
            x["texture"] = _noise(NOISE_TEXTURE, 17 + k % 2)
    return scenes.mipmapped(surf), cam


def _prepare_render(case, seed):
    surf, cam = _scene(case, seed)
    pt = PathTracer(0)
    load_box_scene(pt, surf)
    if case["scene"] in ("sky", "production"):
        pt.set_env(_sky())
    if case.get("spectral"):
        pt.set_spectral(*_spectral())
    p = PathTracer.params(case["width"], case["height"], case["spp"], cam, max_depth=case["depth"], rr_start=3,
                          seed=seed & 0x7FFFFFFF, sampler=case.get("sampler", "independent"),
                          samples_per_pass=case["spp"] if case["kind"] == "guided" else 0)
    if case["kind"] == "guided":
        pt.guide_create()
    return {"pt": pt, "params": p}


def _run_render(s):
    return s["pt"].render(s["params"])


def _run_guided(s):
    s["pt"].guide_clear()                   # StartRender: learning begins anew
    return s["pt"].render_guided(s["params"])


def _prepare_adjoint(case, seed):
    s, gen = seed & 0xFFFF, _generator(seed)
    surf = scenes.box_scene(s)
    pos, idx, uv = _uv_sphere()
    m = np.array([1, 0, 0, 0.35, 0, 1, 0, 0.2, 0, 0, 1, 0.25], np.float32)
    surf.insert(len(surf) - 1, dict(pos=pos, idx=idx, uv=uv, m34=m, kind="lambert", albedo=[0.5] * 3, cull=False))
    pt = PathTracer(0)
    for x in surf:
        inst = pt.add_surface(x["pos"], x["idx"], x["m34"], cull=x.get("cull", True), uv=x.get("uv"))
        if x["kind"] == "light":
            pt.set_area_light(inst, x["radiance"])
        else:
            pt.set_lambert(inst, x["albedo"])
        if "uv" in x:
            sphere = inst
    t = case["texture"]
    tex = _cuda(_noise(t, 5, True)) * (0.5 + 0.5 * torch.rand((t, t, 4), generator=gen, device=DEV))
    tid = pt.add_texture(tex.contiguous())
    pt.set_albedo_texture(sphere, tid)
    pt.build()
    p = PathTracer.params(case["width"], case["height"], case["spp"], scenes.box_camera(), max_depth=case["depth"],
                          rr_start=case["depth"], seed=seed & 0x7FFFFFFF)
    delta = torch.randn((case["height"], case["width"], 4), generator=gen, device=DEV) * 1e-5 + 2e-5
    return {"pt": pt, "params": p, "tex": tid, "size": t, "delta": delta}


def _run_adjoint(s):
    pt, p = s["pt"], s["params"]
    image = torch.zeros((p.height, p.width, 4), device=DEV)
    emission = torch.zeros((pt.n_instances, 4), device=DEV)
    grad = pt.adjoint(p, s["tex"], s["delta"], image=image, grad_emission=emission)
    return {"image": image, "texture": grad, "emission": emission}


# ---------------------------------------------------------------------------
# Radiance cache
# ---------------------------------------------------------------------------
def _samples(n, gen):
    """Path ends on 48 spheres in the cache's box, in no order: position and
    roughness, direction, normal, albedo."""
    def unit(k):
        d = torch.randn((k, 3), generator=gen, device=DEV)
        return d / d.norm(dim=1, keepdim=True)
    x = torch.zeros((n, 16), device=DEV)
    mid = torch.rand((48, 3), generator=gen, device=DEV) * 3.0 - 1.5
    rad = torch.rand(48, generator=gen, device=DEV) * 0.4 + 0.05
    k = torch.randint(0, 48, (n,), generator=gen, device=DEV)
    nrm = unit(n)
    x[:, 0:3] = mid[k] + nrm * rad[k][:, None]
    x[:, 3] = torch.rand(n, generator=gen, device=DEV)
    x[:, 4:7] = unit(n)
    x[:, 8:11] = nrm
    x[:, 12:15] = torch.rand((48, 3), generator=gen, device=DEV)[k] * 0.8 + 0.1
    return x


def _cache_params(case, seed):
    gen = torch.Generator().manual_seed(seed & 0x7FFFFFFF)
    w = (torch.rand(WEIGHTS, generator=gen) * 2.0 - 1.0) * 0.25
    t = ((torch.rand(case["levels"] * 2 << case["log2_table"], generator=gen) * 2.0 - 1.0) * 0.5).half().float()
    return w.numpy(), t.numpy()


def _prepare_cache(case, seed):
    acc = Accelerator(0)
    train = case["kind"] == "train"
    cache = RadianceCache(owner=acc, levels=case["levels"], log2_table_size=case["log2_table"],
                          learning_rate=1e-3 if train else 1e-2, epsilon=1e-8 if train else 1e-15,
                          max_batch=65536, seed=seed & 0x7FFFFFFF, aabb=CACHE_BOX)
    n, gen = case["samples"], _generator(seed)
    state = {"cache": cache}
    if train:
        x = _samples(n * case["steps"], gen)
        # a smooth field of position and direction, as radiance on surfaces is
        y = torch.zeros((x.shape[0], 4), device=DEV)
        for c in range(3):
            y[:, c] = (1.5 + torch.sin(3.0 * x[:, c] + c) + 0.3 * x[:, 4 + c]) * x[:, 12 + c]
        state.update(x=list(x.split(n)), y=list(y.split(n)))
    else:
        cache.set_params(*_cache_params(case, seed))
        state.update(x=_samples(n, gen))
    return state


def _run_query(s):
    return s["cache"].query(s["x"])


def _run_train(s):
    c = s["cache"]
    for x, y in zip(s["x"], s["y"]):
        c.train(x, y, loss=False)
    weights, table = c.get_params()
    return {"weights": weights, "table": table}


def _exact_query(case, seed):
    """The hash-grid encoding and the MLP in 64 bits."""
    w, t = _cache_params(case, seed)
    x = _samples(case["samples"], _generator(seed))
    w, table = _cuda(w).double(), _cuda(t).double().reshape(case["levels"], -1, 2)
    mats = [w[4096 * i:4096 * (i + 1)].reshape(64, 64) for i in range(5)] + [w[5 * 4096:].reshape(16, 64)]
    size, levels = 1 << case["log2_table"], case["levels"]
    grow = (math.log2(2048.0) - math.log2(16.0)) / (levels - 1)
    scale = [float(np.float32(2.0 ** (l * grow) * 16.0 - 1.0)) for l in range(levels)]
    lo = torch.tensor(CACHE_BOX[:3], device=DEV, dtype=torch.float64)
    ext = torch.tensor(CACHE_BOX[3:], device=DEV, dtype=torch.float64) - lo
    outs = []
    for xs in x.split(1 << 18):
        xd = xs.double()
        u = ((xd[:, 0:3] - lo) / ext).clamp(0.0, 1.0)
        f = torch.zeros((xd.shape[0], 64), dtype=torch.float64, device=DEV)
        for l in range(levels):
            p = u * scale[l] + 0.5
            b = p.floor()
            r, b, res = p - b, b.long(), int(math.ceil(scale[l])) + 2
            for c in range(8):
                o = (c & 1, c >> 1 & 1, c >> 2 & 1)
                q = [b[:, k] + o[k] for k in range(3)]
                if res ** 3 <= size:
                    at = (q[0] + q[1] * res + q[2] * res * res) & (size - 1)
                else:
                    at = (q[0] ^ (q[1] * 2654435761) ^ (q[2] * 805459861)) & (size - 1)
                weight = torch.ones_like(r[:, 0])
                for k in range(3):
                    weight = weight * (r[:, k] if o[k] else 1.0 - r[:, k])
                f[:, 2 * l:2 * l + 2] += weight[:, None] * table[l][at]
        dx, dy, dz = xd[:, 4], xd[:, 5], xd[:, 6]
        xx, yy, zz = dx * dx, dy * dy, dz * dz
        f[:, 32:48] = torch.stack([
            torch.full_like(dx, 0.5 / math.sqrt(math.pi)), -0.4886025119029199 * dy, 0.4886025119029199 * dz,
            -0.4886025119029199 * dx, 1.0925484305920792 * dx * dy, -1.0925484305920792 * dy * dz,
            0.94617469575756 * zz - 0.31539156525252, -1.0925484305920792 * dx * dz, 0.5462742152960396 * (xx - yy),
            0.5900435899266435 * dy * (yy - 3.0 * xx), 2.890611442640554 * dx * dy * dz,
            0.4570457994644657 * dy * (1.0 - 5.0 * zz), 0.3731763325901154 * dz * (5.0 * zz - 3.0),
            0.4570457994644657 * dx * (1.0 - 5.0 * zz), 1.445305721320277 * dz * (xx - yy),
            0.5900435899266435 * dx * (3.0 * yy - xx)], 1)
        f[:, 48:51] = (xd[:, 8:11] + 1.0) * 0.5
        f[:, 51:54] = xd[:, 12:15]
        f[:, 54] = xd[:, 3]
        f[:, 55] = 1.0
        for m in mats[:-1]:
            f = (f @ m.T).clamp_min(0.0)
        y = f @ mats[-1].T
        outs.append(torch.cat([y[:, :3], torch.zeros_like(y[:, :1])], 1))
    return torch.cat(outs)


# ---------------------------------------------------------------------------
_PREPARE = {"closest": _prepare_cast, "shadow": _prepare_cast, "rebuild": _prepare_rebuild, "render": _prepare_render,
            "guided": _prepare_render, "adjoint": _prepare_adjoint, "query": _prepare_cache, "train": _prepare_cache}
_RUN = {"closest": _run_closest, "shadow": _run_shadow, "rebuild": _run_rebuild, "render": _run_render,
        "guided": _run_guided, "adjoint": _run_adjoint, "query": _run_query, "train": _run_train}


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state["kind"] = case["kind"]
    return state


def run(state):
    return _RUN[state["kind"]](state)


def exact(case, seed):
    if case["kind"] == "closest":
        return _exact_closest(case, seed)
    if case["kind"] == "query":
        return _exact_query(case, seed)
    return None             # images, gradients and training: no independent 64-bit path tracer or optimiser here


def work(case):
    """Bytes: each input read once, each output written once.  Operations: a ray
    has to be moved into an instance (33) and tested against one triangle (48);
    a path vertex costs about 250 more for its surface, light and BxDF sample,
    two rays each, and four vertices stand for a path; a cache sample is its
    MLP's products and 16 x 8 table reads."""
    kind = case["kind"]
    if kind in ("closest", "shadow", "rebuild"):
        tris = 20 * 4 ** case["level"] * case.get("meshes", 1)
        geometry = tris * 18 + 48 * case["instances"]            # vertices (half as many as triangles) and indices
        if kind == "rebuild":
            return {"bytes": geometry + case["rays"] * 60, "flops": tris * 100 + case["rays"] * 81}
        per_ray = 60 if kind == "closest" else 32.125
        return {"bytes": geometry + case["rays"] * per_ray, "flops": case["rays"] * 81}
    if kind in ("render", "guided", "adjoint"):
        pixels = case["width"] * case["height"]
        paths = pixels * case["spp"]
        flops = paths * min(case["depth"], 4) * (250 + 2 * 81)
        if kind == "adjoint":
            return {"bytes": pixels * 32 + case["texture"] ** 2 * 32, "flops": 2 * flops}
        return {"bytes": pixels * 16, "flops": flops}
    mlp = 2 * WEIGHTS
    table = case["levels"] * 2 << case["log2_table"]
    if kind == "query":
        return {"bytes": case["samples"] * (64 + 16) + min(2 * table, case["samples"] * case["levels"] * 32),
                "flops": case["samples"] * (mlp + case["levels"] * 40)}
    n = case["samples"] * case["steps"]
    # parameters, two moments and the half-precision copy of what a step touches, and the read-back
    touched = min(table, case["samples"] * case["levels"] * 16)
    return {"bytes": n * 80 + case["steps"] * touched * 26 + table * 4, "flops": n * 3 * mlp}
