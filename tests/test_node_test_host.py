"""The traversal's half-precision node test (traverse.cu: intersect_node) never
culls a child box that the ray meets: numpy restates the builder's plane
quantisation and the test, halves rounded as the GPU rounds them, and a
64-bit slab test of the boxes before padding decides."""
import numpy as np
import pytest

F = np.float32


def f16(x):
    with np.errstate(over="ignore", invalid="ignore"):
        return np.asarray(x, np.float64).astype(np.float16)


def quantise(lo, hi, inflate):
    """Per axis: frame origin, 2^e and the children's padded plane bytes (bvh_build.cu: k_collapse)."""
    nlo = np.nextafter((lo.min(0) - F(inflate)).astype(F), F(-np.inf))
    nhi = np.nextafter((hi.max(0) + F(inflate)).astype(F), F(np.inf))
    ext = np.nextafter((nhi - nlo).astype(F), F(np.inf))
    e = np.ceil(np.log2(np.maximum(ext.astype(np.float64) / 252.0, 2.0 ** -126)))
    e = np.where(2.0 ** e * 252.0 < ext, e + 1, e)
    step = (2.0 ** e).astype(F)
    p = np.nextafter((nlo - step).astype(F), F(-np.inf))
    qlo = np.floor((lo.astype(np.float64) - inflate - p) / step) - 1.0
    qhi = np.ceil((hi.astype(np.float64) + inflate - p) / step) + 1.0
    return p, step, np.clip(qlo, 0, 255), np.clip(qhi, 0, 255)


def half_test(p, step, qlo, qhi, o, d, tmin, tmax):
    """intersect_node's decision for every child (fp32 steps in fp32, fmas as one rounding)."""
    with np.errstate(all="ignore"):
        dd = np.where(np.abs(d) > 1e-20, d, np.copysign(F(1e-20), d)).astype(F)
        i = (F(1.0) / dd).astype(F)
        s = (step * i).astype(F)
        a = ((p - o).astype(F) * i).astype(F)
        t0 = max(np.minimum(a, (a + 256.0 * s.astype(np.float64)).astype(F)).max(), F(tmin))
        rate = F(1.0) / max(np.abs(s).min(), F(1e-37))
        g, gt = F(4.0) * rate, F(2.0 ** -22) * rate
        S, A = (s * g).astype(F), ((a - t0).astype(F) * gt).astype(F)
        if np.abs(S).max() > 65504.0:
            c = np.minimum(F(1.0), F(65504.0) / np.abs(S)).astype(F)
            S, A = (S * c).astype(F), (A * c).astype(F)
        S, A = f16(S).astype(np.float64), f16(A).astype(np.float64)
        end = f16(np.float64(F(tmax) - t0) * np.float64(gt * F(1.0009765625)) + 2.0 ** -24)
        near = np.where(d < 0, qhi, qlo) * 2.0 ** -24
        far = np.where(d < 0, qlo, qhi) * 2.0 ** -24
        tn, tf = f16(near * S + A), f16(far * S + A)
        as_int = lambda h: h.view(np.int16)  # noqa: E731  (the packed min / max compare the bits)
        n = np.maximum(as_int(tn).max(1), 0).astype(np.int16).view(np.float16)
        f = np.minimum(as_int(tf).min(1), as_int(np.array([end]))[0]).astype(np.int16).view(np.float16)
        return n <= f


def exact_test(lo, hi, o, d, tmin, tmax):
    o, d = o.astype(np.float64), d.astype(np.float64)
    n, f = np.full(len(lo), float(tmin)), np.full(len(lo), float(tmax))
    for k in range(3):
        if d[k] == 0.0:
            inside = (o[k] >= lo[:, k]) & (o[k] <= hi[:, k])
            f = np.where(inside, f, -np.inf)
            continue
        t = np.stack([(lo[:, k].astype(np.float64) - o[k]) / d[k], (hi[:, k].astype(np.float64) - o[k]) / d[k]])
        n, f = np.maximum(n, t.min(0)), np.minimum(f, t.max(0))
    return n <= f


@pytest.mark.parametrize("kind", ["plain", "flat", "thin_ray", "axis_ray", "inside", "far", "tiny", "huge", "shrunk"])
def test_no_child_is_lost(kind):
    rng = np.random.default_rng(sum(map(ord, kind)))
    seen = 0
    for _ in range(1500):
        scale = {"tiny": 1e-4, "huge": 1e4}.get(kind, 1.0) * 10.0 ** rng.uniform(-1, 1)
        mid = rng.uniform(-1, 1, 3) * scale * (3.0 if kind != "far" else 50.0)
        lo = (mid + rng.uniform(-1, 1, (8, 3)) * scale).astype(F)
        size = rng.uniform(0, 0.5, (8, 3)) * scale
        if kind == "flat":
            k = rng.integers(3)
            lo[:, k] = F(mid[k])
            size[:, k] = 0.0
        hi = (lo + size.astype(F)).astype(F)
        extent = max(np.abs(lo).max(), np.abs(hi).max(), (hi.max(0) - lo.min(0)).max())
        p, step, qlo, qhi = quantise(lo, hi, float(extent) * 1e-5)
        # aim at a point of one of the boxes: corners and edges among them
        c = rng.integers(8)
        w = np.where(rng.random(3) < 0.3, rng.integers(0, 2, 3), rng.random(3))
        target = lo[c].astype(np.float64) * (1 - w) + hi[c].astype(np.float64) * w
        if kind == "inside":
            o = (target + rng.uniform(-0.2, 0.2, 3) * scale).astype(F)
        else:
            o = (mid + rng.normal(size=3) * scale * (4.0 if kind != "far" else 300.0)).astype(F)
        d = target - o
        if kind == "thin_ray":                 # components that differ by up to seven decades
            d = rng.choice([-1.0, 1.0], 3) * 10.0 ** rng.uniform(-7, 0, 3)
            o = (target - d / np.linalg.norm(d) * scale * rng.uniform(0, 5)).astype(F)
        if kind == "axis_ray":
            k = rng.integers(3)
            d[:] = 0.0
            d[k] = 1.0
            o = (target - d * scale * rng.uniform(0, 5)).astype(F)
        nrm = np.linalg.norm(d)
        if nrm == 0.0:
            continue
        d = (d / nrm * (10.0 ** rng.uniform(-2, 2))).astype(F)
        tmax = 3.4e38 if kind != "shrunk" else float(np.linalg.norm(target - o) / np.linalg.norm(d)) * rng.uniform(0.9, 1.1)
        tmin = 0.0 if rng.random() < 0.5 else 1e-4
        need = exact_test(lo, hi, o, d, tmin, tmax)
        got = half_test(p, step, qlo, qhi, o, d, tmin, tmax)
        assert not (need & ~got).any(), (kind, lo, hi, o, d)
        seen += int(need.sum())
    assert seen > 800
