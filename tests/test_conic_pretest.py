"""The tile's conic pretest (trace.cu, conic_coefficients): a CPU restatement in float32, operation by
operation, never drops a ray that the intersection program's hit decision accepts."""
import math

import numpy as np
import pytest

F = np.float32


def fma(a, b, c):
    return (np.float64(a) * np.float64(b) + np.float64(c)).astype(F)


def dot(a, b):
    """fma chain over the last axis, as fdot3."""
    return fma(a[..., 2], b[..., 2], fma(a[..., 1], b[..., 1], a[..., 0] * b[..., 0]))


def cross(a, b):
    def part(i, j):
        return fma(a[..., i], b[..., j], -(a[..., j] * b[..., i]))
    return np.stack([part(1, 2), part(2, 0), part(0, 1)], -1)


def norm(a):
    return np.sqrt(dot(a, a))


def camera_rays(w, fov, fx, fy, width, height):
    """camera_ray at the (possibly jittered) pixel positions fx, fy."""
    vs = F(np.tan(F(fov) / F(2)))
    aspect = F(width) / F(height)
    y = vs * (F(1) - F(2) * (fy + F(0.5)) / F(height))
    x = aspect * vs * (F(2) * (fx + F(0.5)) / F(width) - F(1))
    v = np.stack([w[e] * x + w[3 + e] * y - w[6 + e] for e in range(3)], -1)
    inv = F(1) / np.sqrt(v[..., 0] * v[..., 0] + v[..., 1] * v[..., 1] + v[..., 2] * v[..., 2])
    return v * inv[..., None]


def basis(w, fov, cx, cy, width, height):
    vs = F(np.tan(F(fov) / F(2)))
    ax = F(width) / F(height) * vs
    x0 = ax * (F(2) * (F(cx) + F(0.5)) / F(width) - F(1))
    y0 = vs * (F(1) - F(2) * (F(cy) + F(0.5)) / F(height))
    v0 = np.array([w[e] * x0 + w[3 + e] * y0 - w[6 + e] for e in range(3)], F)
    du = w[0:3] * (F(2) * ax / F(width))
    dv = w[3:6] * (F(-2) * vs / F(height))
    n = [F(np.sqrt(np.sum(w[3 * i:3 * i + 3] ** 2, dtype=F))) for i in range(3)]
    return v0, du, dv, F(2) * (n[0] * abs(ax) + n[1] * abs(vs)) + n[2]


def conic(m, lo, v0, du, dv, mag, hx, hy):
    """The six coefficients per candidate: m [n,3,3], lo [n,3]."""
    def rows(v):
        return np.stack([dot(m[:, i], np.broadcast_to(v, lo.shape)) for i in range(3)], -1)
    l0, lu, lv = rows(v0), rows(du), rows(dv)
    c0, cu, cv = cross(lo, l0), cross(lo, lu), cross(lo, lv)
    lm = fma(hy, norm(lv), fma(hx, norm(lu), norm(l0)))
    cm = fma(hy, norm(cv), fma(hx, norm(cu), norm(c0)))
    mf = np.sqrt(np.sum(m * m, axis=(1, 2), dtype=F))
    nl = norm(lo)
    eta = F(2.0 ** -18) * (nl + F(1)) * mf * mag
    margin = fma(eta, fma(F(2.1), lm, eta), F(1.5 * 2.0 ** -19) * fma(lm, lm, cm * cm))
    ok = (lm >= 2.0 ** -50) & (lm <= 2.0 ** 50) & (cm <= 2.0 ** 50) & (nl <= 2.0 ** 40) & (eta <= 2.0 ** 50)
    q = [(dot(l0, l0) - dot(c0, c0)) + margin, F(2) * (dot(l0, lu) - dot(c0, cu)), F(2) * (dot(l0, lv) - dot(c0, cv)),
         dot(lu, lu) - dot(cu, cu), F(2) * (dot(lu, lv) - dot(cu, cv)), dot(lv, lv) - dot(cv, cv)]
    return [np.where(ok, a, F(np.inf) if i == 0 else F(0)) for i, a in enumerate(q)]


def keeps(q, x, y):
    """Sign bit of h clear, NaN included, for every (candidate, ray)."""
    f, d, e, a, b, c = [v[:, None] for v in q]
    h = fma(x, a, d)
    h = fma(y, b, h)
    h = fma(x, h, f)
    h = fma(y, fma(y, c, e), h)
    return ~np.signbit(h) | np.isnan(h)


def hits(m, lo, rd):
    """The intersection program's decision (intersect_lo) for every (candidate, ray)."""
    ld = np.stack([dot(np.broadcast_to(m[:, None, i], (m.shape[0],) + rd.shape), np.broadcast_to(rd, (m.shape[0],) + rd.shape))
                   for i in range(3)], -1)
    o = np.broadcast_to(lo[:, None], ld.shape)
    b = dot(o, ld)
    t = -b / dot(ld, ld)
    u = np.stack([fma(t, ld[..., k], o[..., k]) for k in range(3)], -1)
    return ~(b > 0) & ~(dot(u, u) > 1)


@pytest.mark.parametrize("size", [(1, 1), (7, 5), (64, 48), (1920, 1080), (3840, 2160)])
@pytest.mark.parametrize("aniso", [0.0, 1.0, 4.0])
@pytest.mark.parametrize("jitter", [False, True])
def test_conic_pretest_never_drops_a_hit(size, aniso, jitter):
    """Gaussians whose support sphere the tile's rays graze (within 1e-3 and 1e-6 of it, and well inside
    and outside), at 1e-2 to 1e5 object-space radii from the camera, with axes up to 10^aniso apart."""
    width, height = size
    rng = np.random.default_rng(int(aniso) * 10 + width + jitter)
    tested = kept = accepted = 0
    with np.errstate(all="ignore"):
        for rep in range(12):
            a = np.linalg.qr(rng.standard_normal((3, 3)))[0]
            w = a.astype(F).reshape(-1) * F(1.0 if rep % 3 else rng.uniform(0.2, 5.0))
            fov = F(rng.uniform(0.05, 2.6))
            tx, ty = 8 * int(rng.integers(0, -(-width // 8))), 16 * int(rng.integers(0, -(-height // 16)))
            px, py = [g.reshape(-1).astype(F) for g in np.meshgrid(np.arange(tx, tx + 8), np.arange(ty, ty + 16))]
            inside = (px < width) & (py < height)
            if jitter:
                px = px + (rng.integers(0, 65536, 128).astype(F) * F(2.0 ** -16) - F(0.5))
                py = py + (rng.integers(0, 65536, 128).astype(F) * F(2.0 ** -16) - F(0.5))
            half = F(0.5) if jitter else F(0)
            rd = camera_rays(w, fov, px, py, width, height)
            x, y = px - F(tx) - F(3.5), py - F(ty) - F(7.5)
            v0, du, dv, mag = basis(w, fov, F(tx) + F(3.5), F(ty) + F(7.5), width, height)
            n = 60
            inv = 10.0 ** rng.uniform(-1, 4, (n, 1)) * 10.0 ** rng.uniform(-aniso / 2, aniso / 2, (n, 3))
            rot = np.linalg.qr(rng.standard_normal((n, 3, 3)))[0]
            m64 = inv[:, :, None] * np.swapaxes(rot, 1, 2)
            # a point of the unit sphere's tangent plane to one of the tile's rays, off by eps
            r = rd[rng.integers(0, 128, n)].astype(np.float64)
            ld = np.einsum("nij,nj->ni", m64, r)
            side = rng.standard_normal((n, 3))
            side -= (side * ld).sum(1, keepdims=True) * ld / (ld * ld).sum(1, keepdims=True)
            side /= np.linalg.norm(side, axis=1, keepdims=True)
            eps = np.where(np.arange(n) % 3 == 0, 1e-6, np.where(np.arange(n) % 3 == 1, 1e-3, 0.5))
            away = 10.0 ** rng.uniform(-2, 5, (n, 1))
            lo = (-away * ld / np.linalg.norm(ld, axis=1, keepdims=True)
                  + (1.0 + eps * rng.uniform(-1, 1, n))[:, None] * side).astype(F)
            m = m64.astype(F)
            q = conic(m, lo, v0, du, dv, mag, F(3.5) + half, F(7.5) + half)
            keep, hit = keeps(q, x, y)[:, inside], hits(m, lo, rd)[:, inside]
            assert not (hit & ~keep).any(), np.argwhere(hit & ~keep)[:3]
            tested, kept, accepted = tested + hit.size, kept + keep.sum(), accepted + hit.sum()
    assert accepted >= 12


def test_conic_pretest_keeps_non_finite_and_extreme_candidates():
    w = np.eye(3, dtype=F).reshape(-1)
    v0, du, dv, mag = basis(w, F(0.8), F(35.5), F(39.5), 64, 64)
    special = np.array([np.inf, -np.inf, np.nan, 1e-30, 3e38, 1e25], F)
    m = np.tile(np.eye(3, dtype=F), (54, 1, 1))
    lo = np.tile(np.array([0.1, 0.2, 5.0], F), (54, 1))
    for i in range(54):
        if i % 3 == 0:
            lo[i, (i // 3) % 3] = special[(i // 9) % 6]
        elif i % 3 == 1:
            m[i, (i // 3) % 3, (i // 9) % 3] = special[(i // 9) % 6]
        else:
            m[i] *= special[(i // 9) % 6]
    with np.errstate(all="ignore"):
        px, py = [g.reshape(-1).astype(F) for g in np.meshgrid(np.arange(32, 40), np.arange(32, 48))]
        rd = camera_rays(w, F(0.8), px, py, 64, 64)
        keep = keeps(conic(m, lo, v0, du, dv, mag, F(3.5), F(7.5)), px - F(35.5), py - F(39.5))
        assert not (hits(m, lo, rd) & ~keep).any()


def test_conic_pretest_is_tight_at_the_benchmarks_magnitudes():
    """Gaussians of 0.02 radius and up to 3:1 axes, 4 to 12 units from a 1920x1080 camera: within 2% of
    the accepted pairs are kept in vain."""
    rng = np.random.default_rng(5)
    w = np.eye(3, dtype=F).reshape(-1)
    fov = F(2.0 * math.atan(0.5 * 1080 / (0.75 * 1920)))
    px, py = [g.reshape(-1).astype(F) for g in np.meshgrid(np.arange(960, 968), np.arange(544, 560))]
    rd = camera_rays(w, fov, px, py, 1920, 1080)
    v0, du, dv, mag = basis(w, fov, F(963.5), F(551.5), 1920, 1080)
    n = 3000
    inv = 1.0 / (0.02 * 3.0 ** rng.uniform(-0.5, 0.5, (n, 3)))
    m = (inv[:, :, None] * np.swapaxes(np.linalg.qr(rng.standard_normal((n, 3, 3)))[0], 1, 2)).astype(F)
    centre = rd[60].astype(np.float64) * rng.uniform(4.0, 12.0, (n, 1)) + 0.03 * rng.standard_normal((n, 3))
    lo = np.einsum("nij,nj->ni", m.astype(np.float64), -centre).astype(F)
    keep = keeps(conic(m, lo, v0, du, dv, mag, F(3.5), F(7.5)), px - F(963.5), py - F(551.5))
    hit = hits(m, lo, rd)
    assert hit.sum() > 50_000 and (keep & ~hit).sum() <= 0.02 * hit.sum(), (hit.sum(), (keep & ~hit).sum())
