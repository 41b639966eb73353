"""The margin of the tile's conic pretest (trace.cu, make_conic_basis, ray_cone): its magnitude V covers every
term of a tile's directions, and with it no hit is dropped on images smaller than a tile, for every shape
of tile and packet, and for cones of supplied rays."""
import numpy as np
import pytest

from tests.test_conic_pretest import F, camera_rays, conic, cross, dot, hits, keeps

SHAPES = [(8, 16), (16, 8), (4, 8), (8, 4)]
IMAGES = [(1, 1), (1, 40), (37, 1), (2, 3), (3, 1), (5, 5), (9, 33), (64, 48), (1920, 1080)]


def tile_basis(w, fov, tx, ty, tw, th, half, width, height):
    """make_conic_basis for the tile of tw x th pixels at (tx, ty), reaching `half` a pixel further."""
    hx, hy = F(tw - 1) * F(0.5), F(th - 1) * F(0.5)
    cx, cy = F(tx) + hx, F(ty) + hy
    hx, hy = hx + half, hy + half
    vs = F(np.tan(F(fov) / F(2)))
    ax = F(width) / F(height) * vs
    x0 = ax * (F(2) * (cx + F(0.5)) / F(width) - F(1))
    y0 = vs * (F(1) - F(2) * (cy + F(0.5)) / F(height))
    dx, dy = F(2) * ax / F(width), F(-2) * vs / F(height)
    v0 = np.array([w[e] * x0 + w[3 + e] * y0 - w[6 + e] for e in range(3)], F)
    n = [F(np.sqrt(np.sum(w[3 * i:3 * i + 3] ** 2, dtype=F))) for i in range(3)]
    mx = max(F(2) * abs(ax), abs(x0) + hx * abs(dx))
    my = max(F(2) * abs(vs), abs(y0) + hy * abs(dy))
    return v0, w[0:3] * dx, w[3:6] * dy, n[0] * mx + n[1] * my + n[2], hx, hy, cx, cy


def cone_basis(rd):
    """ray_cone for a tile of the caller's rays [n,3]; each ray's place in its plane too."""
    length = np.sqrt(dot(rd, rd))
    m = np.sum(rd / length[:, None], axis=0, dtype=F)
    m = m / F(np.sqrt(np.sum(m * m, dtype=F)))
    u = np.array([0, m[2], -m[1]] if abs(m[0]) < 0.7 else [-m[2], 0, m[0]], F)
    u = u / F(np.sqrt(np.sum(u * u, dtype=F)))
    v = cross(m, u)
    c = dot(rd, np.broadcast_to(m, rd.shape))
    assert (c >= F(0.6) * length).all()
    a, b = dot(rd, np.broadcast_to(u, rd.shape)) / c, dot(rd, np.broadcast_to(v, rd.shape)) / c
    wide = F(4e-6) * (F(1) + max(abs(a.min()), abs(a.max())) + max(abs(b.min()), abs(b.max())))
    a0, a1, b0, b1 = a.min() - wide, a.max() + wide, b.min() - wide, b.max() + wide
    ca, cc = F(0.5) * (a0 + a1), F(0.5) * (b0 + b1)
    v0 = np.array([np.float64(cc) * v[e] + F(np.float64(ca) * u[e] + np.float64(m[e])) for e in range(3)]).astype(F)
    mag = F(2) * (F(1) + max(abs(a0), abs(a1)) + max(abs(b0), abs(b1)))
    return v0, u, v, mag, F(0.5) * (a1 - a0), F(0.5) * (b1 - b0), a - ca, b - cc


def grazing(rd, rng, n, aniso):
    """n Gaussians whose support sphere one of the rays [m,3] grazes: matrices and object-space origins."""
    inv = 10.0 ** rng.uniform(-1, 4, (n, 1)) * 10.0 ** rng.uniform(-aniso / 2, aniso / 2, (n, 3))
    m64 = inv[:, :, None] * np.swapaxes(np.linalg.qr(rng.standard_normal((n, 3, 3)))[0], 1, 2)
    ld = np.einsum("nij,nj->ni", m64, rd[rng.integers(0, rd.shape[0], n)].astype(np.float64))
    side = rng.standard_normal((n, 3))
    side -= (side * ld).sum(1, keepdims=True) * ld / (ld * ld).sum(1, keepdims=True)
    side /= np.linalg.norm(side, axis=1, keepdims=True)
    eps = np.where(np.arange(n) % 3 == 0, 1e-6, np.where(np.arange(n) % 3 == 1, 1e-3, 0.5))
    away = 10.0 ** rng.uniform(-2, 5, (n, 1))
    lo = (-away * ld / np.linalg.norm(ld, axis=1, keepdims=True)
          + (1.0 + eps * rng.uniform(-1, 1, n))[:, None] * side).astype(F)
    return m64.astype(F), lo


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("image", IMAGES)
def test_margin_of_camera_tiles(shape, image):
    (tw, th), (width, height) = shape, image
    rng = np.random.default_rng(tw * 1000 + width)
    accepted = 0
    with np.errstate(all="ignore"):
        for rep in range(24):
            w = np.linalg.qr(rng.standard_normal((3, 3)))[0].astype(F).reshape(-1) * F(rng.choice([1.0, 0.2, 5.0]))
            fov = F(rng.uniform(0.05, 2.6) if rep % 2 else rng.uniform(2.6, 3.0))
            tx, ty = tw * int(rng.integers(0, -(-width // tw))), th * int(rng.integers(0, -(-height // th)))
            half = F(0.5) if rep % 3 == 0 else F(0)
            v0, du, dv, mag, hx, hy, cx, cy = tile_basis(w, fov, tx, ty, tw, th, half, width, height)
            # V is no less than the largest sum of the magnitudes that make up a direction of the tile
            vs = np.tan(np.float64(fov) / 2)
            ax = width / height * vs
            n = [np.linalg.norm(w[3 * i:3 * i + 3].astype(np.float64)) for i in range(3)]
            terms = (n[0] * (abs(ax * (2 * (cx + 0.5) / width - 1)) + hx * 2 * ax / width)
                     + n[1] * (abs(vs * (1 - 2 * (cy + 0.5) / height)) + hy * 2 * vs / height) + n[2])
            assert mag >= terms * (1 - 1e-5) and mag >= (n[0] * 2 * ax + n[1] * 2 * vs + n[2]) * (1 - 1e-5)
            px, py = [g.reshape(-1).astype(F) for g in np.meshgrid(np.arange(tx, tx + tw), np.arange(ty, ty + th))]
            inside = (px < width) & (py < height)
            px, py = px[inside], py[inside]
            if half:
                px = px + (rng.integers(0, 65536, px.size).astype(F) * F(2.0 ** -16) - F(0.5))
                py = py + (rng.integers(0, 65536, py.size).astype(F) * F(2.0 ** -16) - F(0.5))
            rd = camera_rays(w, fov, px, py, width, height)
            m, lo = grazing(rd, rng, 60, float(rep % 5))
            keep, hit = keeps(conic(m, lo, v0, du, dv, mag, hx, hy), px - cx, py - cy), hits(m, lo, rd)
            assert not (hit & ~keep).any(), np.argwhere(hit & ~keep)[:3]
            accepted += hit.sum()
    assert accepted >= 24


@pytest.mark.parametrize("spread", [1e-4, 0.05, 0.6])
@pytest.mark.parametrize("lengths", [False, True])
def test_margin_of_supplied_rays(spread, lengths):
    rng = np.random.default_rng(int(spread * 1e4) + lengths)
    accepted = 0
    with np.errstate(all="ignore"):
        for rep in range(24):
            axis = rng.standard_normal(3)
            axis /= np.linalg.norm(axis)
            d = axis + spread * rng.uniform(-1, 1, (int(rng.integers(1, 129)), 3)) / np.sqrt(3)
            d /= np.linalg.norm(d, axis=1, keepdims=True)
            rd = (d * (2.0 ** rng.uniform(-10, 10, (d.shape[0], 1)) if lengths else 1.0)).astype(F)
            v0, du, dv, mag, hx, hy, x, y = cone_basis(rd)
            m, lo = grazing(rd, rng, 60, float(rep % 5))
            keep, hit = keeps(conic(m, lo, v0, du, dv, mag, hx, hy), x, y), hits(m, lo, rd)
            assert not (hit & ~keep).any(), np.argwhere(hit & ~keep)[:3]
            accepted += hit.sum()
    assert accepted >= 24
