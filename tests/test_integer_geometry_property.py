"""The integer form of the fused kernel's geometry, restated in numpy: wherever it decides a deposit
(inside the voxel or not, hit or miss, which sphere), the FP64 arithmetic decides the same.

Covers lattices from one sphere to 2^21 per axis, shifts over the whole range, random deposits and
deposits placed at and around the radii, the cell faces and the voxel's faces. The share of
deposits that it leaves to FP64 stays small on the lattices of the benchmark configurations."""
import numpy as np
import pytest

F32 = np.float32


def _geometry(hl, d):
    n = int(np.floor(2 * hl / d))
    length = n * d
    h = length / 2
    if d / 2 > h:
        n, h, length = 1, d / 2, d
    return n, h, length, -h + d / 2


def _setup(n, d):
    s = 22
    while s > 0 and (n << s) > (1 << 30):
        s -= 1
    h = np.ldexp(0.5, s)
    err = 5.0 * h + 4.0 + h * h * 2.0 ** -20
    lo = np.nextafter(F32(h * h - err), F32(-np.inf))
    hi = np.nextafter(F32(h * h + err), F32(np.inf))
    return s, np.ldexp(1.0 / d, s), lo, hi


def _wrap(v):
    return (np.asarray(v, dtype=np.int64) & 0xFFFFFFFF).astype(np.uint32)


def _integer(x, y, dz, sx, sy, n, d, gso):
    """(in, near, hit, maybe, kx, ky) as the kernel forms them (d2 in float64: the kernel's float
    roundings are inside its bound)."""
    s, scale, lo, hi = _setup(n, d)
    half = 1 << s >> 1
    ns = n << s
    v = []
    for c, shift in ((x, sx), (y, sy)):
        r = np.rint(c * scale).astype(np.int64) + (np.int64(np.rint((shift - gso) * scale)) + half)
        v.append(_wrap(r))
    inside = (v[0] - np.uint32(2) <= np.uint32(ns - 4)) & (v[1] - np.uint32(2) <= np.uint32(ns - 4))
    near = (v[0] + np.uint32(1) <= np.uint32(ns + 2)) & (v[1] + np.uint32(1) <= np.uint32(ns + 2))
    f = [((w & np.uint32((1 << s) - 1)).astype(np.float64) - half) for w in v]
    gz = (dz * scale)
    d2 = f[0] ** 2 + f[1] ** 2 + F32(gz * gz).astype(np.float64)
    hit = inside & (d2 <= lo)
    maybe = np.where(inside, ~hit & (d2 <= hi), near)
    k = [(w.astype(np.int32) >> s).astype(np.int64) for w in v]
    return inside, near, hit, maybe, k[0], k[1]


def _fp64(x, y, dz, sx, sy, h, d, gso):
    x1, y1 = x + sx, y + sy
    inb = (np.abs(x1) < h) & (np.abs(y1) < h)
    ax, ay = x1 - gso, y1 - gso
    kx, ky = np.rint(ax / d), np.rint(ay / d)
    dist = ((kx * d - ax) ** 2 + (ky * d - ay) ** 2) + dz * dz
    return inb, inb & (dist <= (d / 2) * (d / 2)), kx.astype(np.int64), ky.astype(np.int64)


def _deposits(rs, n, h, d, gso, sx, sy, m):
    x, y = rs.uniform(-2 * h, 2 * h, (2, m))
    dz = rs.uniform(-d / 2, d / 2, m)
    q = m // 4
    # on the sphere surfaces, a few units off them, on the cell faces and on the voxel's faces
    k = rs.integers(0, n, (2, q))
    th, u = rs.uniform(0, 2 * np.pi, q), rs.uniform(-1, 1, q)
    rad = d / 2 * (1 + rs.choice([0, 1e-15, -1e-15, 1e-9, -1e-9, 1e-6, -1e-6, 1e-4, -1e-4], q))
    dz[:q] = rad * u
    x[:q] = k[0] * d + gso - sx + rad * np.sqrt(1 - u * u) * np.cos(th)
    y[:q] = k[1] * d + gso - sy + rad * np.sqrt(1 - u * u) * np.sin(th)
    off = rs.choice([0, 1e-12, -1e-12, 1e-7, -1e-7, 1e-5, -1e-5], q) * d
    x[q:2 * q] = (k[0] + 0.5) * d + gso - sx + off
    dz[q:2 * q] = rs.choice([0.0, 1e-9, 1e-3, 0.3], q) * d
    y[2 * q:2 * q + q // 2] = rs.choice([-h, h], q // 2) - sy + off[: q // 2]
    keep = (np.abs(x) < 2 * h * (1 + 2.0 ** -30)) & (np.abs(y) < 2 * h * (1 + 2.0 ** -30))
    return x[keep], y[keep], dz[keep]


@pytest.mark.parametrize("hl,d", [(2500.0, 2.0), (2500.0, 10.0), (2500.0, 100.0), (2500.0, 1000.0),
                                  (5000.0, 2.0), (5000.0, 10.0), (3.0, 1000.0), (1.0, 2.0),
                                  (1e6, 1.0), (0.37, 1e-3), (1e-9, 3e-12), (5e12, 7e6)])
def test_integer_geometry_decides_as_fp64(hl, d):
    rs = np.random.default_rng(abs(hash((hl, d))) % 2 ** 32)
    n, h, length, gso = _geometry(hl, d)
    undecided = random = 0
    for u in (1.0, 2.0 ** -24, 0.5, *rs.random(5)):
        sx, sy = u * length - h, rs.random() * length - h
        x, y, dz = _deposits(rs, n, h, d, gso, sx, sy, 200_000)
        inside, near, hit, maybe, kx, ky = _integer(x, y, dz, sx, sy, n, d, gso)
        inb, ehit, ex, ey = _fp64(x, y, dz, sx, sy, h, d, gso)
        sure = ~maybe
        assert np.array_equal(inside[sure], inb[sure])
        assert np.array_equal(hit[sure], ehit[sure])
        assert np.array_equal(kx[hit], ex[hit]) and np.array_equal(ky[hit], ey[hit])
        undecided += maybe[-len(x) // 4:].sum()      # (the uniformly distributed ones)
        random += len(maybe[-len(x) // 4:])
    if n <= 5000:
        assert undecided / random < 2e-4
    # a padding record stays outside the voxel for every shift
    s, scale, _, _ = _setup(n, d)
    c = np.array([np.int64(np.rint((u * length - h - gso) * scale)) + (1 << s >> 1)
                  for u in (2.0 ** -24, 0.3, 1.0)])
    v = _wrap(np.int64(-2 ** 31) + c)
    assert not np.any(v + np.uint32(1) <= np.uint32((n << s) + 2))
