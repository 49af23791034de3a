"""The slabs' windows of the system-matrix build, checked on the host.

slab_window in csrc/kernels_sm.cu bounds the voxels that a row's rays reach in each
slab of its axis by the hull of the two crystals' corners (4 x 4 pairs in (x, z), two
bounds in y), taken at the slab's two faces, with 0.02 voxel of margin in
sm_slab_kernel and one voxel in sm_window_kernel.  That a ray's voxels lie inside
is what the kernels rest on: an offset beside its window, but within the row's slots,
would be another voxel's and go unnoticed.  Here the windows are restated in
float32 and held against the exact walk's voxels, on rays between the crystals' own
corners and edges (the hull's extremes) and on drawn ones."""
import dataclasses

import numpy as np
import pytest

from raptr_b200 import config as cfg

F = np.float32
CORNERS = np.array([[c & 1, c >> 1, c >> 1] for c in range(4)], F)
BELOW_1 = np.nextafter(F(1), F(0))


def crystals(O, g, cnl):
    ida, id0z, id0y, id1z, id1y = (int(v) for v in O.channel_split(g, cnl))
    return [(det, ida, idz, idy) for det, (idz, idy) in enumerate(((id0z, id0y), (id1z, id1y)))]


def slab_axis(g, p, q, ab):
    o, d, n = np.array(g.grid_o, F), np.array(g.grid_d, F), np.array(g.grid_n)
    first = 0 if abs(ab[0]) >= abs(ab[2]) else 2
    for a in (first, 2 - first):
        c0, c1 = o[a], F(o[a] + F(F(n[a]) * d[a]))
        m = F(F(1e-6) * F(F(1) + abs(c0) + abs(c1)))
        if n[a] <= 256 and ((p[:, a].max() + m < c0 and q[:, a].min() - m > c1) or
                            (q[:, a].max() + m < c0 and p[:, a].min() - m > c1)):
            return a
    return None


def windows(g, A, p, q, margin):
    """Per slab (first, last) voxel along y and along the other axis of x and z."""
    o, d, n = np.array(g.grid_o, F), np.array(g.grid_d, F), np.array(g.grid_n)
    w = 2 - A
    pa, qa, pw, qw = p[:, None, A], q[None, :, A], p[:, None, w], q[None, :, w]
    y0, y1 = (p[0, 1], p[2, 1]), (q[0, 1], q[2, 1])
    out = []
    for s in range(n[A]):
        t = np.array([F(F(F(o[A] + F(F(s + k) * d[A])) - pa) * F(F(1) / (qa - pa))) for k in (0, 1)], F)
        x = pw + t * (qw - pw)
        ylo = y0[0] + min(t.min() * (y1[0] - y0[0]), t.max() * (y1[0] - y0[0]))
        yhi = y0[1] + max(t.min() * (y1[1] - y0[1]), t.max() * (y1[1] - y0[1]))
        row = []
        for ax, lo, hi in ((1, ylo, yhi), (w, x.min(), x.max())):
            inv = F(F(1) / d[ax])
            a = int(np.floor(F(F(F(lo - o[ax]) * inv) - F(margin))))
            b = int(np.floor(F(F(F(hi - o[ax]) * inv) + F(margin))))
            a = min(max(a, 0), n[ax] - 1)
            row.append((a, max(min(max(b, 0), n[ax] - 1), a)))
        out.append(row)
    return out


def eps(g, ray):
    """The bound on a ray's roundings in voxels above which the slab kernel leaves it."""
    worst = 0.0
    for k in range(3):
        d, o = g.grid_d[k], g.grid_o[k]
        worst = max(worst, 4.2e-7 * (2 * abs(ray[k] - o) / d + abs(ray[3 + k] - ray[k]) / d + 2 * abs(o) / d +
                                     g.grid_n[k] + 2))
    return worst


FULL = cfg.FULL
CASES = {
    "40^3": cfg.SMALL, "70^3": FULL, "100^3": cfg.FINE,
    "anisotropic, off centre": cfg.Geometry((-0.061, -0.047, -0.039), (0.002, 0.0025, 0.0018), (60, 40, 48), -0.240,
                                            0.240, 12, 13, 13, 13, 13, 15.0, 0.020, 0.004, 0.004),
    "steep": dataclasses.replace(FULL, grid_n=(18, 60, 60), grid_d=(0.005, 0.001, 0.001), grid_o=(-0.045, -0.03, -0.03)),
    "large crystals": dataclasses.replace(FULL, segy=0.02, segz=0.02, n0y=3, n0z=3, n1z=3, n1y=3),
    # roundings near the most that the slab kernel takes (0.01 voxel)
    "far": dataclasses.replace(FULL, pos0x=-2.5, pos1x=2.5, grid_d=(0.0005,) * 3, grid_o=(-0.0175,) * 3, na=7, da=25.7),
}


@pytest.mark.parametrize("name", CASES)
def test_walked_voxels_lie_inside_the_hull(oracle, name):
    O, g = oracle, CASES[name]
    rng = np.random.default_rng(31)
    n = np.array(g.grid_n)
    taken = 0
    for cnl in rng.integers(0, g.n_channels, 16):
        cr = crystals(O, g, int(cnl))
        p, q = (O.trafo_f(g, *c, CORNERS) for c in cr)
        mid = [O.trafo_f(g, *c, np.full((1, 3), 0.5, F))[0] for c in cr]
        A = slab_axis(g, p, q, mid[1] - mid[0])
        if A is None:
            continue
        u, v = (1, 2) if A == 0 else (0, 1)
        ends = []
        for c in cr:
            local = rng.uniform(0, 1, (24, 3)).astype(F)
            local[:16] = np.where(rng.random((16, 3)) < 0.5, F(0), BELOW_1)  # corners
            local[16:20, rng.integers(0, 3)] = BELOW_1                       # points of faces
            ends.append(O.trafo_f(g, *c, local))
        drawn = O.rays(g, np.array([cnl], np.int32), 8, 1251)[0]
        rays = [np.concatenate([a, b]) for a, b in zip(*ends)] + list(drawn)
        for margin in (0.02, 1.0):
            rows = windows(g, A, p, q, margin)
            for ray in rays:
                if eps(g, ray) > 0.01 or np.any(ray[:3] == ray[3:]):
                    continue
                taken += 1
                for vid, length in zip(*O.walk_ray(g, ray.astype(F))):
                    if not length > 0:
                        continue
                    ijk = (vid // (n[1] * n[2]), (vid // n[2]) % n[1], vid % n[2])
                    (ylo, yhi), (wlo, whi) = rows[ijk[A]]
                    assert ylo <= ijk[1] <= yhi and wlo <= ijk[2 - A] <= whi, (int(cnl), margin, ijk)
    assert taken > 200
