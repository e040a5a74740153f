"""DS rays whose squared length overflows or underflows FP32 (points beyond 1e12 m or within 1e-12 m of the
sensor: a sensor's marker for no return, a return at the sensor itself). The reference's FP32 neighbour
test (measurement_grid.cu:88-99) is no window around the half-line for them; csrc/evidence.cu applies it to
every cell of the 4x4x2 sub-blocks near the half-line, formed in FP32 (ds_reaches_sub_block), in the tiles
that the ray's binned segment meets. Here the same rule over all (cell, ray) pairs in numpy float32, with
the first-100 rule in input order; cells whose pOcc comparison is within 4 ulp of flipping are left out,
pOcc is compared to the 2.5e-7 of expf's 2 ulp."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F = np.float32


def params(G, Gz, res, n, sensor):
    import k3dom_b200 as K
    return K.make_params("dsphdmib", size=(G + 0.5) * res, size_z=(Gz + 0.5) * res, resolution=res, particle_count=2048,
                         new_born_particle_count=512, max_points=n, map_shift_thresh=1000, max_range=50.0,
                         meas_occ_stddev=0.1, sensor_off_x=sensor[0], sensor_off_y=sensor[1], sensor_off_z=sensor[2])


def measure(p, pts, tuning, sensor):
    import k3dom_b200 as K
    with K.DOM(p, "dsphdmib") as d:
        d.set_tuning(*tuning)
        for t in (0.1, 0.2):
            d.updatePose(*sensor)
            d.updateGrid(t, pts)
        i = d.info()
        rel = np.array([i.sensor_x - i.center_x, i.sensor_y - i.center_y, i.sensor_z - i.center_z], F)
        return d.get_cell_field("meas_occ"), d.get_cell_field("meas_free"), d.diagnostics()["kernel_evaluations"], rel


def listed(m, sq, rel, G, Gz, res, R, tile):
    """(tile x, y, z) -> whether the ray's binned segment, clipped to the grid's cell centres grown by R,
    meets the tile's cell centres grown by R."""
    a = np.array([rel[0] / res + F(G) / F(2) - F(0.5), rel[1] / res + F(G) / F(2) - F(0.5),
                  rel[2] / res + F(Gz) / F(2) - F(0.5)], F)
    half = F(0.5) * (np.array([G, G, Gz], F) - F(1))
    diag = np.sqrt(F(2 * G * G + Gz * Gz))
    L = max(diag, F(0.5) * diag + np.sqrt(((a - half) ** 2).sum(dtype=F))) + F(2) * R + F(4)
    d = m / res * (L / (np.sqrt(sq) / res))
    nt = [-(-g // t) for g, t in zip((G, G, Gz), tile)]
    t0, t1 = np.zeros(nt, F), np.ones(nt, F)
    for k in range(3):
        lo = np.arange(nt[k], dtype=F) * F(tile[k]) - R
        hi = np.minimum(lo + F(tile[k] - 1) + F(2) * R, F((G, G, Gz)[k] - 1) + R)
        if d[k] == 0:
            e0 = np.where((a[k] >= lo) & (a[k] <= hi), F(-np.inf), F(np.inf))
            e1 = -e0
        else:
            e0, e1 = (lo - a[k]) / d[k], (hi - a[k]) / d[k]
        shape = [1, 1, 1]
        shape[k] = nt[k]
        t0 = np.maximum(t0, np.minimum(e0, e1).reshape(shape))
        t1 = np.minimum(t1, np.maximum(e0, e1).reshape(shape))
    return t0 <= t1


def expected(p, G, Gz, rel, pts, tile):
    max_range, delta = p.max_range, p.meas_occ_stddev
    res, hg, hz = F(p.resolution), F(G) / F(2), F(Gz) / F(2)
    x = (np.arange(G + 4, dtype=F) + F(0.5) - hg) * res - rel[0]
    y = (np.arange(G + 4, dtype=F) + F(0.5) - hg) * res - rel[1]
    z = (np.arange(Gz + 4, dtype=F) + F(0.5) - hz) * res - rel[2]
    iz, iy, ix = [v.ravel() for v in np.meshgrid(np.arange(Gz), np.arange(G), np.arange(G), indexing="ij")]
    cx, cy, cz = x[ix], y[iy], z[iz]
    hres = F(0.5) * res
    qx, qy, qz = x[(ix & ~3) + 2] - hres, y[(iy & ~3) + 2] - hres, z[(iz & ~1) + 1] - hres
    acs = (cx * cx + cy * cy) + cz * cz
    wr = res * F(0.866)
    wr2 = wr * wr
    ext = F(2) * (F(G) * res * F(1.7320508) + F(p.size_z))
    R = np.sqrt(wr2 + F(64.0 * 5.96e-8) * ext * ext) / res + F(1e-3)
    rls2 = (R * res) ** 2
    nb = np.zeros((len(pts), len(cx)), bool)
    r2 = np.empty(nb.shape, F)
    closer = np.zeros(nb.shape, bool)
    with np.errstate(all="ignore"):
        for i, (mx, my, mz) in enumerate(pts.astype(F)):
            sq = (mx * mx + my * my) + mz * mz
            if not sq > 0:
                continue
            ip = (cx * mx + cy * my) + cz * mz
            ok = (ip > 0) & (acs - (ip * ip) / sq < wr2)
            if not (2.0**-80 <= sq <= 2.0**80):
                inv = F(1) / np.sqrt(sq)
                ux, uy, uz = mx * inv, my * inv, mz * inv
                t = np.maximum(qx * ux + qy * uy + qz * uz, F(0))
                Dx, Dy, Dz = qx - t * ux, qy - t * uy, qz - t * uz
                D2 = Dx * Dx + Dy * Dy + Dz * Dz
                v = D2 - (F(3) * hres * (abs(Dx) + abs(Dy)) + hres * abs(Dz))
                ok &= (v <= 0) | (v * v < rls2 * D2)
                ok &= listed(np.array([mx, my, mz], F), sq, rel, G, Gz, res, R, tile)[
                    ix // tile[0], iy // tile[1], iz // tile[2]]
            nb[i], closer[i] = ok, ok & (acs > sq)
            r2[i] = ((cx - mx) ** 2 + (cy - my) ** 2) + (cz - mz) ** 2
        nb &= np.cumsum(nb, 0) <= 100  # the first 100 in input order
        any_nb, far = nb.any(0), ~(nb & closer).any(0)
        mx = F(0.95) * np.exp(F(-0.5) * np.where(nb, r2, F(np.inf)).min(0) / (F(delta) * F(delta))).astype(F)
        unc = F(0.15) + np.sqrt(acs) / F(max_range) * (F(1) - F(0.15))
        lim = np.where(far, unc, F(0.5))
        tie = any_nb & (abs(mx - lim) <= 4 * np.finfo(F).eps * np.maximum(mx, lim))
        mo, mf = np.where(mx > lim, mx, F(0)), np.where(far & ~(mx > unc), F(1) - unc, F(0))
        clip = lambda v: np.where(any_nb, np.clip(v, F(1e-5), F(1) - F(1e-5)), F(0))
    return clip(mo), clip(mf), tie, int(nb.sum()), int((nb.sum(0) == 100).sum())


def rays(kind, n, seed):
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3)) * np.array([1.0, 1.0, 0.3])
    if kind == "bundle":
        d = np.array([1.0, 0.4, 0.1]) + 0.02 * rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    lo, hi = {"infinite": (19.4, 20.5), "large": (11.0, 37.0), "small": (-23.0, -11.0), "bundle": (17.5, 19.1)}[kind]
    r = 10.0 ** rng.uniform(lo, hi, n)
    plain = np.arange(n) % 3 == 0  # beside ordinary rays
    r[plain] = rng.uniform(0.5, 4.0, plain.sum())
    return (d * r[:, None]).astype(F)


@pytest.mark.parametrize("kind,n", [("infinite", 60), ("infinite", 700), ("large", 400), ("small", 400), ("bundle", 900)])
@pytest.mark.parametrize("sensor", [(0.07, -0.05, 0.03), (1.9, 2.1, -0.31)])
def test_extreme_ranges(kind, n, sensor):
    G, Gz, res = 26, 9, 0.2
    pts = rays(kind, n, n)
    p = params(G, Gz, res, n, sensor)
    tiles = {1: (8, 8, 4), 2: (16, 16, 4), 3: (16, 16, 8)}
    for tuning in ((1, 1024), (1, 32), (2, 64), (3, 512)):
        mo, mf, ev, rel = measure(p, pts, tuning, sensor)
        emo, emf, tie, n_nb, full = expected(p, G, Gz, rel, pts, tiles[tuning[0]])
        assert tie.mean() < 0.01 and (kind != "bundle" or full > 0)
        assert ev == n_nb
        for mine, exp in ((mo, emo), (mf, emf)):
            np.testing.assert_array_equal(mine[~tie] <= 1e-5, exp[~tie] <= 1e-5)
            np.testing.assert_allclose(mine[~tie], exp[~tie], rtol=2.5e-7, atol=0)
