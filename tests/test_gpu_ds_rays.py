"""The DS measurement grid by rays (csrc/evidence.cu, k_ds_rays and the passes after it) where its walk
or its first-100 rule can go wrong: ragged grids, rays along an axis, steep rays, rays that start and
end outside the grid, cells with far more than 100 neighbours spread over several work items, and a
sensor on a cell centre. Neighbour sets against the oracle's FP32 restatement (cells whose pOcc
comparison is within 4 ulp of flipping left out, pOcc to the 2.5e-7 of expf's 2 ulp), and every tiling
and item size against the others bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def measure(G, Gz, res, pts, tuning, sensor=(0.0, 0.0, 0.0)):
    import k3dom_b200 as K
    p = K.make_params("dsphdmib", size=(G + 0.5) * res, size_z=(Gz + 0.5) * res, resolution=res, particle_count=2048,
                      new_born_particle_count=512, max_points=max(1, len(pts)), map_shift_thresh=1000, max_range=50.0,
                      meas_occ_stddev=0.1, sensor_off_x=sensor[0], sensor_off_y=sensor[1], sensor_off_z=sensor[2])
    with K.DOM(p, "dsphdmib") as d:
        d.set_tuning(*tuning)
        d.updatePose(*sensor)
        d.updateGrid(0.1, pts)
        d.updateGrid(0.2, pts)  # a steady frame: the measurement beside the particles
        i = d.info()
        rel = np.array([i.sensor_x - i.center_x, i.sensor_y - i.center_y, i.sensor_z - i.center_z], np.float32)
        ev = d.diagnostics()["kernel_evaluations"]
        return d.get_cell_field("meas_occ"), d.get_cell_field("meas_free"), d.get_cell_field("occ_mass"), rel, p, ev


def rays(kind, n, reach, seed):
    rng = np.random.default_rng(seed)
    if kind == "scan":  # beams in input order, as a scanner delivers them
        el = np.deg2rad(np.linspace(-30, 30, 16)).repeat(-(-n // 16))[:n]
        az = np.tile(np.linspace(0, 2 * np.pi, -(-n // 16), endpoint=False), 16)[:n]
        d = np.stack([np.cos(el) * np.cos(az), np.cos(el) * np.sin(az), np.sin(el)], 1)
    elif kind == "steep":
        d = rng.normal(size=(n, 3)) * np.array([0.3, 0.3, 1.0])
    elif kind == "axis":
        d = np.eye(3)[np.arange(n) % 3] * np.where(np.arange(n) % 2, 1.0, -1.0)[:, None]
        d[: n // 4] += 1e-4 * rng.normal(size=(n // 4, 3))
    else:  # a narrow bundle: every ray passes the same cells
        d = np.array([1.0, 0.31, 0.12]) + 0.01 * rng.normal(size=(n, 3))
    d = d / np.linalg.norm(d, axis=1)[:, None]
    return (d * rng.uniform(0.3 * reach, 1.3 * reach, (n, 1))).astype(np.float32)


@pytest.mark.parametrize("G,Gz,res,kind,n,sensor", [
    (33, 9, 0.2, "scan", 1, (0, 0, 0)), (33, 9, 0.2, "scan", 33, (0, 0, 0)), (33, 9, 0.2, "scan", 6000, (0.13, -0.4, 0.2)),
    (40, 12, 0.1, "steep", 3000, (0, 0, 0)), (36, 11, 0.1, "axis", 300, (0.05, 0.05, 0.05)),
    (50, 10, 0.1, "bundle", 2500, (-1.0, 0.2, 0.0)), (24, 10, 0.4, "bundle", 700, (0, 0, 0)),
    (20, 6, 0.1, "scan", 4000, (0, 0, 0)), (47, 17, 0.1, "scan", 20000, (3.0, -4.0, 0.3)),
])
def test_measurement_matches_oracle(G, Gz, res, kind, n, sensor):
    from oracle import binding as O
    pts = rays(kind, n, 0.5 * G * res, n + G)
    ref = None
    for tuning in ((1, 1024), (1, 64), (2, 256), (3, 1000), (0, 32)):
        mo, mf, occ, rel, p, ev = measure(G, Gz, res, pts, tuning, sensor)
        if ref is None:
            o = O.ds_measgrid(G, Gz, p.resolution, rel, p.max_range, p.meas_occ_stddev, pts)
            ok = o["tie"] == 0
            assert ok.mean() > 0.9
            for mine, exp in ((mo, o["meas_occ"]), (mf, o["meas_free"])):
                np.testing.assert_array_equal(mine[ok] <= 1e-5, exp[ok] <= 1e-5)
                np.testing.assert_allclose(mine[ok], exp[ok], rtol=2.5e-7, atol=0)
            ref = (mo, mf, occ, ev)
        for a, b in zip((mo, mf, occ, ev), ref):
            assert np.array_equal(a, b, equal_nan=True), tuning
