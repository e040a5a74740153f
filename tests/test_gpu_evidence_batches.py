"""K3DOM evidence at the sizes where its batches are partial: ray counts around the 32-candidate
batches, the 8-ray steps and the work items, ragged grids, and a sensor at the centre of a 4x4x2
sub-block (a centroid at distance 0 from every ray). Each against the FP64 oracle, to 1e-5 (the
kernel table's 1.2e-7, a few FP32 roundings of O(ls) quantities) outside pairs tied on the
d_proj < d_m test."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def evidence(G, Gz, res, ls, sigma, pts, tuning=None, sensor=(0.0, 0.0, 0.0)):
    import k3dom_b200 as K
    p = K.make_params("k3dom", size=(G + 0.5) * res, size_z=(Gz + 0.5) * res, resolution=res, particle_count=1024,
                      new_born_particle_count=256, sigma=sigma, ls=ls, max_points=max(1, len(pts)), mass_scale=2.5,
                      map_shift_thresh=1000, sensor_off_x=sensor[0], sensor_off_y=sensor[1], sensor_off_z=sensor[2])
    with K.DOM(p, "k3dom") as d:
        if tuning:
            d.set_tuning(*tuning)
        d.updatePose(*sensor)
        d.updateGrid(0.1, pts)
        i = d.info()
        rel = np.array([i.sensor_x - i.center_x, i.sensor_y - i.center_y, i.sensor_z - i.center_z], np.float32)
        return d.get_cell_field("del_occ"), d.get_cell_field("del_free"), rel, p


def check(G, Gz, res, ls, sigma, pts, **kw):
    from oracle import binding as O
    occ, free, rel, p = evidence(G, Gz, res, ls, sigma, pts, **kw)
    ref = O.bgki(G, Gz, p.resolution, rel, p.ls, p.sigma, pts)
    for got, want, tie in ((occ, ref["del_occ"], 0.0), (free, ref["del_free"], ref["tie_mass"])):
        err = np.abs(got.astype(np.float64) - want) - tie
        assert np.all(err <= 1e-5 * np.maximum(want, 1e-2 * p.sigma))
    assert ref["del_free"].max() > 0
    return occ, free


def scan(n, seed, reach):
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3)) * np.array([1.0, 1.0, 0.3])
    d /= np.linalg.norm(d, axis=1)[:, None]
    return (d * rng.uniform(0.2 * reach, 1.2 * reach, (n, 1))).astype(np.float32)


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 40, 63, 64, 65, 97, 511, 513, 1025, 2100])
def test_partial_batches(n):
    check(33, 9, 0.2, 0.5, 0.1, scan(n, n, 3.3))


@pytest.mark.parametrize("tuning", [(1, 32), (1, 1024), (2, 64), (2, 512), (3, 1000)])
def test_item_sizes_agree(tuning):
    pts = scan(3000, 5, 4.0)
    a = check(48, 12, 0.1, 0.3, 1.0, pts, tuning=tuning)
    b = evidence(48, 12, 0.1, 0.3, 1.0, pts, tuning=(0, 1024))
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])  # exact sums: same bits


@pytest.mark.parametrize("G,Gz", [(12, 6), (20, 10), (44, 14)])
def test_sensor_at_a_sub_block_centroid(G, Gz):
    check(G, Gz, 0.1, 0.3, 0.1, scan(700, G, 0.05 * G))


@pytest.mark.parametrize("ls,res", [(0.3, 0.4), (0.3, 0.1), (0.7, 0.1)])
def test_support_smaller_and_larger_than_a_sub_block(ls, res):
    """Rays ending in the grid (near and edge rays) and passing it, sensor off the centre."""
    check(29, 11, res, ls, 0.7, scan(400, 3, 20 * res), sensor=(3.3 * res, -5.1 * res, 1.7 * res))
