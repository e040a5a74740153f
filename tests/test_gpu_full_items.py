"""The evidence sums of a full work item (csrc/evidence.cu, FxSum): coincident rays through cell centres,
so that every ray adds the same integer number of units and the cells on the line add values of 1, the
largest. A sum over n rays has to be exactly n times one ray's, for the unsigned K3DOM sums at up to 1,024
rays an item and for the calibration's, whose derivative sums are signed, at up to 768."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
G, GZ, RES = 24, 8, 0.25  # exact in FP32, as are the cell centres
RAY = np.array([[1.75, 0.0, 0.0]], np.float32)
SENSOR = (0.125, 0.125, 0.125)  # a cell centre


def k3dom_sums(n, rule):
    import k3dom_b200 as K
    p = K.make_params("k3dom", size=(G + 0.5) * RES, size_z=(GZ + 0.5) * RES, resolution=RES, particle_count=1024,
                      new_born_particle_count=256, max_points=n, ls=0.6, sigma=1.0, map_shift_thresh=1000,
                      sensor_off_x=SENSOR[0], sensor_off_y=SENSOR[1], sensor_off_z=SENSOR[2])
    with K.DOM(p, "k3dom") as d:
        d.set_tuning(rule, 1024)
        d.updatePose(*SENSOR)
        d.updateGrid(0.1, np.repeat(RAY, n, 0))
        return d.get_cell_field("del_occ"), d.get_cell_field("del_free")


@pytest.mark.parametrize("rule", [1, 2, 3])
def test_k3dom_items(rule):
    one = k3dom_sums(1, rule)
    assert one[0].max() > 0.5 and one[1].max() == 1.0
    for n in (512, 1024, 4096):  # powers of two: the FP32 results scale exactly
        for a, b in zip(k3dom_sums(n, rule), one):
            assert np.array_equal(a, np.float32(n) * b)


@pytest.mark.parametrize("n", [2, 767, 768, 769, 3000])
def test_calibration_items(n):
    from k3dom_b200 import calib
    import k3dom_b200 as K
    p = K.make_params("k3dom", size=(G + 0.5) * RES, size_z=(GZ + 0.5) * RES, resolution=RES)
    sums = []
    for m in (1, n):
        c = calib.Calibration(p)
        try:
            c.add_frame(0.0, np.array(SENSOR, np.float32), np.repeat(RAY, m, 0), None)
            sums.append(c.sums(0.6, 0) * 2.0**40)  # units
        finally:
            c.close()
    one, many = sums
    assert np.array_equal(one, np.rint(one)) and one[1].max() == 2.0**40 and np.abs(one[2:]).max() > 0.5 * 2.0**40
    assert np.array_equal(many, n * one)  # below 2^53, exact in FP64
