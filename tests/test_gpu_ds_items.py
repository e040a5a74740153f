"""The DS summaries per (item, cell) are sized for a tenth of the work items that full ray lists would make
(csrc/evidence.cu, ds_spare_items): the memory a handle takes, and frames with more entries than that,
whose items grow instead. The measurement does not depend on the item size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(G, Gz, res, n):
    import k3dom_b200 as K
    p = K.make_params("dsphdmib", size=(G + 0.5) * res, size_z=(Gz + 0.5) * res, resolution=res, particle_count=2048,
                      new_born_particle_count=512, max_points=n, max_range=50.0, meas_occ_stddev=0.1)
    return K.DOM(p, "dsphdmib")


# what the lane-per-cell kernel's one-byte counts and sorted lists took at the same tuning
@pytest.mark.parametrize("rule,chunk,limit_mb", [(0, 512, 1005), (3, 1024, 958), (3, 32, 2389), (2, 32, 4429), (1, 32, 8521)])
def test_memory(rule, chunk, limit_mb):
    import torch
    torch.cuda.init()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with make(256, 32, 0.1, 120000) as d:
        d.set_tuning(rule, chunk)
        assert free - torch.cuda.mem_get_info()[0] < limit_mb * 1e6


def test_items_grow_with_the_lists():
    """1,000,000 points in 24x24x6 voxels: a quarter of the lists' capacity is used."""
    rng = np.random.default_rng(4)
    n = 1000000
    v = rng.normal(size=(n, 3)) * np.array([1.0, 1.0, 0.2])
    pts = (v / np.linalg.norm(v, axis=1)[:, None] * rng.uniform(0.5, 3.0, (n, 1))).astype(np.float32)
    ref = None
    for tuning in ((1, 1024), (1, 32), (1, 100), (3, 32), (2, 512)):
        with make(24, 6, 0.2, n) as d:
            d.set_tuning(*tuning)
            for t in (0.1, 0.2):
                d.updatePose(0.013, 0.021, -0.017)
                d.updateGrid(t, pts)
            got = [d.get_cell_field(k) for k in ("meas_occ", "meas_free", "occ_mass", "free_mass")]
            g = d.diagnostics()
        assert not g["overflow"] and g["kernel_evaluations"] > 100000
        if tuning[1] == 32:
            assert g["work_items"] < g["ray_list_entries"] // 40  # 32-ray items: more than // 32
        ref = ref or got
        for a, b in zip(got, ref):
            assert np.array_equal(a, b, equal_nan=True), tuning
