"""DS ray lists placed through bit masks (csrc/evidence.cu, k_ds_mark) against lists sorted by tile: a
grid whose 8x8x4 tiles are more than the placed lists take and whose 16x16x8 tiles are not, at ray
counts around a mask word, a block of 128 rays and a group of 32 blocks. The measurement depends on
each tile's rays and their order, not on the tiles, so the cells must be the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cells(n, rule):
    import k3dom_b200 as K
    from k3dom_b200 import scene
    cfg = scene.small(seed=7, variant="dsphdmib", G=512, Gz=12, res=0.1, P=2048, B=512, n_points=max(n, 64), ego=0.0)
    cfg.params["seed"] = 5
    import torch
    rng = np.random.default_rng(n)
    with K.DOM(K.make_params("dsphdmib", **cfg.params), "dsphdmib") as d:
        d.set_tuning(rule, 256)
        for f in range(2):
            v = rng.normal(size=(n, 3)) * np.array([1.0, 1.0, 0.02])
            v[: n // 2, :2] = np.abs(v[: n // 2, :2])  # crowds one quadrant: cells past the first-100 rule
            pts = (v / np.linalg.norm(v, axis=1)[:, None] * rng.uniform(2.0, 24.0, (n, 1))).astype(np.float32)
            if n > 3:
                pts[n // 3] = np.nan  # device scans skip such points
            d.updatePose(0.0, 0.0, 0.0)
            d.updateGrid(0.1 * (f + 1), torch.from_numpy(pts).cuda())
        return [d.get_cell_field(k) for k in ("meas_occ", "meas_free", "free_mass", "occ_mass")]


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 4095, 4096, 4097, 9000])
def test_placed_and_sorted_lists_agree(n):
    a, b = cells(n, 3), cells(n, 1)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    assert max(a[0].max(), a[1].max()) > 0
