"""K3DOM ray lists of many tiles: placed through histograms past 48 KB of shared memory up to 28,416
tiles, sorted by tile above (csrc/evidence.cu, build_ray_lists). Frames with 8x8x4 tiles on both sides
of the limits against the same frames with 16x16x4 tiles: the sums are exact, so the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cells(G, Gz, rule):
    import k3dom_b200 as K
    from k3dom_b200 import scene
    cfg = scene.small(seed=G, G=G, Gz=Gz, res=0.1, P=2048, B=512, n_points=3000, ego=0.0)
    rng = np.random.default_rng(G)
    with K.DOM(K.make_params("k3dom", **cfg.params), "k3dom") as d:
        d.set_tuning(rule, 512)
        for f in range(3):
            v = rng.normal(size=(3000, 3)) * np.array([1.0, 1.0, 0.02])
            pts = (v / np.linalg.norm(v, axis=1)[:, None] * rng.uniform(1.0, 0.05 * G, (3000, 1))).astype(np.float32)
            d.updatePose(0.0, 0.0, 0.0)
            d.updateGrid(0.1 * (f + 1), pts)
        return [d.get_cell_field(k) for k in ("del_occ", "del_free", "free_mass", "static_mass")]


# 8x8x4 tiles: 12,288, 12,675, 28,227, 28,812 and 30,000
@pytest.mark.parametrize("G", [512, 520, 776, 784, 800])
def test_many_tiles(G):
    for a, b in zip(cells(G, 12, 1), cells(G, 12, 2)):
        assert np.array_equal(a, b)
