"""The default tile rule on both sides of its lines (2^19 cells K3DOM, 2^17 DS) gives the cells that
8x8x4 tiles give, bit for bit, also for grids too flat for its 16x16x8 tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cells(variant, G, Gz, rule):
    import k3dom_b200 as K
    from k3dom_b200 import scene
    cfg = scene.small(seed=G, variant=variant, G=G, Gz=Gz, res=0.2, P=2048, B=512, n_points=2500, ego=0.5)
    with K.DOM(K.make_params(variant, **cfg.params), variant) as d:
        if rule is not None:
            d.set_tuning(rule, 1024)
        for f in range(3):
            s, pts = cfg.scene.scan(f, 0.1 * (f + 1), 2500)
            d.updatePose(*s)
            d.updateGrid(0.1 * (f + 1), pts)
        return [d.get_cell_field(k) for k in ("meas_occ", "meas_free", "free_mass", "occ_mass", "del_occ", "del_free")]


@pytest.mark.parametrize("variant,G,Gz", [("k3dom", 127, 32), ("k3dom", 128, 32), ("k3dom", 300, 6),
                                          ("dsphdmib", 63, 33), ("dsphdmib", 64, 32), ("dsphdmib", 160, 6)])
def test_default_tiles(variant, G, Gz):
    for a, b in zip(cells(variant, G, Gz, None), cells(variant, G, Gz, 1)):
        assert np.array_equal(a, b, equal_nan=True)
