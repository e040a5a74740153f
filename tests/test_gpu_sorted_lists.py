"""Ray lists sorted by tile (csrc/evidence.cu, build_ray_lists: grids with more tiles than placed lists
take) against placed ones, with a moving sensor, long lists and several item sizes: the results depend
neither on the tiles nor on the lists' form, so the frames are the same bits. A sorted frame enqueues more
kernels than a placed one, which shows that each side took its own path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("free_mass", "static_mass", "dynamic_mass", "occ_mass", "pers_mass", "born_mass", "mean_x_vel", "w_UA",
          "meas_occ", "meas_free", "del_occ", "del_free")


def frames(variant, G, tuning, timing):
    import k3dom_b200 as K
    from k3dom_b200 import scene
    cfg = scene.small(seed=3, variant=variant, G=G, Gz=12, res=0.1, P=65536, B=16384, n_points=20000, ego=1.2)
    cfg.params["seed"] = 21
    with K.DOM(K.make_params(variant, **cfg.params), variant) as d:
        d.set_tuning(*tuning)
        for f in range(5):
            if f == 4:  # the ordered frame: K3DOM's evidence kernel updates the cells itself
                d.set_timing(timing)
            t = 0.1 * (f + 1)
            s, pts = cfg.scene.scan(f, t, cfg.n_points)
            d.updatePose(*s)
            d.updateGrid(t, pts)
            if f == 3:
                launches = d.diagnostics()["kernel_launches_per_frame"]
        assert not d.diagnostics()["overflow"]
        assert d.tuning()["tile_rule"] == tuning[0]
        p = d.get_particles("persistent")
        return [d.get_cell_field(k) for k in FIELDS] + [p[k] for k in sorted(p)], launches


# 8x8x4 tiles: 30,000 (K3DOM places up to 28,416) and 12,288 (DS up to 6,144); 16x16x4 ones: 7,500 and 3,072
@pytest.mark.parametrize("variant,G", [("k3dom", 800), ("dsphdmib", 512)])
@pytest.mark.parametrize("timing", [False, True])
def test_sorted_equals_placed(variant, G, timing):
    ref, placed = frames(variant, G, (2, 512), timing)
    for chunk in (256, 1024):
        got, launches = frames(variant, G, (1, chunk), timing)
        assert launches > placed
        for a, b in zip(got, ref):
            assert np.array_equal(a, b, equal_nan=True)
    k = FIELDS.index("del_free" if variant == "k3dom" else "meas_free")
    assert (ref[k] > 0).sum() > 10000
