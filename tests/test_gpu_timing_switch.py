"""Stage timing switched on while no timed frame has run: k3dom_synchronize must not read events that nothing
recorded (the error it left made the next frame fail)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["k3dom", "dsphdmib"])
@pytest.mark.parametrize("before", [True, False])
def test_synchronize_without_a_timed_frame(variant, before):
    import k3dom_b200 as K
    from k3dom_b200 import scene
    cfg = scene.small(seed=4, variant=variant, G=24, Gz=8, res=0.2, P=2048, B=512, n_points=400)
    with K.DOM(K.make_params(variant, **cfg.params), variant) as d, K.DOM(K.make_params(variant, **cfg.params), variant) as ref:
        if before:
            d.set_timing(True)
        for f in range(3):
            t = 0.1 * (f + 1)
            s, pts = cfg.scene.scan(f, t, cfg.n_points)
            for x in (d, ref):
                x.updatePose(*s)
                x.updateGridAsync(t, pts)
                x.synchronize()
            if f == 0:
                d.set_timing(True)
                d.synchronize()
        assert d.stage_times()["total_ms"] > 0.0
        for k in ("free_mass", "pers_mass", "meas_occ", "del_free"):
            assert np.array_equal(d.get_cell_field(k), ref.get_cell_field(k), equal_nan=True)
