"""A K3DOM chunk below 256 rays gives the frames and the work items of 256 (csrc/internal.h, kItemLeast:
smaller items leave the batches part empty, up to 1.5 times the frame's time before)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def frame(rule, chunk):
    import k3dom_b200 as K
    from k3dom_b200 import scene
    cfg = scene.small(seed=5, G=96, Gz=12, res=0.1, P=4096, B=1024, n_points=60000, ego=0.3)
    cfg.params["seed"] = 3
    with K.DOM(K.make_params("k3dom", **cfg.params), "k3dom") as d:
        d.set_tuning(rule, chunk)
        assert d.tuning()["chunk"] == chunk
        for f in range(3):
            s, pts = cfg.scene.scan(f, 0.1 * (f + 1), cfg.n_points)
            d.updatePose(*s)
            d.updateGrid(0.1 * (f + 1), pts)
        return [d.get_cell_field(k) for k in ("del_occ", "del_free", "free_mass")], d.diagnostics()["work_items"]


@pytest.mark.parametrize("rule", [1, 2, 3])
def test_small_chunks(rule):
    ref, items = frame(rule, 256)
    for chunk in (32, 100, 255, 512):
        got, n = frame(rule, chunk)
        assert n == items if chunk < 256 else n < items
        for a, b in zip(got, ref):
            assert np.array_equal(a, b)
