"""Evidence work items shrink with the scene (csrc/evidence.cu, item_rays) so that a small scan still
makes enough of them to fill the GPU. The sums are exact, so the item size must not change a bit:
frames at scan sizes on both sides of the rule's limits against the same frames with items of at most
32 rays, for placed and for sorted ray lists."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def frames(n, tuning, G=40, Gz=9, res=0.2):
    import k3dom_b200 as K
    from k3dom_b200 import scene
    cfg = scene.small(seed=n, G=G, Gz=Gz, res=res, P=4096, B=1024, n_points=n, ego=1.0)
    cfg.params["seed"] = 3
    with K.DOM(K.make_params("k3dom", **cfg.params), "k3dom") as d:
        d.set_tuning(*tuning)
        for f in range(3):
            s, pts = cfg.scene.scan(f, 0.1 * (f + 1), n)
            d.updatePose(*s)
            d.updateGrid(0.1 * (f + 1), pts)
        d.set_timing(True)  # the ordered frame, whose evidence kernel updates the cells itself
        s, pts = cfg.scene.scan(3, 0.4, n)
        d.updatePose(*s)
        d.updateGrid(0.4, pts)
        items = d.diagnostics()["work_items"]
        return [d.get_cell_field(k) for k in ("del_occ", "del_free", "free_mass", "static_mass", "dynamic_mass")], items


@pytest.mark.parametrize("n", [1, 33, 500, 4000, 30000])
def test_item_size_changes_nothing(n):
    a, few = frames(n, (1, 1024))
    b, many = frames(n, (1, 32))
    assert few <= many
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


def test_sorted_lists():
    """More tiles than the placed lists take (8x8x4 tiles of a 512x512x12 grid)."""
    a, few = frames(20000, (1, 1024), G=512, Gz=12, res=0.1)
    b, many = frames(20000, (1, 32), G=512, Gz=12, res=0.1)
    assert few < many
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
