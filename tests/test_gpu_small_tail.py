"""A frame's tail picks its kernels by size: the exact scans skip the group pass up to 1,024 tiles, the
cell update stages cells by bulk copies from 1.5M cells on, and resampling takes one draw per thread
below 2M particles. A batch adds up its scenes' sizes, so the same scene goes one way alone and the
other way inside a large batch, and has to give the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("free_mass", "static_mass", "dynamic_mass", "pers_mass", "born_mass", "mean_x_vel", "w_UA")


def config(k, P, B):
    from k3dom_b200 import scene
    cfg = scene.small(seed=11 + k, G=60, Gz=12, res=0.2, P=P, B=B, n_points=1500, ego=1.0)
    cfg.params["seed"] = 50 + k
    return cfg


def state(d):
    p = d.get_particles("persistent")
    return ([d.get_cell_field(f) for f in FIELDS] + [p[k] for k in ("pos", "vel", "weight", "cell", "associated")]
            + [d.ancestors(), d.resampling_state()[0]])


# 43,200 cells a scene: 1.47M, 1.51M and 1.60M cells; 1.98M, 2.01M and 2.13M particles; in each the
# joint scan of the batch has more than 1,024 tiles, and a scene alone fewer than 50
@pytest.mark.parametrize("scenes,P,B", [(34, 58323, 17003), (35, 57429, 16411), (37, 57568, 19999)])
def test_scene_alone_and_in_a_large_batch(scenes, P, B):
    import k3dom_b200 as K
    cfgs = [config(k, P, B) for k in range(3)]
    which = [0] * (scenes - 2) + [1, 2]
    probe = [0, scenes - 2, scenes - 1]
    plain = [K.DOM(K.make_params("k3dom", **c.params), "k3dom") for c in cfgs]
    batch = K.BatchDOM([K.make_params("k3dom", **cfgs[w].params) for w in which], "k3dom")
    try:
        for f in range(4):
            t = 0.1 * (f + 1)
            scans = [c.scene.scan(f, t, 1500 - 7 * f) for c in cfgs]
            for d, (s, pts) in zip(plain, scans):
                d.updatePose(*s)
                d.updateGrid(t, pts)
            for k, w in enumerate(which):
                batch.updatePose(k, *scans[w][0])
            batch.update([t] * scenes, [scans[w][1] for w in which])
        for k in probe:
            for a, b in zip(state(plain[which[k]]), state(batch.scene(k))):
                assert np.array_equal(a, b, equal_nan=True)
    finally:
        batch.close()
        for d in plain:
            d.close()
