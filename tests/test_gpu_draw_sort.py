"""The resampling draws, generated into buckets and sorted there (csrc/drawsort.cu), at particle counts
around its blocks (16,384 draws), Philox blocks (4) and warp-sorted buckets (128 of 4,096), and in a
batch of uneven scenes: every ancestor equals lower_bound of the sorted draws over the library's
cumulative weights, in numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def expected_ancestors(seed, frame, cum):
    import k3dom_b200 as K
    P = expected_ancestors.P
    u = K.debug_draws(seed, frame, 4, 0, P).astype(np.float32)  # (0, 1] on the 2^-24 grid
    om = np.sort(np.float32(1.0) - u)                              # exact
    draws = (cum[-1] * om).astype(np.float32)
    acc = cum.copy()
    acc[-1] = draws[-1]
    return np.minimum(np.searchsorted(acc, draws, side="left"), cum.size - 1)


def check(dom, seed, frame, P):
    cum, _, jmax = dom.resampling_state()
    expected_ancestors.P = P
    assert jmax == cum[-1] and jmax > 0
    assert np.array_equal(dom.ancestors(), expected_ancestors(seed, frame, cum))


def params(P, seed, n):
    import k3dom_b200 as K
    from k3dom_b200 import scene
    cfg = scene.small(seed=2, G=24, Gz=8, res=0.2, P=P, B=max(1, P // 4), n_points=n)
    cfg.params["seed"] = seed
    return cfg, K.make_params("k3dom", **cfg.params)


@pytest.mark.parametrize("P", [1, 2, 3, 5, 127, 4096, 16383, 16384, 16385, 40001, 262147, 600000, 1300000])
def test_sorted_draws(P):
    import k3dom_b200 as K
    cfg, p = params(P, 77 + P, 600)
    with K.DOM(p, "k3dom") as d:
        for f in range(3):
            s, pts = cfg.scene.scan(f, 0.1 * (f + 1), cfg.n_points)
            d.updatePose(*s)
            d.updateGrid(0.1 * (f + 1), pts)
        check(d, p.seed, 2, P)


def test_uneven_batch():
    import k3dom_b200 as K
    sizes = [1, 7000, 16384, 270001, 33, 900000]
    cfgs = [params(P, 5 + P, 300 + k) for k, P in enumerate(sizes)]
    with K.BatchDOM([p for _, p in cfgs], "k3dom") as b:
        for f in range(3):
            scans = [c.scene.scan(f, 0.1 * (f + 1), c.n_points) for c, _ in cfgs]
            for k, (s, _) in enumerate(scans):
                b.updatePose(k, *s)
            b.update([0.1 * (f + 1)] * len(sizes), [p for _, p in scans])
        for k, P in enumerate(sizes):
            check(b.scene(k), cfgs[k][1].seed, 2, P)
