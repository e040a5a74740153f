"""The evidence kernels round each kernel value to an integer number of units of 2^-40 and sum the
integers without conversion instructions: FP32 additions of two constants leave the integer's high
and low part in the mantissas (csrc/evidence.cu, FxSum). The same operations in numpy float32
against exact integer arithmetic: each value rounds to the nearest integer, ties to even, and sums
of up to 1,024 values, pads included, come out exact."""
import numpy as np
import pytest

HI, LO = np.float32(6.0), np.float32(1.5 / (1 << 17))
HI_BITS, LO_BITS = 0x40C00000, 0x37400000
SHIFT = 40


def parts(v):
    """The bit patterns the kernel adds, for float32 values v."""
    v = v.astype(np.float32)
    t = (v + HI).astype(np.float32)
    q = ((v - (t - HI).astype(np.float32)).astype(np.float32) + LO).astype(np.float32)
    return t.view(np.uint32).astype(np.uint64), q.view(np.uint32).astype(np.uint64)


def total(hi, lo, n, signed):
    h = (int(hi) - n * HI_BITS) & 0xFFFFFFFF
    l = (int(lo) - n * LO_BITS) & 0xFFFFFFFF
    l -= (1 << 32) if l >= 1 << 31 else 0
    if signed and h >= 1 << 31:
        h -= 1 << 32
    return (h << 19) + l


def exact(v):
    """round-half-even of v * 2^40, exactly (v * 2^40 is exact in FP64)."""
    return np.rint(v.astype(np.float64) * 2.0**SHIFT).astype(np.int64)


def values(seed):
    rng = np.random.default_rng(seed)
    x = [rng.random(200000), 10.0 ** rng.uniform(-14, 0, 200000), np.array([0.0, 1.0, 0.5, 2.0**-40, 2.0**-41, 2.0**-42]),
         (rng.integers(0, 1 << 22, 100000) + 0.5) * 2.0**-SHIFT,        # ties
         (rng.integers(0, 1 << 19, 1000) * 2.0 + 1.0) * 2.0**-22,       # halves of the high part's step
         np.nextafter(np.float32(1), np.float32(0))[None]]
    return np.concatenate(x).astype(np.float32)


def test_each_value_rounds_to_the_nearest_unit():
    v = values(0)
    hi, lo = parts(v)
    want = exact(v)
    got = np.array([total(h, l, 1, False) for h, l in zip(hi[::7], lo[::7])])
    assert np.array_equal(got, want[::7])
    w = -v[v < 0.9]
    hi, lo = parts(w)
    got = np.array([total(h, l, 1, True) for h, l in zip(hi[::7], lo[::7])])
    assert np.array_equal(got, exact(w)[::7])


@pytest.mark.parametrize("n", [1, 2, 31, 1023, 1024])
def test_sums_are_exact(n):
    rng = np.random.default_rng(n)
    for v in (np.ones(n, np.float32), rng.choice(values(1), n), rng.random(n).astype(np.float32)):
        # the kernel adds pads and cells out of reach as zeros: up to 7 more per batch of 32
        w = np.concatenate([v, np.zeros(7 * (n // 32 + 1), np.float32)])
        hi, lo = parts(w)
        assert total(hi.sum() & 0xFFFFFFFF, lo.sum() & 0xFFFFFFFF, len(w), False) == exact(v).sum()
        s = np.where(rng.random(n) < 0.5, -0.7 * v, 0.7 * v).astype(np.float32)[:1000]
        hi, lo = parts(s)
        assert total(hi.sum() & 0xFFFFFFFF, lo.sum() & 0xFFFFFFFF, len(s), True) == exact(s).sum()
