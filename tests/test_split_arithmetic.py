"""The split's extents and dice grids in the form the kernel takes them, against
the reference's sequence (split.pikostage:240-316): the largest of four lengths by
pairs instead of one after the other, and a float rounded up instead of its
double."""
import itertools

import numpy as np


def std_max(a, b):
    return b if a < b else a


def fmax0(a, b):   # fmaxf: a NaN operand is left out
    return b if a != a else a if b != b else max(a, b)


def test_extent_by_pairs():
    values = [0.0, 1e-30, 3.5, np.inf, np.nan]
    for d in itertools.product(values, repeat=4):
        ref = 0.0
        for x in d:
            ref = std_max(ref, x)
        t = [fmax0(0.0, x) for x in d]
        assert fmax0(fmax0(t[0], t[1]), fmax0(t[2], t[3])) == ref


def test_float_rounded_up():
    g = np.random.Generator(np.random.Philox(3))
    x = np.concatenate([g.uniform(0, 70, 1 << 16), np.exp(g.uniform(-60, 40, 1 << 16)), [0.0, np.inf, 2.0**31, 2.0**24 - 1]])
    x = np.concatenate([x, np.arange(0, 40), np.nextafter(np.arange(1, 40, dtype=np.float32), np.float32(0))]).astype(np.float32)
    assert np.array_equal(np.ceil(x).astype(np.float64), np.ceil(x.astype(np.float64)))
