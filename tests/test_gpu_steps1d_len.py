"""1-D bandwidth steps of 2^a 3^b 5^c lengths (a kernel compiled for the length) against the
plain form, bit for bit: the shortest and longest lengths, many pairs a tile and one, a means
line alone in its tile, z and w one after the other, lines that take the SM alone, and grids so wide
that the density rounds to 0 and the running mean to NaN at most points.  Needs a B200; the
quotient's own test runs anywhere."""
import ctypes
import ctypes.util
import random

import numpy as np
import pytest

from test_gpu_steps1d import _run


@pytest.mark.gpu
@pytest.mark.parametrize("n,B,half", [
    (18, 3, 6.0), (20, 300, 6.0),          # shortest; many pairs a tile
    (100, 80, 6.0), (100, 81, 6.0),        # 40 lines a tile: the means alone in the third one, and not
    (500, 100, 6.0), (500, 40, 60.0),      # 8 lines a tile; mostly empty grid
    (1728, 5, 6.0), (1800, 5, 6.0),        # longest line in pairs, shortest one by one
    (2500, 12, 80.0), (3456, 4, 6.0),      # empty grid one by one; longest twice an SM
    (3600, 4, 6.0), (4050, 3, 40.0),       # a line has the SM alone; near the longest
])
def test_length_equals_plain_form(pk, n, B, half):
    from pkde_b200 import _lib
    x = np.random.default_rng(n).standard_normal((1, 700))
    grid = pk.initialize_grid([(-half, half, n)])
    d, s = _run(grid, x, B, 9)
    _lib.set_step_path(_lib.PKDE_STEPS_PER_STEP_LAUNCH)
    try:
        dp, sp = _run(grid, x, B, 9)
    finally:
        _lib.set_step_path(_lib.PKDE_STEPS_AUTO)
    assert np.array_equal(s, sp)
    assert np.array_equal(d, dp, equal_nan=True)


def test_quotient_steps_round_correctly():
    """The reciprocal and quotient corrections of div_markstein, from any estimate within 2^-20."""
    libm = ctypes.CDLL(ctypes.util.find_library("m"))
    fma = libm.fma
    fma.restype, fma.argtypes = ctypes.c_double, [ctypes.c_double] * 3
    r = random.Random(5)
    for _ in range(50000):
        m = r.uniform(1.0, 2.0) * 2.0 ** r.randint(-60, 60)
        v = r.choice([1.0, -1.0]) * r.uniform(1.0, 2.0) * 2.0 ** r.randint(-60, 60)
        y = 1.0 / m * (1.0 + r.uniform(-1.0, 1.0) * 2.0 ** -20)
        for _ in range(3):
            y = fma(y, fma(-m, y, 1.0), y)
        q = v * y
        assert fma(fma(-m, q, v), y, q) == v / m
