"""The quotients of the 1-D steps (div_int, div_markstein and their fallback) as the kernels apply them: the ratio
of two bootstraps and its running variance against NumPy's IEEE operations, bit for bit, on ordinary values,
at the ends of the exponent range, on mantissas of ones, zeros, infinities and NaN, and on quotients as close to a
rounding midpoint as two 53-bit integers can come.  Needs a B200."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ieee(means, squares, state, ns, first, both):
    mean, m2 = state[:, 0].copy(), state[:, 1].copy()
    with np.errstate(all="ignore"):
        for k in range(2 if both else 1):
            m, a = np.abs(means[:, k]) / ns, np.abs(squares[:, k]) / ns
            x = (a - m * m) / m
            delta = x - mean
            mean = mean + delta / (first + k)
            m2 = m2 + delta * (x - mean)
    return np.stack([mean, m2], axis=1)


def _check(means, squares, state, ns, first, both=True):
    from pkde_b200 import _lib
    got = _lib.diag_vmr_update(means, squares, state, ns, first, both)
    want = _ieee(means, squares, state, ns, first, both)
    same = (got.view(np.int64) == want.view(np.int64)) | (np.isnan(got) & np.isnan(want))
    bad = np.nonzero(~same.all(axis=1))[0]
    assert not len(bad), (len(bad), means[bad[0]], squares[bad[0]], state[bad[0]], got[bad[0]], want[bad[0]])


@pytest.mark.parametrize("ns,first", [(1, 1), (2, 2), (3, 3), (1000, 7), (99999, 100), (2 ** 20, 4095), (2 ** 31 - 2, 65537)])
@pytest.mark.parametrize("both", [True, False])
def test_ordinary_and_wide_values(pk, ns, first, both):
    rng = np.random.default_rng(ns + first)
    n = 1 << 18
    shape = (n, 2)
    means = rng.lognormal(0.0, 3.0, shape) * rng.choice([-1.0, 1.0], shape)
    squares = rng.lognormal(0.0, 3.0, shape)
    state = np.stack([rng.standard_normal(n), rng.lognormal(size=n)], axis=1)
    wide = slice(n // 2, n)  # exponents from subnormals to infinity
    for a, neg in ((means, False), (squares, False), (state[:, :1], True)):
        e = rng.integers(-1074, 1024, a[wide].shape)
        a[wide] = np.ldexp(rng.random(a[wide].shape) + 0.5, e) * rng.choice([-1.0, 1.0], a[wide].shape)
    ones = slice(n // 4, n // 3)  # mantissas of ones
    means[ones] = np.ldexp(2.0 - 2.0 ** -52, rng.integers(-60, 60, means[ones].shape)) * ns
    _check(means, squares, state, ns, first, both)


def test_special_values(pk):
    tiny, big = 5e-324, np.finfo(np.float64).max
    v = np.array([0.0, -0.0, tiny, 2.0 ** -1022, 2.0 ** -723, 2.0 ** -724, 1.0, 2.0 - 2.0 ** -52, 2.0 ** 677, 2.0 ** 678, big,
                  np.inf, -np.inf, np.nan])
    g = np.stack(np.meshgrid(v, v, v, indexing="ij"), axis=-1).reshape(-1, 3)
    means, squares = np.stack([g[:, 0], g[::-1, 0]], axis=1), np.stack([g[:, 1], g[:, 2]], axis=1)
    for mean in (0.0, 0.25, np.nan, np.inf):
        state = np.stack([np.full(len(g), mean), np.full(len(g), 0.5)], axis=1)
        for ns, first in ((1, 1), (7, 2), (1000, 99)):
            _check(means, squares, state, ns, first)


@pytest.mark.parametrize("near", [0, 40, 52])
def test_quotients_next_to_midpoints(pk, near):
    """A / B with (2 Q + 1) B = A 2^s + c, c odd and small: the quotient is c / (2 B) ulp from the midpoint Q + 1/2.
    The mean's square underflows, so the ratio is the quotient of the two integers itself."""
    import random
    r = random.Random(near)
    pairs = []
    while len(pairs) < 60000:
        B = r.getrandbits(52) | 1 << 52 | 1
        if near:  # mantissas near 2
            B = (1 << 53) - r.getrandbits(near) | 1
        if B.bit_length() != 53:
            continue
        for s in (53, 54):
            inv = pow(B, -1, 1 << s)
            for c in (-3, -1, 1, 3):
                M = c * inv % (1 << s)
                for M in ([M, M + (1 << 53)] if s == 53 else [M]):
                    if M.bit_length() == 54 and M & 1:
                        A, rest = divmod(M * B - c, 1 << s)
                        assert rest == 0
                        if A.bit_length() == 53:
                            pairs.append((A, B))
    p = np.array(pairs, dtype=np.float64)
    n = len(p) // 2 * 2
    A, B = p[:n, 0].reshape(-1, 2), p[:n, 1].reshape(-1, 2)
    state = np.zeros((n // 2, 2))
    state[:, 0] = 0.125
    _check(B * 2.0 ** -700, A * 2.0 ** -700, state, 1, 1)
    _check(B * 2.0 ** -650, A * 2.0 ** -600, state, 1, 5)


def test_fused_operations(pk):
    """Power-of-two lengths: |V| / n fused into the difference, 1 / i as a factor, both updates fused."""
    import ctypes
    import ctypes.util
    from pkde_b200 import _lib
    libm = ctypes.CDLL(ctypes.util.find_library("m"))
    libm.fma.restype, libm.fma.argtypes = ctypes.c_double, [ctypes.c_double] * 3
    fma = np.vectorize(libm.fma, otypes=[float])
    rng = np.random.default_rng(8)
    n, ns, first = 20000, 1000, 3
    means, squares = rng.lognormal(0.0, 2.0, (n, 2)), rng.lognormal(0.0, 2.0, (n, 2)) + 1.0
    state = np.stack([rng.standard_normal(n), rng.lognormal(size=n)], axis=1)
    got = _lib.diag_vmr_update(means, squares, state, ns, first, fused=True)
    mean, m2 = state.T.copy()
    for k in range(2):
        inv_n, inv_i = 1.0 / ns, 1.0 / (first + k)
        m = means[:, k] * inv_n
        x = _lib.diag_divide(fma(squares[:, k], inv_n, -(m * m)), m)
        delta = x - mean
        mean = fma(delta, inv_i, mean)
        m2 = fma(delta, x - mean, m2)
    assert np.array_equal(got, np.stack([mean, m2], axis=1))
