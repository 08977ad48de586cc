"""FFT passes whose tiles of lines run across rows and arrays (fewer lines side by side than a tile holds), last
tiles that are not full, axes of one point and long primes, against NumPy.  Needs a B200.

Tolerance: a radix-R stage sums R products, at most a relative (R + 2) eps of the inputs' norm in each output
of norm sqrt(R): eps sum (R + 2) over the stages of all axes bounds the relative L2 error."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _primes(n):
    out, p = [], 2
    while n > 1:
        while n % p == 0:
            out.append(p)
            n //= p
        p += 1
    return out


@pytest.mark.parametrize("dims,batch", [
    ((997,), 1), ((1009,), 3), ((2,), 5), ((1, 7), 3),
    ((2, 5), 7), ((3, 1000), 2), ((5, 33, 2), 3), ((7, 2, 100), 2), ((15, 24), 5), ((16, 24), 5), ((17, 24), 5),
    ((31, 64), 2), ((24, 3, 5, 8), 3), ((2, 2, 2, 2), 9), ((100, 1, 20), 3),
])
def test_fft_matches_numpy(pk, dims, batch):
    from pkde_b200 import raw
    rng = np.random.default_rng(sum(dims))
    x = rng.standard_normal((batch,) + dims[::-1]) + 1j * rng.standard_normal((batch,) + dims[::-1])
    axes = tuple(range(1, x.ndim))
    tol = np.finfo(np.float64).eps * sum(p + 2 for d in dims for p in _primes(d))
    for direction, want in ((-1, np.fft.fftn(x, axes=axes)), (1, np.fft.ifftn(x, axes=axes))):
        got = raw.fft(x, direction)
        assert np.linalg.norm(got - want) <= (tol + 1e-15) * np.linalg.norm(want)
