"""1-D bandwidth steps (one launch for all steps) against the plain form, whose kernels apply
the same operations in the same order: identical results, bit for bit, at the lengths where
the tiles change -- one line a tile, several, a line that takes the SM alone, the z and the w
line one after the other, prime radices first and last.  Power-of-two lengths from 256 fuse
operations the plain form rounds one by one, so they are compared with the FP64 oracle.
Needs a B200."""
import numpy as np
import pytest

from test_gpu_parity import _compare

pytestmark = pytest.mark.gpu


def _run(grid, x, B, steps):
    from pkde_b200 import raw
    G = int(np.prod(grid.dims))
    d, s = np.empty(G), np.empty(G, dtype=np.int32)
    raw.gradepro_host(grid, np.ascontiguousarray(x.T), d, s, seed=3, n_bootstraps=B, n_steps=steps)
    return d, s


@pytest.mark.parametrize("n,B", [(2, 2), (7, 300), (17, 33), (128, 129), (255, 7), (343, 12), (500, 100), (961, 5),
                                 (1420, 6), (1421, 5), (2500, 9), (2867, 4), (2868, 3), (4093, 2), (4095, 5)])
def test_any_length_equals_plain_form(pk, n, B):
    from pkde_b200 import _lib
    rng = np.random.default_rng(n)
    x = rng.standard_normal((1, 700))
    grid = pk.initialize_grid([(-6.0, 6.0, n)])
    d, s = _run(grid, x, B, 9)
    _lib.set_step_path(_lib.PKDE_STEPS_PER_STEP_LAUNCH)
    try:
        dp, sp = _run(grid, x, B, 9)
    finally:
        _lib.set_step_path(_lib.PKDE_STEPS_AUTO)
    assert np.array_equal(s, sp)
    assert np.array_equal(d, dp, equal_nan=True)


@pytest.mark.parametrize("n,B", [(256, 5), (512, 20), (1024, 7), (2048, 6), (4096, 3)])
def test_powers_of_two_match_oracle(pk, oracle, n, B):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((1, 4000))
    _compare(pk, oracle, x, oracle.find_grid(x, grid_dims=(n,)), B, n_steps=20).check()
