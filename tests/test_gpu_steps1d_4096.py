"""1-D steps of 4096 points (z and w in turn on register tiles): one pair, a last pair without its second
half, many pairs, against the FP64 oracle; several in a call equal each alone.  Needs a B200."""
import numpy as np
import pytest

from test_gpu_parity import _compare
from test_gpu_steps1d import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,steps", [(2, 4), (3, 12), (33, 8)])
def test_matches_oracle(pk, oracle, B, steps):
    x = np.random.default_rng(B).standard_normal((1, 4000))
    _compare(pk, oracle, x, oracle.find_grid(x, grid_dims=(4096,)), B, n_steps=steps).check()


def test_several_in_a_call(pk):
    from pkde_b200 import raw
    jobs, alone = [], []
    for B, steps in ((2, 5), (7, 30), (20, 9)):
        x = np.random.default_rng(steps).standard_normal((1, 900))
        grid = pk.initialize_grid([(-40.0, 40.0, 4096)])  # NaN means at most points
        alone.append(_run(grid, x, B, steps))
        jobs.append(dict(grid=grid, data=np.ascontiguousarray(x.T), density=np.empty(4096),
                         selected=np.empty(4096, dtype=np.int32), seed=3, n_bootstraps=B, n_steps=steps))
    raw.gradepro_batch(jobs)
    for j, (d, s) in zip(jobs, alone):
        assert np.array_equal(j["selected"], s) and np.array_equal(j["density"], d, equal_nan=True)
