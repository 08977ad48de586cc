"""The convergence walks of many estimations in a launch: each estimation of a batch gets what it
gets alone, bit for bit, with one, as many as a launch holds, one more, and two launches and one.
Needs a B200."""
import numpy as np
import pytest

from test_gpu_batch import _alone, _batch_jobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 24, 25, 49])
def test_walks_together_equal_alone(pk, count):
    from pkde_b200 import raw
    rng = np.random.default_rng(count)
    mix = []
    for e in range(count):  # sizes around the 16 points of a block; 1-D and 2-D walks
        dims = ((15 + e,), (5, 3 + e))[e % 2]
        x = rng.standard_normal((len(dims), 200 + e))
        mix.append((pk.find_grid(x, grid_dims=dims), x, dict(n_bootstraps=3 + e % 4, n_steps=3 + e)))
    jobs = _batch_jobs(mix)
    raw.gradepro_batch(jobs)
    for e, ((grid, x, kw), j) in enumerate(zip(mix, jobs)):
        dens, sel = _alone(pk, grid, x, kw, 100 + e)
        assert np.array_equal(j["selected"], sel)
        assert np.array_equal(j["density"], dens, equal_nan=True)
