"""The estimators' binning (lanes are resamples, samples pass in cell order) at the counts where
its split changes: one, two, three and five groups of resamples, a warp's samples ragged, long
runs of one cell, every dimension, one sample drawn throughout a resample.  The sums are exact
integers, so the order of the samples must not change a bit of the result; and whole
estimations with three and five groups agree with the FP64 oracle.  Needs a B200."""
import numpy as np
import pytest

from oracle.rng import bootstrap_indices
from test_gpu_parity import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,n,B", [((40,), 31, 2), ((64,), 1000, 33), ((30,), 130, 65), ((50,), 300, 130),
                                      ((12, 10), 4001, 32), ((6, 5, 7), 2000, 5), ((5, 4, 3, 4), 700, 34),
                                      ((8, 8), 262147, 3)])
def test_sample_order_changes_nothing(pk, dims, n, B):
    from pkde_b200 import raw
    rng = np.random.default_rng(n + B)
    x = rng.standard_normal((n, len(dims)))
    if n == 2000:
        x[: n // 2] *= 0.1  # half of the samples in a few cells
    grid = pk.find_grid(x.T, grid_dims=dims)
    idx = bootstrap_indices(11, n, B)
    idx[0] = 1 + n // 2  # resample 0 draws one sample throughout
    perm = rng.permutation(n)  # sample perm[i] comes i-th, so index k + 1 becomes at[k] + 1
    at = np.empty(n, dtype=np.int32)
    at[perm] = np.arange(n, dtype=np.int32)
    out = []
    for data, draws in ((x, idx), (np.ascontiguousarray(x[perm]), np.ascontiguousarray(at[idx - 1] + 1))):
        d, s = np.empty(len(grid)), np.empty(len(grid), dtype=np.int32)
        raw.gradepro_host(grid, data, d, s, idx=draws.astype(np.int32), n_bootstraps=B, n_steps=5,
                          bw_final=[0.3] * len(dims))
        out.append((d, s))
    assert np.array_equal(out[0][1], out[1][1])
    assert np.array_equal(out[0][0], out[1][0], equal_nan=True)


@pytest.mark.parametrize("dims,n,B", [((30,), 3000, 65), ((50,), 5000, 130)])
def test_groups_of_resamples_match_oracle(pk, oracle, dims, n, B):
    data = np.random.default_rng(B).standard_normal((len(dims), n))
    _compare(pk, oracle, data, oracle.find_grid(data, grid_dims=dims), B, n_steps=8).check()
