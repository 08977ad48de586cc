"""Bandwidth steps along axes of 2^a 3^b 5^c points (passes compiled for the length) against the
FP64 oracle: the shortest and the longest such lengths, two, four and eight or more lines a tile,
a last stage of radix 3 and 5, one or two of its butterflies a thread, interleaved sub-lines
(3 2^m, 5 2^m), tiles that the lines do not fill, an odd number of bootstraps.  Needs a B200."""
import numpy as np
import pytest

from test_gpu_parity import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,n,B,steps", [
    ((18, 25), 600, 5, 12),        # shortest; two stages only
    ((27, 30), 800, 4, 10),        # radix 3 three times; three different radices
    ((24, 40, 20), 3000, 3, 6),    # interleaved sub-lines of each kind, 3-D
    ((100, 96), 3000, 5, 9),       # 4 row pairs a tile
    ((96, 101), 3000, 4, 5),       # rows that do not fill the last tile
    ((250, 54), 5000, 3, 5),       # most warps a tile of 8 lines
    ((270, 36), 5000, 4, 5),       # 4 lines a tile
    ((512, 500), 5000, 2, 3),
    ((540, 45), 5000, 3, 4),       # 2 lines a tile: one row of z and w
    ((50, 1000), 5000, 3, 4),
    ((972, 48), 5000, 2, 4),       # longest without a factor 5
    ((48, 960, 18), 8000, 2, 3),   # longest with sub-lines, between two axes
])
def test_lengths_match_oracle(pk, oracle, dims, n, B, steps):
    rng = np.random.default_rng(3 * sum(dims) + B)
    data = rng.standard_normal((len(dims), n))
    _compare(pk, oracle, data, oracle.find_grid(data, grid_dims=dims), B, n_steps=steps).check()
