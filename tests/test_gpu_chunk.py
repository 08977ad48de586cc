"""N-D bandwidth steps in chunks of steps (one launch per pass for several steps) against the
FP64 oracle, at the shapes where its tiles and chunks change: one line a tile, one line an
array, prime radices as the first and as the only stage, every kind of axis as first and as
last axis, the last tile ragged, one bootstrap pair without its second half, several pair
groups a step, f and means kept for one chunk only.  Needs a B200."""
import numpy as np
import pytest

from test_gpu_parity import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,n,B,steps", [
    ((2, 3), 50, 2, 4),               # one butterfly a line
    ((7, 11), 300, 5, 6),             # a generic radix is the only stage
    ((49, 77), 2000, 4, 6),           # generic radices first and last
    ((1024, 3), 3000, 3, 5),          # longest line of the row tiles: one row of z and w
    ((3, 1024), 3000, 3, 5),          # longest line of the column tiles
    ((1009, 4), 3000, 2, 4),          # a prime axis
    ((511, 5), 3000, 3, 5),           # other radices' factors in shared memory, up to 512 points
    ((514, 22), 3000, 3, 5),          # and from the L1; an odd number of lines in pairs
    ((13, 26, 11), 3000, 4, 6),       # one butterfly a line; two lines an item, three axes
    ((33, 33), 3000, 37, 40),         # several steps a chunk, an odd number of bootstraps
    ((96, 100), 5000, 6, 8),          # mixed-radix rows, Stockham columns
    ((100, 40, 16), 5000, 4, 5),      # mixed-radix columns that read the spectra
    ((20, 48, 10), 5000, 4, 6),       # mixed-radix columns in place
    ((10, 12, 14, 9), 4000, 3, 4),    # 4-D
    ((64, 64), 5000, 6, 20),          # powers of two: register tiles
    ((16, 16), 500, 5, 40),           # shortest lines; more steps than a CTA holds spectra for
    ((1024, 16), 5000, 3, 5),         # longest rows: z and w are the whole CTA
    ((16, 1024), 5000, 4, 5),         # longest columns
    ((256, 32, 64), 8000, 5, 6),      # a pass in place between the two
    ((64, 48, 32), 8000, 4, 6),       # register tiles first and last, mixed radix between
    ((300, 300), 20000, 35, 4),       # several pair groups a step
    ((1000, 900), 20000, 2, 38),      # f and means of one chunk at a time
])
def test_chunk_shapes_match_oracle(pk, oracle, dims, n, B, steps):
    rng = np.random.default_rng(sum(dims) + B)
    data = rng.standard_normal((len(dims), n))
    _compare(pk, oracle, data, oracle.find_grid(data, grid_dims=dims), B, n_steps=steps).check()
