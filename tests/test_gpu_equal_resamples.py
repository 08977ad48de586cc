"""Samples that are all the same: every resample is alike, and the variance over the bootstraps is nothing but the
rounding of each ratio, so one operation fused in another way shows at every length.  The chunked steps
against the persistent engine, bit for bit.  Needs a B200."""
import numpy as np
import pytest

from test_gpu_chunk_memory import Context
from test_gpu_engine import EngineContext
from test_gpu_paths import _path

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [
    (64, 64), (256, 32), (16, 16, 16), (32, 16, 64),       # power-of-two register tiles
    (96, 40), (100, 75), (24, 20, 12), (24, 24, 8, 8),     # compiled for the length
    (77, 41), (91, 64), (5, 16), (50, 41, 6), (7, 9, 6, 8),  # runtime stages
])
@pytest.mark.parametrize("B", [5, 12])
def test_chunks_equal_engine(pk, dims, B):
    x = np.repeat(np.random.default_rng(sum(dims)).standard_normal((len(dims), 1)), 60, axis=1)
    grid = pk.initialize_grid([(-7.3, 7.1, d) for d in dims])
    with Context() as ctx:
        assert ctx.lib.pkde_set_autotune(ctx.handle, 0) == 0
        d0, s0, launches = ctx.estimate(grid, x, B, 25, bw_final=0.8)
        assert _path(launches) == "chunks"
    with EngineContext() as ctx:
        assert ctx.lib.pkde_set_autotune(ctx.handle, 0) == 0
        d1, s1, launches = ctx.estimate(grid, x, B, 25, bw_final=0.8)
        assert _path(launches) == "engine"
    assert np.array_equal(s0, s1)
    assert np.array_equal(d0, d1, equal_nan=True)
