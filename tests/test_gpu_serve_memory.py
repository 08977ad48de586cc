"""What a serving lane admits into a wave follows the memory that a request holds.  Needs a B200."""
import ctypes

import numpy as np
import pytest

from test_gpu_chunk_memory import Context

pytestmark = pytest.mark.gpu


def test_two_requests_of_many_samples_share_a_wave(pk):
    """1,000,000 samples on 16^3, 2 bootstraps: 24 MB of samples, 44 MB of binning and 270 MB for the steps; two
    fit a lane of 800 MB (with 256 MB of corner terms per sample, which no estimation stores, they did not)."""
    from pkde_b200 import _lib
    from pkde_b200.serve import PkdeRequest, PkdeResult, _bind
    n, dims, count = 1_000_000, (16, 16, 16), 7
    x = np.random.default_rng(3).standard_normal((n, 3))
    grid = pk.initialize_grid([(-8.0, 8.0, d) for d in dims])
    p = _lib.make_params(_lib.make_grid_struct(grid.lo, grid.hi, grid.h, grid.dims), 2, 4)
    outs = [(np.empty(16 ** 3), np.empty(16 ** 3, dtype=np.int32)) for _ in range(count)]
    with Context() as ctx:
        lib = _bind(ctx.lib)
        assert lib.pkde_serve_config(ctx.handle, 1, 800 << 20) == 0
        tickets = []
        for d, s in outs:
            req = PkdeRequest(params=p, data=_lib.ptr(x), n=n, boot_idx=None, seed=5, density_out=_lib.ptr(d),
                              selected_out=_lib.ptr(s))
            t = ctypes.c_uint64()
            assert lib.pkde_submit(ctx.handle, ctypes.byref(req), ctypes.byref(t)) == 0
            tickets.append(t.value)
        sizes = []
        for t in tickets:
            res = PkdeResult()
            assert lib.pkde_wait(ctx.handle, t, 60_000, ctypes.byref(res)) == 0
            assert res.status == 0, res.message
            sizes.append(res.batch_size)
    assert max(sizes) == 2
    for d, s in outs[1:]:
        assert np.array_equal(d, outs[0][0]) and np.array_equal(s, outs[0][1])
