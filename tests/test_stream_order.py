"""Everything a call queues goes to the call's own stream.  Tables that a context uploads on first use (twiddles,
reciprocals) are read by the next kernels, so a copy on the legacy stream -- which may return before
its last part has arrived, and which a non-blocking stream does not wait for -- would be a race.  The order
is read from the sources; on a GPU, first uses on a non-blocking stream equal later ones."""
import ctypes
import glob
import os
import re

import numpy as np
import pytest

from conftest import REPO

CSRC = os.path.join(REPO, "parallelkde.jl_b200", "csrc")


def test_no_copy_or_launch_outside_the_stream():
    files = sorted(glob.glob(os.path.join(CSRC, "*.cu*")))
    assert files
    for f in files:
        text = re.sub(r"//[^\n]*", "", open(f).read())
        for call in ("cudaMemcpy", "cudaMemset", "cudaMemcpyToSymbol", "cudaMemcpy2D"):
            assert not re.search(rf"\b{call}\s*\(", text), (os.path.basename(f), call)
        for m in re.finditer(r"<<<(.*?)>>>", text, re.S):
            assert m.group(1).split(",")[-1].strip() == "st", (os.path.basename(f), m.group(0))


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(3000,), (4096,), (1021,), (100, 96), (64, 120), (77, 50), (40, 1500)])
def test_first_use_on_a_non_blocking_stream(pk, dims):
    import torch
    from pkde_b200 import _lib
    lib = _lib.load()
    x = np.random.default_rng(5).standard_normal((len(dims), 3000))
    grid = pk.find_grid(x, grid_dims=dims)
    p = _lib.make_params(_lib.make_grid_struct(grid.lo, grid.hi, grid.h, grid.dims), 7, 12)
    data, G = np.ascontiguousarray(x.T), int(np.prod(dims))
    stream = torch.cuda.Stream()  # non-blocking
    outs = []
    for _ in range(3):  # contexts with no table yet
        ctx = ctypes.c_void_p()
        assert lib.pkde_create(ctypes.byref(ctx), 0) == 0
        try:
            assert lib.pkde_set_autotune(ctx, 0) == 0
            for _ in range(2):
                d, s = np.empty(G), np.empty(G, dtype=np.int32)
                rc = lib.pkde_gradepro_estimate(ctx, ctypes.byref(p), _lib.ptr(data), data.shape[0], None, 3,
                                                _lib.ptr(d), _lib.ptr(s), 0, stream.cuda_stream)
                _lib.check(rc, ctx)
                outs.append((d, s))
        finally:
            lib.pkde_destroy(ctx)
    for d, s in outs[1:]:
        assert np.array_equal(s, outs[0][1]) and np.array_equal(d, outs[0][0])
