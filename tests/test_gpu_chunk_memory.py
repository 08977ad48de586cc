"""The memory limits of the chunked N-D steps: PKDE_RING_BUDGET_MB, contexts whose autotuning is
off, and a device that is out of memory make the chunks smaller -- several chunks, a step in
groups of bootstrap pairs with the running variance in memory between them, f and means of one chunk at a time
-- and change no bit of the results.  The launch counts say that the limit took effect.  Needs a B200."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


class Context:
    def __init__(self):
        from pkde_b200 import _lib
        self.lib, self.handle = _lib.load(), ctypes.c_void_p()
        assert self.lib.pkde_create(ctypes.byref(self.handle), 0) == 0

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.lib.pkde_destroy(self.handle)

    def estimate(self, grid, x, B, steps, seed=3, **kw):
        """(density, selected, launches per phase)"""
        from pkde_b200 import _lib
        p = _lib.make_params(_lib.make_grid_struct(grid.lo, grid.hi, grid.h, grid.dims), B, steps, **kw)
        data, G = np.ascontiguousarray(x.T), int(np.prod(grid.dims))
        d, s, st = np.empty(G), np.empty(G, dtype=np.int32), _lib.PkdeStats()
        self.lib.pkde_get_stats(self.handle, ctypes.byref(st), 1)
        rc = self.lib.pkde_gradepro_estimate(self.handle, ctypes.byref(p), _lib.ptr(data), data.shape[0], None, seed,
                                             _lib.ptr(d), _lib.ptr(s), 0, None)
        _lib.check(rc, self.handle)
        self.lib.pkde_get_stats(self.handle, ctypes.byref(st), 1)
        return d, s, {p: int(st.phase_launches[i]) for i, p in enumerate(_lib.PHASES)}


def _problem(pk, dims, n=4000):
    x = np.random.default_rng(sum(dims)).standard_normal((len(dims), n))
    return pk.find_grid(x, grid_dims=dims), x


def _launches(dims, B, S, chunk_mb, keep_mb):
    """Launches of the variance rows, and of the means' rows and the convergence walks, at these limits."""
    G, pairs = int(np.prod(dims)), (B + 1) // 2
    step = 16 * (2 * pairs + 1) * G
    chunks = -(-S // max(1, min(S, chunk_mb * MB // step)))
    groups = 1 if step <= chunk_mb * MB else -(-pairs // max(1, chunk_mb * MB // (32 * G)))
    return chunks * groups, chunks + (1 if 16 * S * G <= keep_mb * MB else chunks)


@pytest.mark.parametrize("dims,B,steps", [
    ((257, 241), 271, 4),      # any length: pair groups, all steps kept; the last pair has no second half
    ((257, 241), 270, 139),    # and f and means of one step at a time
    ((257, 241), 20, 139),     # several steps a chunk, f and means of one chunk at a time
    ((257, 241), 20, 29),      # several chunks, all steps kept
    ((240, 250), 279, 5),      # 2^a 3^b 5^c lengths
    ((240, 250), 20, 140),
    ((192, 320), 274, 4),      # mixed radices
    ((256, 256), 261, 4),      # powers of two
    ((256, 256), 20, 130),
    ((64, 32, 32), 260, 4),    # with a pass in place between
    ((16, 16, 15, 16), 280, 3),
])
def test_small_chunks_keep_results(pk, monkeypatch, dims, B, steps):
    grid, x = _problem(pk, dims)
    S = steps + 1
    with Context() as ctx:
        d0, s0, free = ctx.estimate(grid, x, B, steps)
        monkeypatch.setenv("PKDE_RING_BUDGET_MB", "1")
        d1, s1, capped = ctx.estimate(grid, x, B, steps)
    vmr, means = _launches(dims, B, S, 256, 128)
    assert (free["step_vmr"], free["step_means"]) == _launches(dims, B, S, 8192, 8192) and vmr > free["step_vmr"]
    assert (capped["step_vmr"], capped["step_means"]) == (vmr, means)
    assert np.array_equal(s0, s1)
    assert np.array_equal(d0, d1, equal_nan=True)


def test_batch_in_small_chunks_keeps_results(pk, monkeypatch):
    from pkde_b200 import raw
    jobs = []
    for e, (dims, B, steps) in enumerate([((257, 241), 271, 5), ((240, 250), 20, 140), ((64, 64), 5, 10)]):
        grid, x = _problem(pk, dims)
        G = int(np.prod(dims))
        jobs.append(dict(grid=grid, data=np.ascontiguousarray(x.T), density=np.empty(G),
                         selected=np.empty(G, dtype=np.int32), seed=e, n_bootstraps=B, n_steps=steps))
    raw.gradepro_batch(jobs)
    want = [(j["density"].copy(), j["selected"].copy()) for j in jobs]
    monkeypatch.setenv("PKDE_RING_BUDGET_MB", "1")
    raw.gradepro_batch(jobs)
    for j, (d, s) in zip(jobs, want):
        assert np.array_equal(j["density"], d, equal_nan=True) and np.array_equal(j["selected"], s)


def test_limits_bound_the_scratch(pk, monkeypatch):
    """512 x 512, 64 bootstraps, 21 steps: 5.7 GB of intermediates in one chunk; the spectra and the
    binning take 1.4 GB at any limit."""
    import torch
    grid, x = _problem(pk, (512, 512), 20000)

    def used(**kw):
        with Context() as ctx:
            if kw.get("autotune_off"):
                assert ctx.lib.pkde_set_autotune(ctx.handle, 0) == 0
            before = torch.cuda.mem_get_info(0)[0]
            d, s, launches = ctx.estimate(grid, x, 64, 20)
            return before - torch.cuda.mem_get_info(0)[0], launches["step_vmr"], d, s

    used()  # kernels loaded
    plain, one, d0, s0 = used()
    assert one == 1 and plain > 5 << 30
    off, many, d, s = used(autotune_off=True)
    assert many > 1 and off < plain - (4 << 30)
    assert np.array_equal(d, d0) and np.array_equal(s, s0)
    monkeypatch.setenv("PKDE_RING_BUDGET_MB", "3000")
    some, few, d, s = used()
    assert few == 3 and some < plain - (3 << 30)  # 2 GB a chunk
    assert np.array_equal(d, d0) and np.array_equal(s, s0)


def test_failed_scratch_allocation_takes_smaller_chunks(pk):
    from pkde_b200 import _lib
    grid, x = _problem(pk, (512, 512), 20000)
    with Context() as ctx:
        assert ctx.lib.pkde_set_fault(ctx.handle, _lib.PKDE_FAULT_SCRATCH_ALLOC) == 0
        d1, s1, launches = ctx.estimate(grid, x, 64, 20)
        assert launches["step_vmr"] == 3
        d0, s0, launches = ctx.estimate(grid, x, 64, 20)
        assert launches["step_vmr"] == 1
    assert np.array_equal(d0, d1) and np.array_equal(s0, s1)
