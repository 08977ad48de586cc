"""The persistent step engine, on shapes of all its tiles: axes of more than 1024 points, which it always
runs, and others in a context with a wait limit of its own (large enough never to run out).  Schedules,
ring slots, trials, several estimations a launch and launches that fit a memory budget change no bit; the results
are those of the chunked steps where those take the shape.  Needs a B200."""
import ctypes
import threading

import numpy as np
import pytest

from test_gpu_chunk_memory import Context, _problem
from test_gpu_parity import _compare
from test_gpu_paths import _path

pytestmark = pytest.mark.gpu

# register tiles, mixed radices, Stockham stages; the last three run in the engine at any limit
SHAPES = [(64, 48), (16, 32, 16), (24, 20, 12), (96, 40), (2048, 16), (1500, 96), (30, 1025)]


class EngineContext(Context):
    def __init__(self):
        from pkde_b200 import _lib
        super().__init__()
        assert self.lib.pkde_set_wait_limit(self.handle, 10 * _lib.DEFAULT_WAIT_LIMIT) == 0


@pytest.mark.parametrize("dims", SHAPES)
def test_schedules_keep_results(pk, monkeypatch, dims):
    grid, x = _problem(pk, dims)
    outs = []
    with EngineContext() as ctx:
        assert ctx.lib.pkde_set_autotune(ctx.handle, 0) == 0
        for delay, slot_mb, tpi in ((2, 32, 2), (1, 1, 1), (1, 32, 4), (3, 1, 8), (4, 2, 2)):
            monkeypatch.setenv("PKDE_ENGINE_DELAY", str(delay))
            monkeypatch.setenv("PKDE_ENGINE_SLOT_MB", str(slot_mb))
            monkeypatch.setenv("PKDE_ENGINE_TPI", str(tpi))
            d, s, launches = ctx.estimate(grid, x, 10, 24)
            assert _path(launches) == "engine"
            outs.append((d, s))
    if max(dims) <= 1024:
        with Context() as ctx:
            d, s, launches = ctx.estimate(grid, x, 10, 24)
            assert _path(launches) == "chunks"
            outs.append((d, s))
    for d, s in outs[1:]:
        assert np.array_equal(s, outs[0][1]) and np.array_equal(d, outs[0][0])


@pytest.mark.parametrize("dims,B", [((256, 256), 80), ((2048, 32), 80)])
def test_wide_ring_slots_keep_results(pk, monkeypatch, dims, B):
    """80 MB hold all pairs of a step; 2 MB hold one."""
    grid, x = _problem(pk, dims, 20000)
    outs = []
    with EngineContext() as ctx:
        assert ctx.lib.pkde_set_autotune(ctx.handle, 0) == 0
        for slot_mb, tpi in ((128, 4), (2, 2), (8, 4), (48, 2)):
            monkeypatch.setenv("PKDE_ENGINE_SLOT_MB", str(slot_mb))
            monkeypatch.setenv("PKDE_ENGINE_TPI", str(tpi))
            d, s, launches = ctx.estimate(grid, x, B, 12)
            assert _path(launches) == "engine"
            outs.append((d, s))
    for d, s in outs[1:]:
        assert np.array_equal(s, outs[0][1]) and np.array_equal(d, outs[0][0])


def test_trials_keep_results_and_are_recorded(pk, tmp_path, monkeypatch):
    cache = tmp_path / "schedules.txt"
    monkeypatch.setenv("PKDE_TUNE_CACHE", str(cache))
    grid, x = _problem(pk, (1200, 20))
    with EngineContext() as ctx:
        assert ctx.lib.pkde_set_autotune(ctx.handle, 0) == 0
        d0, s0, launches = ctx.estimate(grid, x, 10, 20)
        assert _path(launches) == "engine" and launches["step_vmr"] == 1 and not cache.exists()
        assert ctx.lib.pkde_set_autotune(ctx.handle, 1) == 0
        d1, s1, launches = ctx.estimate(grid, x, 10, 20)
        assert launches["step_vmr"] > 1
        d2, s2, launches = ctx.estimate(grid, x, 10, 20)
        assert launches["step_vmr"] == 1
    key, slot, tpi, delay = cache.read_text().split()
    assert key == "2x1200x20:p5" and int(slot) > 0 and int(tpi) > 0 and int(delay) > 0
    for d, s in ((d1, s1), (d2, s2)):
        assert np.array_equal(s, s0) and np.array_equal(d, d0)


def _batch(ctx, problems, B, steps):
    """One call for all problems: (results, launches of the step engine)."""
    from pkde_b200 import _lib
    count = len(problems)
    params = (_lib.PkdeGradeproParams * count)()
    vp = ctypes.c_void_p
    data_p, dens_p, sel_p = (vp * count)(), (vp * count)(), (vp * count)()
    n, seeds, keep, out = (ctypes.c_int64 * count)(), (ctypes.c_uint64 * count)(), [], []
    for e, (grid, x) in enumerate(problems):
        params[e] = _lib.make_params(_lib.make_grid_struct(grid.lo, grid.hi, grid.h, grid.dims), B, steps)
        data, G = np.ascontiguousarray(x.T), int(np.prod(grid.dims))
        out.append((np.empty(G), np.empty(G, dtype=np.int32)))
        keep.append(data)
        data_p[e], dens_p[e], sel_p[e] = _lib.ptr(data), _lib.ptr(out[e][0]), _lib.ptr(out[e][1])
        n[e], seeds[e] = data.shape[0], 3
    st = _lib.PkdeStats()
    ctx.lib.pkde_get_stats(ctx.handle, ctypes.byref(st), 1)
    rc = ctx.lib.pkde_gradepro_estimate_batch(ctx.handle, count, params, data_p, n, None, seeds, dens_p, sel_p, 0, None)
    _lib.check(rc, ctx.handle)
    ctx.lib.pkde_get_stats(ctx.handle, ctypes.byref(st), 1)
    launches = {p: int(st.phase_launches[i]) for i, p in enumerate(_lib.PHASES)}
    assert _path(launches) == "engine"
    return out, launches["step_vmr"]


def test_batches_keep_results(pk, monkeypatch):
    """Two launches, of the register tiles and of the others; with no budget one an estimation."""
    problems = [_problem(pk, d) for d in SHAPES + [(32, 32), (8, 6, 10, 7)]]
    with EngineContext() as ctx:
        alone = [ctx.estimate(grid, x, 7, 15)[:2] for grid, x in problems]  # also the trials
        together, few = _batch(ctx, problems, 7, 15)
        monkeypatch.setenv("PKDE_RING_BUDGET_MB", "1")
        packed, many = _batch(ctx, problems, 7, 15)
    assert few == 2 and many == len(problems)
    for (d0, s0), (d1, s1), (d2, s2) in zip(alone, together, packed):
        assert np.array_equal(s1, s0) and np.array_equal(d1, d0)
        assert np.array_equal(s2, s0) and np.array_equal(d2, d0)


@pytest.mark.parametrize("dims,B,steps", [((1500, 24), 6, 20), ((30, 1025), 5, 12), ((2048, 16, 3), 3, 10)])
def test_long_axes_match_oracle(pk, oracle, dims, B, steps):
    data = np.random.default_rng(sum(dims)).standard_normal((len(dims), 4000))
    _compare(pk, oracle, data, oracle.find_grid(data, grid_dims=dims), B, n_steps=steps).check()


@pytest.mark.parametrize("dims,B,steps", [((64, 32), 8, 30), ((16, 20, 12), 6, 20)])
def test_plain_form_agrees(pk, dims, B, steps):
    from pkde_b200 import _lib
    grid, x = _problem(pk, dims)
    with EngineContext() as ctx:
        d0, s0, launches = ctx.estimate(grid, x, B, steps)
        assert _path(launches) == "engine"
        assert ctx.lib.pkde_set_step_path(ctx.handle, _lib.PKDE_STEPS_PER_STEP_LAUNCH) == 0
        d1, s1, _ = ctx.estimate(grid, x, B, steps)
    same = s0 == s1
    assert same.mean() >= 0.99
    assert np.linalg.norm((d0 - d1)[same]) <= 1e-10 * np.linalg.norm(d1[same])


def test_timeout_of_a_long_axis_then_recovers(pk):
    from pkde_b200 import _lib
    grid, x = _problem(pk, (2048, 64))
    with EngineContext() as ctx:
        d0, s0, _ = ctx.estimate(grid, x, 8, 30)
        assert ctx.lib.pkde_set_wait_limit(ctx.handle, 0) == 0
        with pytest.raises(_lib.CudaLibraryError, match="dependency wait timed out"):
            ctx.estimate(grid, x, 8, 30)
        assert ctx.lib.pkde_set_wait_limit(ctx.handle, _lib.DEFAULT_WAIT_LIMIT) == 0
        d1, s1, launches = ctx.estimate(grid, x, 8, 30)
        assert _path(launches) == "engine"
    assert np.array_equal(s0, s1) and np.array_equal(d0, d1)


def test_concurrent_contexts_match_alone(pk):
    problems = [_problem(pk, d) for d in SHAPES]
    with EngineContext() as ctx:
        alone = [ctx.estimate(grid, x, 6, 16)[:2] for grid, x in problems]
    errors, results = [], {}

    def worker(k):
        try:
            with EngineContext() as ctx:
                for rep in range(2):
                    for i in range(len(problems)):
                        j = (i + 3 * k + rep) % len(problems)  # the threads walk the shapes out of phase
                        results[(k, rep, j)] = ctx.estimate(*problems[j], 6, 16)
        except Exception as e:  # reported on the main thread
            errors.append(repr(e))

    threads = [threading.Thread(target=worker, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert len(results) == 2 * 2 * len(problems)
    for (k, rep, j), (d, s, launches) in results.items():
        assert _path(launches) == "engine"
        assert np.array_equal(d, alone[j][0]) and np.array_equal(s, alone[j][1]), (k, rep, SHAPES[j])
