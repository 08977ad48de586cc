"""What chooses between the chunked steps and the persistent engine: the shape and the context's wait limit,
never a schedule that the engine's trials left in the context or in the file of schedules.  The path shows in
the launch counts: the chunked steps launch their column passes by themselves, the engine runs all passes in
one launch.  Needs a B200."""
import numpy as np
import pytest

from test_gpu_chunk_memory import Context, _problem

pytestmark = pytest.mark.gpu

DIMS, B, STEPS = (64, 48), 10, 20


def _path(launches):
    return "chunks" if launches["step_fft"] else "engine"


def _limit(ctx, polls):
    assert ctx.lib.pkde_set_wait_limit(ctx.handle, polls) == 0


def test_trials_under_a_wait_limit_leave_the_path(pk, tmp_path, monkeypatch):
    from pkde_b200 import _lib
    cache = tmp_path / "schedules.txt"
    monkeypatch.setenv("PKDE_TUNE_CACHE", str(cache))
    grid, x = _problem(pk, DIMS)
    with Context() as ctx:
        _limit(ctx, _lib.DEFAULT_WAIT_LIMIT + 1)
        d0, s0, launches = ctx.estimate(grid, x, B, STEPS)
        assert _path(launches) == "engine" and launches["step_vmr"] > 1  # with trials
        assert cache.read_text().split()[0] == "2x64x48:p5"
        _limit(ctx, _lib.DEFAULT_WAIT_LIMIT)
        d1, s1, launches = ctx.estimate(grid, x, B, STEPS)
        assert _path(launches) == "chunks"
        _limit(ctx, _lib.DEFAULT_WAIT_LIMIT + 1)
        _, _, launches = ctx.estimate(grid, x, B, STEPS)
        assert _path(launches) == "engine" and launches["step_vmr"] == 1  # the trials' schedule
    with Context() as ctx:  # a later process reads the file
        _, _, launches = ctx.estimate(grid, x, B, STEPS)
        assert _path(launches) == "chunks"
    assert len(cache.read_text().splitlines()) == 1
    assert np.array_equal(s0, s1) and np.array_equal(d0, d1)


def test_engine_is_tuned_for_a_shape_that_ran_in_chunks(pk, tmp_path, monkeypatch):
    from pkde_b200 import _lib
    cache = tmp_path / "schedules.txt"
    cache.write_text("2x64x48:p5 0 0 0\n")
    monkeypatch.setenv("PKDE_TUNE_CACHE", str(cache))
    grid, x = _problem(pk, DIMS)
    with Context() as ctx:
        d0, s0, launches = ctx.estimate(grid, x, B, STEPS)
        assert _path(launches) == "chunks" and len(cache.read_text().splitlines()) == 1
        _limit(ctx, _lib.DEFAULT_WAIT_LIMIT + 1)
        d1, s1, launches = ctx.estimate(grid, x, B, STEPS)
        assert _path(launches) == "engine" and launches["step_vmr"] > 1
        _limit(ctx, _lib.DEFAULT_WAIT_LIMIT)
        _, _, launches = ctx.estimate(grid, x, B, STEPS)
        assert _path(launches) == "chunks"
    key, *schedule = cache.read_text().splitlines()[1].split()
    assert key == "2x64x48:p5" and int(schedule[0]) > 0
    assert np.array_equal(s0, s1) and np.array_equal(d0, d1)


def test_schedule_of_an_earlier_build_leaves_the_path(pk, tmp_path, monkeypatch):
    cache = tmp_path / "schedules.txt"
    cache.write_text("2x64x48:p5 32 2 2\n2x2048x8:p5 32 2 2\n")
    monkeypatch.setenv("PKDE_TUNE_CACHE", str(cache))
    with Context() as ctx:
        _, _, launches = ctx.estimate(*_problem(pk, DIMS), B, STEPS)
        assert _path(launches) == "chunks"
        _, _, launches = ctx.estimate(*_problem(pk, (2048, 8)), B, STEPS)  # the engine's own shapes
        assert _path(launches) == "engine" and launches["step_vmr"] == 1  # no trials
    assert len(cache.read_text().splitlines()) == 2
