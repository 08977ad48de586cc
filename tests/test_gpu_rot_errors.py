"""A :rot call that is refused for its data leaves the caller's density as it was.  Needs a B200."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(100,), (40, 33), (16, 20, 12)])
@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("bad", [9.0, np.nan])
def test_refused_data_leaves_the_density(pk, dims, device, bad):
    import torch
    from pkde_b200 import raw
    x = np.random.default_rng(1).standard_normal((500, len(dims)))
    grid = pk.initialize_grid([(-7.0, 7.0, d) for d in dims])
    wrong = x.copy()
    wrong[123, -1] = bad
    density = np.full(int(np.prod(dims)), 3.25)
    if device:
        x, wrong, density = (torch.from_numpy(a).cuda() for a in (x, wrong, density))
    with pytest.raises(pk.ArgumentError, match="beyond grid"):
        raw.rot(grid, wrong, density=density, device=device)
    assert (density == 3.25).all()
    raw.rot(grid, x, density=density, device=device)  # the context is usable
    want = raw.rot(grid, np.ascontiguousarray(x.cpu().numpy()) if device else x)
    assert np.array_equal(density.cpu().numpy() if device else density, want)
