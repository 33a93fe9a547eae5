"""Marching cubes with each run of voxels per lane (4, 8, 16) on grids whose rows are no multiple of it, so that
runs cross from one row into the next: forced on small grids, and by default on one of more than 2^26
voxels. Cases and soup against the oracle's, bit for bit."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

O, W = np.array([0.1, -0.2, 0.3]), np.array([1.0, 1.1, 0.9])


def compare(ctx, f, R):
    cube, tri, n = ctx.marching_cubes(f, R, O, W, 0.05)
    want_cube, want_tri, want_n = oracle.marching_cubes(f, R, O, W, 0.05)
    assert n == want_n > 0 and np.array_equal(cube, want_cube)
    assert np.array_equal(tri, np.asarray(want_tri).reshape(-1, 3)[:n])


@pytest.mark.parametrize("R", [15, 16, 17, 19, 33, 47, 81])
@pytest.mark.parametrize("choice", [0, 1, 2])
def test_runs_across_rows(tmp_path, R, choice):
    from its_b200 import Context
    ctx = Context(0)
    cache = tmp_path / "tune.txt"
    keys = ["marching_cubes/f64/res=%d/%s" % (R, form) for form in ("cases", "soup")]
    cache.write_text("".join("%s %d\n" % (k, choice) for k in keys))
    ctx.set_autotune(True, str(cache))
    compare(ctx, np.random.default_rng(R).standard_normal((R + 1) ** 3), R)
    assert all(ctx.autotune_choices()[k] == choice for k in keys)
    ctx.close()


def test_largest_default(ctx):
    R = 411
    g = np.linspace(-1, 1, R + 1)
    f = g[:, None, None] ** 2 + g[None, :, None] ** 2 + g[None, None, :] ** 2 - 0.6 + 0.1 * np.sin(37 * g)
    compare(ctx, f.ravel(), R)
