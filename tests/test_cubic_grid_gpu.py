"""The cubic basis' dense field: grids from far coarser than the octree (depths whose corner box fits
no tile) to four times as fine, remainders of the 32 x 8 x 8 bricks, boxes off the octree's, and
coefficients that are not finite, against the point-by-point restatement bit for bit."""
import numpy as np
import pytest

import oracle
from conftest import prepared_mesh

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sphere(ctx):
    from its_b200 import Svo
    V, F, o, w = prepared_mesh("small")
    ref, svo = oracle.Svo(V, F, 32, o, w), Svo(ctx, V, F, 32, o, w)
    lam = np.random.default_rng(0).standard_normal(svo.num_verts)
    return ref, svo, lam, o, w


@pytest.mark.parametrize("R", [1, 7, 8, 31, 32, 33, 64, 71])
@pytest.mark.parametrize("box", [(0.0, 1.0), (-0.3, 1.7), (0.11, 0.83), (0.4, 0.05), (-3.0, 0.9), (-4.0, 9.0)])
def test_cubic_grid(sphere, R, box):
    ref, svo, lam, o, w = sphere
    bo, bw = o + box[0] * w, box[1] * w
    assert np.array_equal(svo.eval_grid_cubic(lam, bo, bw, R), ref.cubic_eval_grid(lam, bo, bw, R).ravel())


@pytest.mark.parametrize("R", [20, 64])
def test_cubic_coefficient_that_is_not_finite(sphere, R):
    ref, svo, lam, o, w = sphere
    for v in (5, svo.num_verts // 2, svo.num_verts - 1):
        one, without, bad = np.zeros_like(lam), lam.copy(), lam.copy()
        one[v], without[v], bad[v] = 1.0, 0.0, np.inf
        touched = ref.cubic_eval_grid(one, o, w, R).ravel() > 0
        want = np.where(touched, np.inf, ref.cubic_eval_grid(without, o, w, R).ravel())
        assert np.array_equal(svo.eval_grid_cubic(bad, o, w, R), want)
