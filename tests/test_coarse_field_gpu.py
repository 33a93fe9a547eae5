"""The dense field on grids that are not twice as fine as the octree (one point or fewer per finest
cell), on boxes that are the octree's, larger, smaller and off its lattice."""
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
    lam = svo.exact_start(ctx.signed_distance(svo.vertices()[0], V, F))
    return ref, svo, lam, o, w


BOXES = [(0.0, 1.0), (-0.3, 1.7), (0.11, 0.83), (0.4, 0.05), (-3.0, 0.9)]


@pytest.mark.parametrize("R", [1, 3, 16, 31, 32, 33, 40, 63])
@pytest.mark.parametrize("box", BOXES)
def test_coarse_grid_field(sphere, R, box):
    ref, svo, lam, o, w = sphere
    bo, bw = o + box[0] * w, box[1] * w
    want = ref.eval_grid(lam, bo, bw, R).ravel()
    assert np.array_equal(svo.eval_grid(lam, bo, bw, R), want)
    # FP32: at most 8 terms per depth and three roundings each, relative to the sum of their sizes
    size = ref.eval_grid(np.abs(lam), bo, bw, R).ravel()
    assert np.all(np.abs(svo.eval_grid_f32(lam, bo, bw, R) - want) <= (8 * svo.depth + 8) * 2.0 ** -24 * size)


@pytest.mark.parametrize("R", [16, 32, 40])
def test_coefficient_that_is_not_finite_stays_in_its_cells(sphere, R):
    ref, svo, lam, o, w = sphere
    for v in (5, svo.num_verts // 2, svo.num_verts - 1):
        one, without, bad = np.zeros_like(lam), lam.copy(), lam.copy()
        one[v], without[v], bad[v] = 1.0, 0.0, np.inf
        touched = ref.eval_grid(one, o, w, R).ravel() > 0
        want = np.where(touched, np.inf, ref.eval_grid(without, o, w, R).ravel())
        assert np.array_equal(svo.eval_grid(bad, o, w, R), want)
