"""The dense field by prolongation: walks of one and of several coarse intervals, each factor."""
import numpy as np
import pytest

from cascade_np import cascade_numpy
from conftest import prepared_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res,f", [(2, 1), (2, 8), (4, 2), (8, 4), (16, 8), (64, 1), (128, 1), (128, 2), (128, 4)])
def test_walks(ctx, res, f):
    from its_b200 import Svo
    V, F, o, w = prepared_mesh("small")
    svo = Svo(ctx, V, F, res, o, w)
    lam = np.random.default_rng(res + f).uniform(-1, 1, svo.num_verts)
    depth = len(svo.depth_counts()[1])
    unit = np.full(3, np.asarray(w, float)[0] / res)
    want = cascade_numpy(svo.vertices()[0], lam, svo.depth_counts()[1], np.asarray(o, float), unit, res, f)
    want = want.transpose(2, 1, 0).ravel()
    # ten roundings per level of values that sum at most one unit per level, on both sides
    roundings = 20 * (depth + 1) * (depth + 1)
    assert np.abs(svo.eval_grid_fast(lam, o, w, res * f) - want).max() <= roundings * 2.0 ** -53
    fast32 = svo.eval_grid_fast(lam, o, w, res * f, fp32=True)
    assert np.abs(fast32 - want).max() <= roundings * 2.0 ** -24
