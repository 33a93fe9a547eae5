"""The dense field on lattices of any direction, place and size, by every kernel that the autotuner may pick:
lattices that run backwards along some axes, lie off the octree, or take steps of more than 2^32 cells
have no box of cells to stage. The oracle's field bit for bit."""
import numpy as np
import pytest

import oracle
from conftest import prepared_mesh

pytestmark = pytest.mark.gpu

R = 80
BOXES = [((0, 0, 0), (1, 1, 1)), ((1, 0, 0), (-1, 1, 1)), ((1, 1, 1), (-1, -1, -1)), ((0, 1, 0), (1, -1, 0.3)),
         ((0.2, 0.2, 0.9), (0.5, 0.01, -0.001)), ((-3, 0, 0), (2.5, 1, 1)), ((0.3, 0.4, 0.2), (5e10, 1, 1)),
         ((0, 0, 0), (0, 1, 1)), ((0.5, 0.5, 0.5), (1, 1, -1e13))]


@pytest.fixture(scope="module")
def scene():
    V, F, o, w = prepared_mesh("c0")
    ref = oracle.Svo(V, F, 32, o, w)
    lam = np.random.default_rng(0).standard_normal(sum(ref.depth_counts()[1]))
    return V, F, o, w, lam, [ref.eval_grid(lam, o + np.array(a) * w, np.array(b) * w, R).ravel() for a, b in BOXES]


@pytest.mark.parametrize("choice", [None, 0, 1, 2, 3, 4, 5])
def test_lattices(tmp_path, scene, choice):
    from its_b200 import Context, Svo
    V, F, o, w, lam, want = scene
    ctx = Context(0)
    svo = Svo(ctx, V, F, 32, o, w)
    if choice is not None:
        cache = tmp_path / "tune.txt"
        key = "eval_grid/f64/grid=%d/octree=32/depth=%d" % (R, svo.depth)
        cache.write_text("%s %d\n%s/coarse %d\n" % (key, choice, key, choice % 2))
        ctx.set_autotune(True, str(cache))
    for (a, b), field in zip(BOXES, want):
        got = svo.eval_grid(lam, o + np.array(a) * w, np.array(b) * w, R)
        assert np.array_equal(got, field), (a, b)
    svo.close()
    ctx.close()
