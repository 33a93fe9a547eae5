"""Signs of the distance to triangle soups, one triangle to thousands, spread out or all in one place (deep trees
of equal keys): the fast winding number's sum over the tree equals the oracle's, whose order is another, so
signs agree at points in general position."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 8, 9, 17, 65, 129, 1000, 5000])
@pytest.mark.parametrize("spread", [0.0, 0.3, 1.0])
def test_signs_of_soups(ctx, n, spread):
    rng = np.random.default_rng(n)
    # triangles that mostly face outward, so that winding numbers lie around 1/2
    c = rng.standard_normal((n, 1, 3))
    c /= np.linalg.norm(c, axis=-1, keepdims=True)
    e = rng.standard_normal((n, 3, 3)) * 2.5 / np.sqrt(n)
    V = spread * c + e
    flip = np.einsum("ij,ij->i", np.cross(V[:, 1] - V[:, 0], V[:, 2] - V[:, 0]), c[:, 0]) < 0
    V[flip] = V[flip][:, [0, 2, 1]]
    V, F = V.reshape(-1, 3), np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    P = rng.uniform(-1.5, 1.5, (3000, 3))
    got, want = ctx.signed_distance(P, V, F), oracle.signed_distance_bvh(P, V, F)
    assert np.array_equal(got, want)
    assert n < 65 or spread < 1.0 or 0 < (got < 0).sum() < len(P)
