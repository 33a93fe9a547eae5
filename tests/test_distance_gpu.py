"""The signed distance's tree and walks at the sizes where they can go wrong: one triangle, buckets
exactly full and one over, a block's leaves and one more, many triangles with equal keys, and
queries on, near and far from the surface. Distances equal the brute force's bit for bit (the same
per-triangle arithmetic, a minimum over all of them); signs those of the oracle's winding number."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _soup(n, seed, same_place):
    rng = np.random.default_rng(seed)
    c = np.zeros((n, 1, 3)) if same_place else rng.uniform(-1, 1, (n, 1, 3))
    V = (c + 0.2 * rng.standard_normal((n, 3, 3))).reshape(-1, 3)
    return V, np.arange(3 * n, dtype=np.int32).reshape(n, 3)


@pytest.mark.parametrize("n", [1, 2, 3, 8, 9, 15, 64, 65, 127, 128, 129, 257, 1000, 5000])
@pytest.mark.parametrize("same_place", [False, True])
def test_distance_to_soups(ctx, n, same_place):
    V, F = _soup(n, n, same_place)
    rng = np.random.default_rng(1)
    P = np.concatenate([V[: 3 * n : max(1, n // 50)], rng.uniform(-2, 2, (333, 3)), rng.uniform(-50, 50, (41, 3))])
    got, want = ctx.signed_distance(P, V, F), oracle.signed_distance(P, V, F)
    assert np.array_equal(np.abs(got), np.abs(want))


@pytest.mark.parametrize("m", [1, 7, 16, 17, 63, 64, 65, 1000])
def test_signs_inside_and_outside_a_closed_mesh(ctx, m):
    from its_b200 import meshes
    V, F = meshes.torus_mesh(0.75, 0.2, 40, 24)
    P = np.random.default_rng(m).uniform(-1.1, 1.1, (m, 3))
    assert np.array_equal(ctx.signed_distance(P, V, F), oracle.signed_distance_bvh(P, V, F))
