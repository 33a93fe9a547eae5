"""Octree levels where the occupancy pyramid can go wrong: grids of one cell up to several kernels'
levels, roots below the top of the grid, one voxel, and cells at the ends of words and blocks."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _triangles(centres, size):
    rng = np.random.default_rng(7)
    V = (centres[:, None, :] + size * rng.uniform(-1, 1, (len(centres), 3, 3))).reshape(-1, 3)
    return np.clip(V, 0.0, 1.0), np.arange(len(V), dtype=np.int32).reshape(-1, 3)


def _same(gpu, ref):
    assert gpu.depth == ref.depth
    assert (gpu.num_voxels, gpu.num_fine, gpu.num_nodes, gpu.num_verts, gpu.num_edges) == \
        (ref.num_voxels, ref.num_fine, ref.num_nodes, ref.num_verts, ref.num_edges)
    assert np.array_equal(gpu.voxels(), ref.voxels())
    gn, rn = gpu.nodes(), ref.nodes()
    for k in ("morton", "parent", "childs", "is_leaf", "neighbors"):
        assert np.array_equal(gn[k], rn[k]), k
    for a, b in zip(gpu.vertices() + gpu.edges(), ref.vertices() + ref.edges()):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("res", [2, 4, 8, 16, 32, 64, 128, 256])
@pytest.mark.parametrize("kind", ["spread", "corner", "far_corner", "ends"])
def test_levels(ctx, res, kind):
    from its_b200 import Svo
    rng = np.random.default_rng(res)
    if kind == "spread":
        V, F = _triangles(rng.uniform(0, 1, (40, 3)), 0.05)
    elif kind == "corner":  # a few neighbouring cells: the root lies below the top of the grid
        V, F = _triangles(np.full((3, 3), 1.0 / res), 0.6 / res)
    elif kind == "far_corner":
        V, F = _triangles(np.full((3, 3), 1.0 - 1.0 / res), 0.6 / res)
    else:
        V, F = _triangles(np.array([[0.0, 0.0, 0.0], [1.0, 1.0, 1.0], [1.0, 0.0, 0.0], [0.5, 0.5, 0.5]]), 0.4 / res)
    o, w = np.zeros(3), np.ones(3)
    ref = oracle.Svo(V, F, res, o, w)
    if ref.num_voxels < 2:
        pytest.skip("one voxel: the next test's")
    _same(Svo(ctx, V, F, res, o, w), ref)


@pytest.mark.parametrize("res", [1, 2, 64, 256])
def test_one_voxel_is_its_own_root(ctx, res):
    from its_b200 import Svo
    V, F = _triangles(np.full((1, 3), (res - 0.5) / res), 0.2 / res)
    svo = Svo(ctx, V, F, res, np.zeros(3), np.ones(3))
    assert (svo.depth, svo.num_voxels, svo.num_nodes, svo.num_verts, svo.num_edges) == (1, 1, 1, 8, 12)
    n = svo.nodes()
    assert n["neighbors"][0, 13] == 0 and (np.delete(n["neighbors"][0], 13) == 0xFFFFFFFF).all()
    assert n["morton"][0] == svo.voxels()[0] == res ** 3 - 1 and n["is_leaf"][0] == 1
    lam = np.arange(1.0, 9.0)
    val, miss = svo.eval_points(lam, np.full((1, 3), (res - 0.5) / res))
    assert miss[0] == 0 and abs(val[0] - lam.mean()) < 1e-12
