"""Shell samples over the ranges of coordinates that decide between forms: lattices far from the origin (face
candidates narrowed or not, edges met plane by plane or node by node) and small scales that keep their
faces. The same edge points and face points as the oracle's."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _mesh(kind):
    rng = np.random.default_rng(5)
    if kind == "large":  # a few triangles across the whole grid: edges with more hits than are sorted in registers
        V = rng.uniform(0, 1, (60, 3))
    elif kind == "lattice":
        V = rng.integers(0, 17, (90, 3)) / 16.0
    else:
        V = (rng.uniform(0.1, 0.9, (150, 1, 3)) + 0.08 * rng.standard_normal((150, 3, 3))).reshape(-1, 3)
    return V, np.arange(len(V), dtype=np.int32).reshape(-1, 3)


# Cells from the origin at res 16: 5e5 and 1.6e6 (faces are narrowed up to 1e6), 9.6e11 and 1.1e12 (edges go by planes
# up to 1e12), 1.6e14, and 1.6e16 (a coordinate's rounding is two cells).
@pytest.mark.parametrize("kind", ["large", "lattice", "middling"])
@pytest.mark.parametrize("res", [4, 16])
@pytest.mark.parametrize("shift,scale", [(0.0, 0.125), (0.0, 30.0), (3.1e4, 1.0), (1e5, 1.0), (-1e6, 1.0), (1e6, 0.125),
                                         (6e10, 1.0), (7e10, 1.0), (1e13, 1.0), (1e15, 1.0), (1e12, 2.0 ** -10)])
def test_same_points(ctx, kind, res, shift, scale):
    from its_b200 import Svo
    V, F = _mesh(kind)
    V = V * scale + shift
    o, w = np.full(3, shift), np.full(3, scale)
    pts_ref, ne_ref = oracle.Svo(V, F, res, o, w).intersections()
    pts, ne = Svo(ctx, V, F, res, o, w).shell_samples(V, F)
    # (where coordinates round by more than the oracle's sweep tolerance, 1e-9, it finds other faces)
    near = abs(shift) <= 1e6
    assert ne == ne_ref > 100 and (not near or len(pts) == len(pts_ref) > ne + 30)
    for a, b in ((pts[:ne], pts_ref[:ne]), (pts[ne:], pts_ref[ne:]))[:2 if near else 1]:
        assert np.array_equal(a[np.lexsort(a.T)], b[np.lexsort(b.T)])
