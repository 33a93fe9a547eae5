"""The autotuner's choices for the dense field: a grid that is coarse against the octree and one of the same
resolution over a smaller box, which is not, have different candidates and so keys of their own."""
import numpy as np
import pytest

from conftest import prepared_mesh

pytestmark = pytest.mark.gpu
R = 40  # over the octree's box, too few cells a point apart for the fine candidates; over a quarter of it, fine


def run(cache, files=()):
    from its_b200 import Context, Svo
    V, F, o, w = prepared_mesh("c0")
    ctx = Context(0)
    svo = Svo(ctx, V, F, 32, o, w)
    lam = np.random.default_rng(0).standard_normal(svo.num_verts)
    if cache:
        cache.write_text("".join(line % svo.depth + "\n" for line in files))
        ctx.set_autotune(True, str(cache))
    fields = [f(lam, o, box * w, R) for f in (svo.eval_grid, svo.eval_grid_f32) for box in (1.0, 0.25)]
    choices = ctx.autotune_choices()
    svo.close()
    ctx.close()
    return fields, choices


def test_a_box_of_each_kind_has_its_own_choice(tmp_path):
    default, _ = run(None)
    fields, choices = run(tmp_path / "tune.txt")
    for a, b in zip(fields, default):
        assert np.array_equal(a, b)
    for t in ("f64", "f32"):
        assert len([k for k in choices if k.startswith("eval_grid/%s/grid=%d/" % (t, R))]) == 2


@pytest.mark.parametrize("k", [0, 1])
def test_every_candidate_of_coarse_grids_computes_the_same_bits(tmp_path, k):
    default, _ = run(None)
    fields, choices = run(tmp_path / "tune.txt", ["eval_grid/%s/grid=%d/octree=32/depth=%%d/coarse %d" % (t, R, k)
                                                  for t in ("f64", "f32")])
    assert [v for c, v in choices.items() if c.endswith("/coarse")] == [k, k]
    for a, b in zip(fields, default):
        assert np.array_equal(a, b)
