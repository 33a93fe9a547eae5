"""The residual's rows a depth at a time (batches with many rows above the finest depth) against the
single octree's two bands, and a batch's learned starts, features and shares in one launch against
each octree's own: more octrees than a launch carries inline, of several depths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [2, 17, 60])
def test_batch_equals_the_single_octrees(ctx, count):
    from its_b200 import Svo, meshes, model_to_unit_cube, sharenet, uniform_bbox
    from its_b200.api import ShareNet, exact_start_batch, fit_residual_batch, learned_start_batch
    params, norm = sharenet.load()
    net = ShareNet(ctx, batch=4096, params=params)
    svos, bs = [], []
    for i in range(count):
        V, F = meshes.torus_mesh(0.75, 0.15 + 0.01 * (i % 7), 60 + i, 30)
        V = model_to_unit_cube(V)
        o, _, w = uniform_bbox(V)
        svos.append(Svo(ctx, V, F, (16, 64, 128)[i % 3], o, w))
        bs.append(ctx.signed_distance(svos[-1].vertices()[0], V, F))
    lams = learned_start_batch(svos, net, bs, norm)
    for s, b, lam in zip(svos, bs, lams):
        assert np.array_equal(lam, learned_start_batch([s], net, [b], norm)[0])
    for got, s, b in zip(exact_start_batch(svos, bs), svos, bs):
        assert np.array_equal(got, s.exact_start(b))
    # arbitrary coefficients: a residual far from rounding, whichever bands its sums were formed in
    rng = np.random.default_rng(1)
    any_lam = [lam + 0.1 * np.abs(b).max() * rng.standard_normal(lam.shape) for lam, b in zip(lams, bs)]
    batch = fit_residual_batch(svos, bs, any_lam)
    single = np.array([s.residual(b, x) for s, b, x in zip(svos, bs, any_lam)])
    assert np.all(np.abs(batch - single) <= 1e-12 * single)
    assert fit_residual_batch(svos, bs, lams).max() <= 1e-13
