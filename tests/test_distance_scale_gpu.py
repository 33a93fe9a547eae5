"""The signed distance of meshes at scales far from 1, on either side of the line from which they are
scaled: the distances are those at scale 1 times the scale, bit for bit, and the tree leaves as much
out as it does there."""
import time

import numpy as np
import pytest
import torch

from conftest import prepared_mesh

pytestmark = pytest.mark.gpu


def best(fn):
    fn()
    times = []
    for _ in range(5):
        t = time.perf_counter()
        fn()
        times.append(time.perf_counter() - t)
    return min(times)


@pytest.fixture(scope="module")
def scene():
    V, F, o, w = prepared_mesh("knot", rings=1000, segs=50, seed=0)
    P = o + np.random.default_rng(0).uniform(0, 1, (50000, 3)) * w
    return V, np.ascontiguousarray(F, np.int32), P


@pytest.mark.parametrize("exponent", [-120, -80, -33, -32, 31, 32, 80, 120])
def test_distance_at_a_scale(ctx, scene, exponent):
    def run(scale):
        V, F, P = (torch.from_numpy(a).cuda() for a in (scene[0] * scale, scene[1], scene[2] * scale))
        out = torch.empty(len(P), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        t = best(lambda: ctx.signed_distance(P, V, F, out=out))
        return t, out
    scale = 2.0 ** exponent
    (t1, d1), (ts, ds) = run(1.0), run(scale)
    assert torch.equal(ds, d1 * scale)
    assert ts < 3 * t1  # 75 times where nothing is left out
