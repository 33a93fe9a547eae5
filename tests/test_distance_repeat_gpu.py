"""The signed distance is the same from call to call, signs included, also in the opening of a bowl of few
triangles, where the winding number is 1/2 and its rounding decides."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rings,segs", [(1, 16), (2, 5), (2, 16)])
def test_signs_in_an_opening_do_not_change(ctx, rings, segs):
    theta = np.linspace(0, np.pi / 2, rings + 1)[1:, None]
    phi = np.linspace(0, 2 * np.pi, segs, endpoint=False)[None, :]
    ring = np.stack([np.sin(theta) * np.cos(phi), np.sin(theta) * np.sin(phi), np.cos(theta) + 0 * phi], -1)
    V = np.concatenate([[[0.0, 0.0, 1.0]], ring.reshape(-1, 3)])
    V[-segs:, 2] = 0.0

    def at(i, j):
        return 1 + i * segs + j % segs

    F = [[0, at(0, j), at(0, j + 1)] for j in range(segs)]
    for i in range(rings - 1):
        for j in range(segs):
            F += [[at(i, j), at(i + 1, j), at(i + 1, j + 1)], [at(i, j), at(i + 1, j + 1), at(i, j + 1)]]
    P = np.random.default_rng(0).uniform(-3.0, 3.0, (400000, 3))
    P[:, 2] = 0.0
    V, F, P = (torch.from_numpy(a).cuda() for a in (V, np.array(F, np.int32), P))
    first, again = (torch.empty(len(P), dtype=torch.float64, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    ctx.signed_distance(P, V, F, out=first)
    for _ in range(10):
        ctx.signed_distance(P, V, F, out=again)
        assert torch.equal(first, again)
