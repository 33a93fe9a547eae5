"""The fused gradient at the edges of its tiles and its grid: half a tile, one, a remainder, a CTA's first
and second tile, more tiles than CTAs, features at an address that allows no 16-byte loads. The same
bars as the network's other gradient test: each parameter block to 2e-2 relative (Frobenius) of the
oracle's, which rounds to BF16 where the kernel does."""
import ctypes

import numpy as np
import pytest

from oracle import mlp as ref

pytestmark = pytest.mark.gpu


def _close(g, g_ref):
    k = 0
    for name, shape in ref.SHAPES:
        m = int(np.prod(shape))
        a, b = g[k:k + m], g_ref[k:k + m]
        assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b) + 1e-7, (name, np.linalg.norm(a - b) / np.linalg.norm(b))
        k += m


@pytest.mark.parametrize("n", [64, 128, 192, 256, 148 * 128, 148 * 128 + 64, 149 * 128, 40000])
def test_gradient_of_batches(ctx, n):
    from its_b200.api import ShareNet
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, ref.N_IN)).astype(np.float32)
    y = (np.sin(X[:, 0]) + 0.5 * X[:, 1] * X[:, 2]).astype(np.float32)
    P = ref.init_params(n)
    net = ShareNet(ctx, batch=(n + 127) // 128 * 128, params=P)
    g, loss = net.gradient(X, y)
    g_ref, loss_ref = ref.gradient(P, X, y)
    assert abs(loss - loss_ref) <= 1e-3 * loss_ref
    _close(g, g_ref)
    again, _ = net.gradient(X, y)
    assert np.array_equal(g, again)
    net.close()


def test_gradient_of_features_at_an_odd_address(ctx):
    import torch
    from its_b200 import lib
    from its_b200.api import ShareNet
    n = 320
    rng = np.random.default_rng(5)
    X = rng.standard_normal((n, ref.N_IN)).astype(np.float32)
    y = X[:, 0].copy()
    net = ShareNet(ctx, batch=384, params=ref.init_params(1))
    want, _ = net.gradient(X, y)
    buf = torch.zeros(n * ref.N_IN + 1, dtype=torch.float32, device="cuda")
    buf[1:] = torch.from_numpy(X).cuda().reshape(-1)
    yd, g, loss = torch.from_numpy(y).cuda(), np.zeros(net.num_params, np.float32), ctypes.c_float(0)
    torch.cuda.synchronize()
    ctx.check(lib().its_mlp_gradient(net.h, ctypes.c_void_p(buf.data_ptr() + 4), ctypes.c_void_p(yd.data_ptr()), n,
                                     g.ctypes.data_as(ctypes.c_void_p), ctypes.byref(loss)), "its_mlp_gradient")
    assert np.array_equal(g, want)
    net.close()
