"""Marching cubes over fields where its tiles can go wrong: rows shorter and longer than a thread's run
of voxels, remainders, every voxel crossed, nothing crossed, values that are not numbers, and case
bytes at an odd address. Cases and soup against the oracle's, bit for bit."""
import ctypes

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

O, W = np.array([0.1, -0.2, 0.3]), np.array([1.0, 1.1, 0.9])


def _field(kind, R):
    rng = np.random.default_rng(R)
    M = R + 1
    if kind == "noise":
        return rng.standard_normal(M ** 3)
    if kind == "flat":
        return np.full(M ** 3, 1.0)
    g = np.linspace(-1, 1, M)
    z, y, x = np.meshgrid(g, g, g, indexing="ij")
    f = (np.sqrt(x * x + y * y + z * z) - 0.7).ravel()
    if kind == "nan":
        f[rng.integers(0, M ** 3, max(1, M ** 3 // 50))] = np.nan
    return f


@pytest.mark.parametrize("R", [1, 2, 3, 4, 5, 8, 15, 16, 17, 31, 32, 33, 47, 64, 65])
@pytest.mark.parametrize("kind", ["noise", "flat", "ball", "nan"])
def test_cases_and_soup(ctx, R, kind):
    f = _field(kind, R)
    cube, tri, n = ctx.marching_cubes(f, R, O, W, 0.05)
    want_cube, want_tri, want_n = oracle.marching_cubes(f, R, O, W, 0.05)
    assert n == want_n and np.array_equal(cube, want_cube)
    assert np.array_equal(tri, np.asarray(want_tri).reshape(-1, 3)[:n], equal_nan=True)


@pytest.mark.parametrize("R", [16, 33, 64])
@pytest.mark.parametrize("shift", [1, 4, 8])
def test_case_bytes_anywhere_and_a_short_soup(ctx, R, shift):
    import torch
    from its_b200 import lib
    f = _field("noise", R)
    want_cube, want_tri, want_n = oracle.marching_cubes(f, R, O, W, 0.05)
    want_tri = np.asarray(want_tri).reshape(-1, 3)
    fd = torch.from_numpy(f).cuda()
    buf = torch.zeros(R ** 3 + 2 * shift, dtype=torch.uint8, device="cuda")
    cap = want_n // 2 + 1
    tri = torch.zeros((want_n, 3), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    n = ctypes.c_int64(0)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    ctx.check(lib().its_marching_cubes(ctx.h, p(fd), R, O.ctypes.data_as(ctypes.c_void_p), W.ctypes.data_as(ctypes.c_void_p),
                                       0.05, ctypes.c_void_p(buf.data_ptr() + shift), p(tri), cap, ctypes.byref(n)), "mc")
    got = buf.cpu().numpy()
    assert n.value == want_n and np.array_equal(got[shift:shift + R ** 3], want_cube)
    assert not got[:shift].any() and not got[shift + R ** 3:].any()
    t = tri.cpu().numpy()
    assert np.array_equal(t[:cap], want_tri[:cap]) and not t[cap:].any()
