"""The triangular solves of one to four columns without thread-block clusters, as
they run where none of 16 CTAs fit: sizes around the 64-row blocks and the 16
blocks of a cluster, both triangles and directions, against FP64 substitution and
against the clustered launch."""
import ctypes

import numpy as np
import pytest
import torch

import remifa_b200 as rb
from remifa_b200 import _lib

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def solve_alone(lu, x, upper, trans):
    n, k = x.shape
    scratch = torch.empty(256 + (8 * n * k + 255) // 256 * 256, dtype=torch.uint8, device="cuda")
    st = _lib.lib().lu_selftest_solve_alone_c(
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), n, k, _p(lu), rb.ld(lu), _p(x),
        x.stride(1) if k > 1 else n, int(upper), int(trans), _p(scratch), scratch.numel())
    assert st == _lib.SUCCESS


@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("nrhs", [1, 2, 3])
@pytest.mark.parametrize("n,pad", [(1, 0), (64, 0), (65, 1), (1000, 0), (1090, 3)])
def test_alone(built, n, pad, nrhs, trans):
    rng = np.random.default_rng(n + nrhs)
    f = rng.uniform(-1.0, 1.0, (n, n)) / n
    f[np.diag_indices(n)] = rng.uniform(1.0, 2.0, n)
    f = f.astype(np.float32)
    lu = rb.colmajor_empty(n, n, n + pad, torch.float32)
    lu.copy_(torch.from_numpy(f))
    b = rng.standard_normal((n, nrhs))
    w = f.astype(np.float64)
    low, up = np.tril(w, -1) + np.eye(n), np.triu(w)
    for upper, t in ((False, low), (True, up)):
        x = torch.empty((nrhs, n), dtype=torch.float64, device="cuda").t()
        x.copy_(torch.from_numpy(b))
        solve_alone(lu, x, upper, trans)
        torch.cuda.synchronize()
        want = np.linalg.solve(t.T if trans else t, b)
        # cond <= 2 e^2 here; n u64 per substitution
        assert np.abs(x.cpu().numpy() - want).max() <= 64 * n * 2.0 ** -53 * np.abs(want).max()
    # both triangles in turn: what the clustered launches give, bit for bit
    x = torch.empty((nrhs, n), dtype=torch.float64, device="cuda").t()
    x.copy_(torch.from_numpy(b))
    y = torch.empty_like(x)
    y.copy_(x)
    solve_alone(lu, x, trans, trans)
    solve_alone(lu, x, not trans, trans)
    rb.lu_solve(lu, y, trans=trans)
    assert torch.equal(x, y)


def test_arguments(built):
    f = _lib.lib().lu_selftest_solve_alone_c
    q = ctypes.c_void_p(256)
    for args in ((None, 0, 1, q, 8, q, 8, 0, 0, q, 1024), (None, 8, 5, q, 8, q, 8, 0, 0, q, 1024),
                 (None, 8, 1, q, 7, q, 8, 0, 0, q, 1024), (None, 8, 1, q, 8, q, 8, 2, 0, q, 1024),
                 (None, 8, 1, q, 8, None, 8, 0, 0, q, 1024)):
        assert f(*args) == _lib.ERR_INVALID_ARG
    assert f(None, 8, 1, q, 8, q, 8, 0, 0, q, 64) == _lib.ERR_WORKSPACE
