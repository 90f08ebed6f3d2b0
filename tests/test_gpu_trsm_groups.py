"""Triangular solves of several right-hand sides around the edges of their
64-row blocks and 8-column groups, both directions, aligned and odd leading
dimensions of the factors and the right-hand sides, against FP64 substitution
with the same factors."""
import numpy as np
import pytest
import torch

import remifa_b200 as rb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 7, 8, 9, 20])
@pytest.mark.parametrize("n,pad", [(1, 0), (63, 1), (64, 0), (65, 3), (128, 0), (129, 7),
                                   (1000, 0), (1001, 1)])
def test_against_substitution(built, n, pad, nrhs, trans):
    rng = np.random.default_rng(100 * n + nrhs)
    f = rng.uniform(-1.0, 1.0, (n, n)) / n
    f[np.diag_indices(n)] = rng.uniform(1.0, 2.0, n)
    f = f.astype(np.float32)
    lu = rb.colmajor_empty(n, n, n + pad, torch.float32)
    lu.copy_(torch.from_numpy(f))
    b = rng.standard_normal((n, nrhs))
    buf = torch.full((nrhs, n + pad), 7.0, dtype=torch.float64, device="cuda")
    x = buf.t()[:n]
    x.copy_(torch.from_numpy(b))
    rb.lu_solve(lu, x, trans=trans)
    torch.cuda.synchronize()
    f = f.astype(np.float64)
    m = (np.tril(f, -1) + np.eye(n)) @ np.triu(f)
    want = np.linalg.solve(m.T if trans else m, b)
    # cond(L) cond(U) <= e^2 * 2 e^2 here; n u64 per substitution
    assert np.abs(x.cpu().numpy() - want).max() <= 512 * n * 2.0 ** -53 * np.abs(want).max()
    assert bool((buf[:, n:] == 7.0).all())


@pytest.mark.parametrize("nrhs", [1, 3])
def test_zero_pivot_stays_local(built, nrhs):
    n = 200
    rng = np.random.default_rng(5)
    f = rng.uniform(-1.0, 1.0, (n, n)) / n
    f[np.diag_indices(n)] = 1.5
    f[100, 100] = 0.0
    f = f.astype(np.float32)
    lu = rb.colmajor_empty(n, n, n, torch.float32)
    lu.copy_(torch.from_numpy(f))
    x = torch.ones(nrhs, n, dtype=torch.float64, device="cuda").t()
    rb.lu_solve(lu, x)
    torch.cuda.synchronize()
    got = x.cpu().numpy()
    f = f.astype(np.float64)
    y = np.linalg.solve(np.tril(f, -1) + np.eye(n), np.ones((n, nrhs)))
    # the block of rows 64 .. 127 holds the pivot: later blocks do not see it
    want = np.linalg.solve(np.triu(f)[128:, 128:], y[128:])
    assert not np.isfinite(got[:101]).any()
    assert np.abs(got[128:] - want).max() <= 1e-12 * np.abs(want).max()
