"""The FP64 residual of several right-hand sides at the edges of its tiles: every
group width (8, 16, 32, 64 columns and one past each), sizes around multiples
of its 16 rows and 32-value stages, both directions, aligned and odd leading
dimensions.  max_iter = 0 leaves X = (LU)^-1 B and reports the largest backward
error of its residual, which is formed again in FP64 on the host."""
import numpy as np
import pytest
import torch

import remifa_b200 as rb
from remifa_b200.autograd import adjoint, refine_ex

pytestmark = pytest.mark.gpu


def colmajor64(x):
    t = torch.empty((x.shape[1], x.shape[0]), dtype=torch.float64, device="cuda").t()
    t.copy_(torch.from_numpy(np.ascontiguousarray(x)))
    return t


@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("n,pad", [(15, 0), (257, 1), (512, 0), (700, 4)])
@pytest.mark.parametrize("nrhs", [2, 8, 9, 16, 17, 32, 33, 64, 65])
def test_backward_error_of_first_solve(built, nrhs, n, pad, trans):
    a = rb.gen_matrix(n, seed=n + nrhs, kind=1, alpha=1.5, lda=n + pad)
    lu = rb.colmajor(a)
    rb.lu_nopiv_rl(lu, outer=rb.TC32, nb=128)
    # factors off by a few percent: a residual far above rounding
    lu.mul_(1.03)
    rng = np.random.default_rng(n * nrhs)
    b = rng.standard_normal((n, nrhs))
    x = colmajor64(np.zeros((n, nrhs)))
    it, be = refine_ex(a, lu, colmajor64(b), x, trans=trans, max_iter=0)
    A = a.cpu().numpy().astype(np.float64)
    A = A.T if trans else A
    X = x.cpu().numpy()
    r = b - A @ X
    den = np.abs(A).sum(axis=1).max() * np.abs(X).max(axis=0) + np.abs(b).max(axis=0)
    want = (np.abs(r).max(axis=0) / den).max()
    assert it == 0
    # each residual entry is exact to n u64 of |A||x| + |b|
    assert abs(be - want) <= 2 * n * 2.0 ** -53 + 1e-12 * want, (be, want)


@pytest.mark.parametrize("n", [1, 63, 65, 300])
@pytest.mark.parametrize("nrhs", [1, 3, 4, 31, 33, 64, 70])
def test_outer_product(built, n, nrhs):
    a = rb.gen_matrix(max(n, 2), seed=3, kind=1, alpha=2.0)[:n, :n]
    a = rb.colmajor(a)
    if n == 1:
        a.fill_(2.0)
    lu = rb.colmajor(a)
    rb.lu_nopiv_rl(lu, outer=rb.FP32)
    rng = np.random.default_rng(nrhs)
    x, g = rng.standard_normal((n, nrhs)), rng.standard_normal((n, nrhs))
    gd = colmajor64(g)
    da = rb.colmajor_empty(n, n, n + 1, torch.float32)
    adjoint(lu, colmajor64(x), gd, da=da)
    db = gd.cpu().numpy()
    want = -db @ x.T
    bound = (nrhs * 2.0 ** -53 * (np.abs(db) @ np.abs(x).T) + 2.0 ** -24 * np.abs(want)) * 1.01
    assert (np.abs(da.cpu().numpy() - want) <= bound + 1e-300).all()
