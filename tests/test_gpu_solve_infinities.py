"""An infinite factor entry in the last, partial block of columns: its row of the
solution is infinite and the rows that do not depend on it stay what
substitution gives, in the triangular solves of few and of many right-hand sides
and in the batched solve."""
import numpy as np
import pytest
import torch

import remifa_b200 as rb
from remifa_b200.batch import BatchPlan, MatrixBatch, RhsBatch

pytestmark = pytest.mark.gpu


def factors(n, trans, seed):
    """f with one infinite entry, in U's first row / last column (transposed: L's
    last row / first column); the same f with a zero there."""
    rng = np.random.default_rng(seed)
    f = rng.uniform(-1.0, 1.0, (n, n)) / n
    f[np.diag_indices(n)] = rng.uniform(1.0, 2.0, n)
    at = (n - 1, 0) if trans else (0, n - 1)
    f[at] = 0.0
    f = f.astype(np.float32)
    g = f.copy()
    g[at] = np.inf
    return g, f.astype(np.float64)


def check(got, f, b, trans, alone):
    """Row 0 comes last in both directions; rows alone .. do not see its block."""
    n = f.shape[0]
    m = (np.tril(f, -1) + np.eye(n)) @ np.triu(f)
    want = np.linalg.solve(m.T if trans else m, b)
    assert np.isinf(got[0]).all()
    assert (np.sign(got[0]) == -np.sign(want[n - 1])).all()
    assert np.abs(got[alone:] - want[alone:]).max() <= 512 * n * 2.0 ** -53 * np.abs(want).max()


@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("nrhs", [1, 2, 8])
@pytest.mark.parametrize("n,pad", [(130, 0), (187, 1)])
def test_lu_solve(built, n, pad, nrhs, trans):
    g, f = factors(n, trans, n)
    lu = rb.colmajor_empty(n, n, n + pad, torch.float32)
    lu.copy_(torch.from_numpy(g))
    b = np.random.default_rng(nrhs).standard_normal((n, nrhs))
    x = torch.empty((nrhs, n), dtype=torch.float64, device="cuda").t()
    x.copy_(torch.from_numpy(b))
    rb.lu_solve(lu, x, trans=trans)
    torch.cuda.synchronize()
    check(x.cpu().numpy(), f, b, trans, 64)


@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("nrhs", [1, 2, 3])
@pytest.mark.parametrize("n", [70, 100, 127])
def test_batched_solve(built, n, nrhs, trans):
    g, f = factors(n, trans, n)
    sizes = np.array([n], np.int32)
    lu = MatrixBatch(sizes)
    lu.matrix(0).copy_(torch.from_numpy(g))
    x = RhsBatch(sizes, nrhs)
    b = np.random.default_rng(nrhs).standard_normal((n, nrhs))
    x.block(0).copy_(torch.from_numpy(b))
    BatchPlan(sizes, outer=rb.FP32).solve(lu, x, trans=trans)
    torch.cuda.synchronize()
    check(x.block(0).cpu().numpy(), f, b, trans, 1)
