"""The blocked batched solve at the edges of its 32-unknown blocks: every
right-hand-side group width (1, 2, 4 and a ragged last group), dense and
padded leading dimensions, both directions, against FP64 substitution with the
same factors; a zero pivot reaches only the unknowns that depend on it."""
import numpy as np
import pytest
import torch

import remifa_b200 as rb
from remifa_b200.batch import BatchPlan, MatrixBatch, RhsBatch

pytestmark = pytest.mark.gpu

SIZES = np.array([1, 2, 31, 32, 33, 63, 64, 65, 95, 97, 128, 130, 160, 191, 224, 257, 385, 512],
                 np.int32)


def packed_factors(sizes, align, seed):
    """Packed L\\U with |L| <= 1/n off the diagonal and a dominant U."""
    rng = np.random.default_rng(seed)
    mats = MatrixBatch(sizes, align=align)
    host = []
    for i, n in enumerate(sizes):
        f = rng.uniform(-1.0, 1.0, (n, n)) / n
        f[np.diag_indices(n)] = rng.uniform(1.0, 2.0, n)
        f = f.astype(np.float32)
        mats.matrix(i).copy_(torch.from_numpy(f))
        host.append(f.astype(np.float64))
    return mats, host


@pytest.mark.parametrize("align", [1, 4])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 5])
@pytest.mark.parametrize("trans", [False, True])
def test_block_edges(built, trans, nrhs, align):
    mats, host = packed_factors(SIZES, align, 10 * nrhs + align)
    plan = BatchPlan(SIZES, outer=rb.FP32)
    x = RhsBatch(SIZES, nrhs)
    x.data.copy_(torch.from_numpy(np.random.default_rng(1).standard_normal(x.data.numel())))
    b = x.data.clone()
    plan.solve(mats, x, trans=trans)
    torch.cuda.synchronize()
    for i, f in enumerate(host):
        n = f.shape[0]
        L, U = np.tril(f, -1) + np.eye(n), np.triu(f)
        m = (L @ U).T if trans else L @ U
        want = np.linalg.solve(m, RhsBatch(SIZES, nrhs, data=b).block(i).cpu().numpy())
        got = x.block(i).cpu().numpy()
        # cond(L) cond(U) <= e^2 * 2 e^2 here; n u64 per substitution
        assert np.abs(got - want).max() <= 512 * n * 2.0 ** -53 * np.abs(want).max(), n


def test_zero_pivot_stays_local(built):
    sizes = np.array([100], np.int32)
    mats, host = packed_factors(sizes, 4, 3)
    m = mats.matrix(0)
    m[57, 57] = 0.0
    plan = BatchPlan(sizes, outer=rb.FP32)
    x = RhsBatch(sizes, 1)
    x.data.fill_(1.0)
    plan.solve(mats, x)
    torch.cuda.synchronize()
    got = x.data.cpu().numpy()
    f = host[0]
    y = np.linalg.solve(np.tril(f, -1) + np.eye(100), np.ones(100))
    want = np.linalg.solve(np.triu(f)[58:, 58:], y[58:])
    assert not np.isfinite(got[:58]).any()
    assert np.abs(got[58:] - want).max() <= 1e-12 * np.abs(want).max()
