"""One batched solve over several launches: small matrices in great number as a
warp per column, the others in size classes of their own.  Every column against
FP64 substitution with the same factors, both directions, with and without
refinement; chains of calls and a graph replay give what single calls give."""
import numpy as np
import pytest
import torch

import remifa_b200 as rb
from remifa_b200.batch import BatchPlan, MatrixBatch, RhsBatch

pytestmark = pytest.mark.gpu

# sizes (count, n): all small; small ones under a few large; every class at once,
# with a gap between them; a large class too small for a launch of its own
BATCHES = {
    "small": [(3000, 1), (3000, 7), (2000, 32), (1000, 33)],
    "small_and_one": [(1, 512), (9000, 20)],
    "classes": [(20, 512), (700, 300), (1000, 150), (12000, 9), (3000, 31)],
    "gap": [(3, 500), (900, 100), (4000, 16)],
    "few": [(2, 400), (5, 200), (7, 30)],
}


def make(parts, seed):
    rng = np.random.default_rng(seed)
    sizes = rng.permutation(np.concatenate([np.full(c, n) for c, n in parts])).astype(np.int32)
    mats = MatrixBatch(sizes, align=4)
    # one factor pair per size, |L| <= 1/n, a dominant U; A = L U rounded
    idx, host = {}, {}
    for n in np.unique(sizes):
        f = rng.uniform(-1.0, 1.0, (n, n)) / n
        f[np.diag_indices(n)] = rng.uniform(1.0, 2.0, n)
        host[int(n)] = f.astype(np.float32)
    lu = np.zeros(mats.data.numel(), np.float32)
    a = np.zeros_like(lu)
    for n, f in host.items():
        w = f.astype(np.float64)
        full = ((np.tril(w, -1) + np.eye(n)) @ np.triu(w)).astype(np.float32)
        ld = int(mats.lda[np.nonzero(sizes == n)[0][0]])
        at = (np.arange(n)[:, None] + ld * np.arange(n)[None, :])
        where = mats.offsets[:-1][sizes == n]
        lu[where[:, None, None] + at] = f
        a[where[:, None, None] + at] = full
        idx[n] = np.nonzero(sizes == n)[0]
    mats.data.copy_(torch.from_numpy(lu))
    return sizes, mats, mats.like(torch.from_numpy(a).cuda()), host, idx


@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("nrhs", [1, 2, 5])
@pytest.mark.parametrize("batch", list(BATCHES))
def test_every_column(built, batch, nrhs, trans):
    sizes, lu, a, host, idx = make(BATCHES[batch], nrhs)
    plan = BatchPlan(sizes, outer=rb.FP32)
    b = RhsBatch(sizes, nrhs)
    b.data.copy_(torch.from_numpy(np.random.default_rng(2).standard_normal(b.data.numel())))
    for iters in (0, 2):
        x = b.like(b.data.clone())
        plan.solve(lu, x, a=a if iters else None, trans=trans, refine_iters=iters)
        torch.cuda.synchronize()
        got, rhs = x.data.cpu().numpy(), b.data.cpu().numpy()
        for n, f in host.items():
            w = f.astype(np.float64)
            m = (np.tril(w, -1) + np.eye(n)) @ np.triu(w)
            if iters:
                m = m.astype(np.float32).astype(np.float64)
            at = b.offsets[:-1][idx[n]][:, None] + np.arange(n * nrhs)
            bb = rhs[at].reshape(-1, nrhs, n)
            xx = got[at].reshape(-1, nrhs, n)
            want = np.linalg.solve(m.T if trans else m, bb.reshape(-1, n).T).T.reshape(xx.shape)
            scale = np.abs(want).max(axis=2, keepdims=True)
            # cond(L) cond(U) <= e^2 * 2 e^2 here; n u64 per substitution
            assert (np.abs(xx - want) <= 512 * n * 2.0 ** -53 * scale).all(), n


def test_chains_and_replay(built):
    sizes, lu, a, _, _ = make(BATCHES["classes"], 3)
    plan = BatchPlan(sizes, outer=rb.FP32)
    x = RhsBatch(sizes, 1)
    b = torch.randn(x.data.numel(), dtype=torch.float64, device="cuda")
    c = torch.randn_like(b)

    def chain(v, wait=lambda: None):
        x.data.copy_(v)
        wait()
        plan.solve(lu, x, a=a, refine_iters=1)
        wait()
        x.data.mul_(2.0)
        wait()
        plan.solve(lu, x, trans=True)
        wait()

    chain(b, torch.cuda.synchronize)
    want_b = x.data.clone()
    chain(c, torch.cuda.synchronize)
    want_c = x.data.clone()
    for v, want in ((b, want_b), (c, want_c), (b, want_b)):
        chain(v)
        assert torch.equal(x.data, want)
    v = b.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(v)
    for new, want in ((c, want_c), (b, want_b)):
        v.copy_(new)
        graph.replay()
        assert torch.equal(x.data, want)
