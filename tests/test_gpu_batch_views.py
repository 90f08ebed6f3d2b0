"""The device-side pointer arrays batched_lu_solve forms for its buffers equal
those of the public constructors; its checks stay theirs."""
import copy
import pickle

import numpy as np
import pytest
import torch

import remifa_b200 as rb
from remifa_b200.batch import BatchPlan, MatrixBatch, RhsBatch, batched_lu_solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("align", [1, 4])
@pytest.mark.parametrize("sizes", [[1], [5, 1, 512, 33], list(range(1, 130))])
def test_pointers(built, sizes, align):
    sizes = np.array(sizes, np.int32)
    lay = MatrixBatch(sizes, align=align)
    data = torch.zeros(int(lay.offsets[-1]) + 3, device="cuda")
    got, want = lay._over(data), lay.like(data)
    assert got.ptrs.tolist() == want.ptrs.tolist() and got.data is data
    assert got.d_n.tolist() == want.d_n.tolist() and got.d_lda.tolist() == want.d_lda.tolist()
    for k in (1, 3):
        x = torch.zeros(int(sizes.sum()) * k, dtype=torch.float64, device="cuda")
        assert RhsBatch._over(lay, k, x).ptrs.tolist() == RhsBatch(sizes, k, data=x).ptrs.tolist()
        with pytest.raises(ValueError):
            RhsBatch._over(lay, k, x[:-1])
    with pytest.raises(ValueError):
        lay._over(data.double())
    with pytest.raises(ValueError):
        lay._over(data[:int(lay.offsets[-1]) - 1])


def test_shared_arrays_outlive_their_layout_on_another_stream(built):
    """A layout dropped while another stream still has to read its device arrays:
    their memory is not handed out to its own stream meanwhile."""
    sizes = np.full(1500, 4, np.int32)
    lay = MatrixBatch(sizes).generate(seed=1)
    plan = BatchPlan(sizes, outer=rb.FP32)
    shared = {t.untyped_storage().data_ptr(): t.untyped_storage().nbytes()
              for t in (lay.d_lda, lay._d_off)}
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        a = lay.data.clone().requires_grad_(True)
        b = torch.ones(int(sizes.sum()), dtype=torch.float64, device="cuda", requires_grad=True)
        # once before, so that nothing below loads a kernel or takes new memory
        warm = batched_lu_solve(a, b, MatrixBatch(sizes), plan)
        torch.autograd.grad(warm, (a, b), torch.ones_like(warm))
        del warm
        x = batched_lu_solve(a, b, lay, plan)
        torch.cuda._sleep(200_000_000)
        grads = torch.autograd.grad(x, (a, b), torch.ones_like(x))
    del x, lay
    new = [torch.empty(n, dtype=torch.uint8, device="cuda") for n in shared.values()
           for _ in range(8)]
    assert not side.query()
    assert not {t.data_ptr() for t in new} & set(shared)
    side.synchronize()
    assert all(bool(torch.isfinite(g).all()) for g in grads)


def test_copies_and_views_know_their_stream(built):
    """A view shares its layout's arrays and so their stream; a copy's arrays are
    new, on whatever stream it is made, and are recorded wherever they are used."""
    lay = MatrixBatch(np.array([3, 5], np.int32))
    assert lay._home == torch.cuda.current_stream().cuda_stream
    assert lay._over(torch.zeros_like(lay.data))._home == lay._home
    for other in (copy.copy(lay), copy.deepcopy(lay), pickle.loads(pickle.dumps(lay))):
        assert other._home is None
        assert other.lda.tolist() == lay.lda.tolist()
