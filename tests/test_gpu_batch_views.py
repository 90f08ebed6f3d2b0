"""The device-side pointer arrays batched_lu_solve forms for its buffers equal
those of the public constructors; its checks stay theirs."""
import numpy as np
import pytest
import torch

from remifa_b200.batch import MatrixBatch, RhsBatch

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
