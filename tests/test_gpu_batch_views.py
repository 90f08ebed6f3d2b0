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


@pytest.mark.parametrize("view", ["matrices", "right_hand_sides"])
def test_shared_arrays_outlive_their_layout_on_another_stream(built, view):
    """A layout dropped while another stream still reads its device arrays: the
    arrays' memory is not handed out to its own stream meanwhile."""
    sizes = np.full(1500, 4, np.int32)
    lay = MatrixBatch(sizes)
    mem = [t.untyped_storage() for t in (lay.d_lda, lay._d_off)]
    used = {m.data_ptr(): m.nbytes() for m in mem}
    mem.clear()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        data = torch.zeros(int(lay.offsets[-1]), device="cuda")
        x = torch.zeros(int(sizes.sum()), dtype=torch.float64, device="cuda")
        torch.cuda._sleep(100_000_000)
        got = lay._over(data) if view == "matrices" else RhsBatch._over(lay, 1, x)
    shared = [lay._d_off.untyped_storage().data_ptr()]
    if view == "matrices":
        shared.append(lay.d_lda.untyped_storage().data_ptr())
    del got, lay
    new = [torch.empty(n, dtype=torch.uint8, device="cuda") for n in used.values()
           for _ in range(8)]
    assert not side.query()
    assert not {t.data_ptr() for t in new} & set(shared)
    side.synchronize()
