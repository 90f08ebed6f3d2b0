"""Block-column elimination of the batched LU where the largest matrix sets the
shared-memory leading dimension (partial tiles and row blocks reach into the
padding), and with more rows than threads."""
import numpy as np
import pytest
import torch

import oracle as O
import remifa_b200 as rb
from remifa_b200.batch import BUCKETS, BatchPlan, MatrixBatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", list(range(2, 20)) + [43, 45, 46, 67, 71, 263, 264, 265, 321, 325])
def test_largest_matrix_sets_the_padding(n):
    sizes = np.array([n, max(n - 1, 2), n], np.int32)
    for nb in (32, 64):
        mats = MatrixBatch(sizes).generate(seed=40)
        plan = BatchPlan(sizes, outer=rb.FP32,
                         tuning={"nb": [nb] * BUCKETS, "outer": [int(rb.FP32)] * BUCKETS})
        info = plan(mats)
        torch.cuda.synchronize()
        assert info.tolist() == [0, 0, 0]
        for i, m in enumerate(sizes):
            a = O.gen_matrix(int(m), seed=40 + i, kind=0, alpha=1.5)
            assert np.array_equal(mats.matrix(i).cpu().numpy(), O.lu_rl(a, nb=nb, outer_fmt=0))


@pytest.mark.parametrize("align", [1, 4])
@pytest.mark.parametrize("outer", ["FP32", "TC32"])
@pytest.mark.parametrize("nb,n", [(32, n) for n in (33, 36, 40, 41, 44, 48, 52, 60, 68)]
                         + [(64, n) for n in (65, 68, 72, 76, 80, 100, 136)])
def test_rows_below_the_last_tile(nb, n, outer, align):
    """Many copies of one matrix whose block columns have few rows below them:
    the block is stored (and copied for the fp16 update) right after its last
    tile is eliminated, so every copy has to come out the same."""
    outer = getattr(rb, outer)
    copies = 592
    sizes = np.full(copies, n, np.int32)
    mats = MatrixBatch(sizes, align=align)
    a = O.gen_matrix(n, seed=n, kind=0, alpha=1.5)
    first = mats.matrix(0)
    first.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    per = int(mats.offsets[1])
    blocks = mats.data[:copies * per].view(copies, per)
    blocks[1:] = blocks[0].clone()
    plan = BatchPlan(sizes, outer=outer,
                     tuning={"nb": [nb] * BUCKETS, "outer": [int(outer)] * BUCKETS})
    info = plan(mats)
    torch.cuda.synchronize()
    assert not bool(info.any())
    assert bool((blocks == blocks[0]).all())
    got = first.cpu().numpy()
    fp16 = outer == rb.TC32
    want = O.lu_rl(a, nb=nb, outer_fmt=O.FMT_FP16 if fp16 else 0)
    if fp16:
        # the first block column and row see no fp16 product
        assert np.array_equal(got[:, :nb], want[:, :nb])
        assert np.array_equal(got[:nb], want[:nb])
        assert np.abs(got - want).max() <= 64 * n * 2.0 ** -24 * np.abs(want).max()
    else:
        assert np.array_equal(got, want)
