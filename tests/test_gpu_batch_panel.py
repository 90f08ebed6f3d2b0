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
