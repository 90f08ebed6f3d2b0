"""The panel kernel's item counts per CTA (32 in small launches, 64 in large
ones): FP32 factorizations, whose every element has a fixed operation order,
around the size where the first panel changes over, and around multiples of
both, with aligned and odd leading dimensions, against the oracle bit for bit."""
import numpy as np
import pytest
import torch

import oracle as O
import remifa_b200 as rb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["rl", "ll"])
@pytest.mark.parametrize("n,pad", [(159, 1), (192, 0), (257, 3), (2495, 1), (2496, 0), (2497, 0),
                                   (2561, 7)])
def test_item_counts_bit_exact(built, variant, n, pad):
    a = O.gen_matrix(n, seed=n, kind=1, alpha=1.5)
    nb = 128
    want = O.lu_rl(a, nb=nb) if variant == "rl" else O.lu_ll(a, nb=nb)
    d = rb.colmajor_empty(n, n, n + pad, torch.float32)
    d.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    f = rb.lu_nopiv_rl if variant == "rl" else rb.lu_nopiv_ll
    info = f(d, nb=nb, lookahead=False)
    torch.cuda.synchronize()
    assert int(info.item()) == 0
    np.testing.assert_array_equal(d.cpu().numpy(), want)
