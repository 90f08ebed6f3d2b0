"""The FP64 residual of more than 32 right-hand sides on both sides of the size
where the rows per CTA change, at ragged sizes.  max_iter = 0 reports the backward
error of X = (LU)^-1 B, formed again in FP64 by matrix products."""
import pytest
import torch

import remifa_b200 as rb
from remifa_b200.autograd import refine_ex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("n,nrhs", [(4735, 33), (4737, 64), (4801, 65)])
def test_backward_error_of_first_solve(built, n, nrhs, trans):
    a = rb.gen_matrix(n, seed=n, kind=1, alpha=1.5, lda=n + 3)
    lu = rb.colmajor(a)
    rb.lu_nopiv_rl(lu, outer=rb.TC32)
    lu.mul_(1.03)   # a residual far above rounding
    g = torch.Generator(device="cuda").manual_seed(nrhs)
    b = torch.randn((nrhs, n), generator=g, device="cuda", dtype=torch.float64).t()
    x = torch.zeros((nrhs, n), device="cuda", dtype=torch.float64).t()
    _, be = refine_ex(a, lu, b, x, trans=trans, max_iter=0)
    m = a.double().t() if trans else a.double()
    r = (b - m @ x).abs().amax(0)
    den = m.abs().sum(1).amax() * x.abs().amax(0) + b.abs().amax(0)
    want = float((r / den).max())
    # each residual entry is exact to n u64 of |A||x| + |b|
    assert abs(be - want) <= 2 * n * 2.0 ** -53 + 1e-12 * want, (be, want)
