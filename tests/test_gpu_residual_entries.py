"""Every entry of the FP64 residual of several right-hand sides: with factors a few
percent off, one round of refinement gives X0 + (LU)^-1 (B - op(A) X0), whose
second term moves every entry far more than rounding does.  All group widths (8, 16,
32, 64 columns, with 32 and with 64 rows per CTA), one past each, sizes around the
16-row tiles, both directions."""
import pytest
import torch

import remifa_b200 as rb
from remifa_b200.autograd import refine_ex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("n,pad,nrhs", [(n, p, k) for n, p in ((15, 1), (257, 0), (700, 4))
                                        for k in (2, 8, 9, 17, 33, 65)]
                         + [(4737, 1, 33), (4801, 0, 65)])
def test_one_round(built, n, pad, nrhs, trans):
    a = rb.gen_matrix(n, seed=n + nrhs, kind=1, alpha=1.5, lda=n + pad)
    lu = rb.colmajor(a)
    rb.lu_nopiv_rl(lu, outer=rb.TC32, nb=128)
    lu.mul_(1.03)
    g = torch.Generator(device="cuda").manual_seed(n * nrhs)
    b = torch.randn((nrhs, n), generator=g, dtype=torch.float64, device="cuda").t()
    x = torch.empty((nrhs, n), dtype=torch.float64, device="cuda").t()
    it, _ = refine_ex(a, lu, b, x, trans=trans, max_iter=1, tol=0.0)
    assert it == 1
    f, A = lu.double(), a.double()
    tri = torch.linalg.solve_triangular

    def solve(r):
        if not trans:
            return tri(f, tri(f, r, upper=False, unitriangular=True), upper=True)
        return tri(f.t(), tri(f.t(), r, upper=False), upper=True, unitriangular=True)

    x0 = solve(b)
    want = x0 + solve(b - (A.t() if trans else A) @ x0)
    # dominance 1.5: both systems well conditioned; n u64 per sum, four in turn
    assert bool(((x - want).abs() <= 64 * n * 2.0 ** -53 * want.abs().amax(0)).all())
    # the round moved the entries: a residual entry left out would show
    assert float(((want - x0).abs() > 1e-4 * want.abs().amax(0)).double().mean()) > 0.9
