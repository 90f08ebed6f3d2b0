"""A call whose kernel cannot be launched returns its error and leaves nothing
behind: the next launches, the library's and the program's, succeed."""
import pytest
import torch

import remifa_b200 as rb

pytestmark = pytest.mark.gpu


def test_refused_launch_leaves_no_error(built):
    k = 65536 * 64 + 8  # the operand copy's grid has a 64-value block per y: too many
    a = torch.zeros((k, 1), dtype=torch.float16, device="cuda").t()
    b = torch.zeros((1, k), dtype=torch.float16, device="cuda").t()
    c = torch.ones((1, 1), dtype=torch.float32, device="cuda")
    with pytest.raises(RuntimeError):
        rb.gemmex(rb.TC32, -1.0, a, b, 1.0, c)
    assert float((c + 1.0).item()) == 2.0
    out = rb.colmajor_empty(64, 64, 64, torch.float16)
    src = rb.colmajor(torch.eye(64, device="cuda"))
    rb.convert(src, out)
    rb.lu_solve(src, torch.ones(64, dtype=torch.float64, device="cuda"))
    torch.cuda.synchronize()
    assert torch.equal(out.float(), src)
