"""Dependent launches: chains of calls on one stream, on a second stream after an
event, and captured in a graph and replayed on new values, give what the same
calls give one by one with a synchronisation after each."""
import pytest
import torch

import remifa_b200 as rb

pytestmark = pytest.mark.gpu


def _inputs(n, nrhs, seed):
    a = rb.colmajor_empty(n, n, n, torch.float32)
    g = torch.Generator(device="cuda").manual_seed(seed)
    a.copy_(torch.rand((n, n), generator=g, device="cuda") - 0.5)
    a.diagonal().add_(float(n))
    b = torch.rand((nrhs, n), generator=g, device="cuda", dtype=torch.float64).t()
    return a, b


@pytest.mark.parametrize("nrhs", [1, 2, 9])
@pytest.mark.parametrize("n,outer", [(130, "FP32"), (700, "TC32"), (1300, "TC32_E4M3")])
def test_chains_match_single_calls(built, n, outer, nrhs):
    outer = getattr(rb.compute_type, outer)
    sync = torch.cuda.synchronize
    lu = rb.colmajor_empty(n, n, n, torch.float32)
    x = torch.empty((nrhs, n), device="cuda", dtype=torch.float64).t()
    info = torch.zeros(1, device="cuda", dtype=torch.int32)
    ws = torch.empty(rb.workspace_size(n, outer=outer), dtype=torch.uint8, device="cuda")

    def chain(a, b, wait=lambda: None):
        lu.copy_(a)
        x.copy_(b)
        wait()
        rb.lu_nopiv_rl(lu, outer=outer, workspace=ws, info=info)
        wait()
        rb.lu_solve(lu, x)
        wait()
        rb.lu_solve(lu, x, trans=True)
        wait()

    cases = [_inputs(n, nrhs, s) for s in (1, 2, 3)]
    want = []
    for a, b in cases:
        chain(a, b, sync)
        want.append((lu.clone(), x.clone()))
    for (a, b), (wl, wx) in zip(cases, want):          # one stream
        chain(a, b)
        assert torch.equal(lu, wl) and torch.equal(x, wx)
    side = torch.cuda.Stream()                         # another, after an event
    for (a, b), (wl, wx) in zip(cases, want):
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            chain(a, b)
        torch.cuda.current_stream().wait_stream(side)
        assert torch.equal(lu, wl) and torch.equal(x, wx)
    ga, gb = cases[0][0].clone(), cases[0][1].clone()  # captured and replayed
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(ga, gb)
    for _ in range(2):
        for (a, b), (wl, wx) in zip(cases, want):
            ga.copy_(a)
            gb.copy_(b)
            graph.replay()
            assert torch.equal(lu, wl) and torch.equal(x, wx)
