"""Operand copies of the tensor-core update: fp16 B read in place or copied (by
alignment and overlap), A by 16-byte or single loads, and the scaled kinds'
one-launch copies at the edges of their 64-value and 128-row blocks."""
import numpy as np
import pytest
import torch

import oracle as O
import remifa_b200 as rb
from test_gpu_tc import rounded_operands, split_tiles

pytestmark = pytest.mark.gpu


def _view(x, ld, off):
    """x as a column-major view with leading dimension ld, off elements past a
    16-byte boundary."""
    m, n = x.shape
    store = torch.zeros(off + ld * n, dtype=x.dtype, device="cuda")
    v = store[off:].as_strided((m, n), (1, ld))
    v.copy_(x)
    return v


@pytest.mark.parametrize("M,N,K,pad,off", [
    (1, 1, 1, 0, 0), (64, 128, 64, 0, 0), (130, 257, 72, 0, 0), (130, 257, 72, 8, 1),
    (200, 130, 65, 7, 0), (128, 128, 63, 1, 8), (333, 77, 500, 4, 0), (333, 77, 500, 0, 4)])
@pytest.mark.parametrize("c_half", [False, True])
def test_fp16_operands_any_layout(M, N, K, pad, off, c_half):
    rng = np.random.default_rng(M + N + K)
    A = torch.from_numpy(rng.uniform(-1, 1, (M, K)).astype(np.float16)).cuda()
    B = torch.from_numpy(rng.uniform(-1, 1, (K, N)).astype(np.float16)).cuda()
    C = torch.from_numpy(rng.uniform(-1, 1, (M, N)).astype(np.float32)).cuda()
    if c_half:
        C = C.half()
    dA, dB = _view(A, M + pad, off), _view(B, K + pad, off)
    dC = _view(C, M, 0)
    rb.gemmex(rb.TC32, -1.0, dA, dB, 1.0, dC)
    want = C.double() - A.double() @ B.double()
    u = 2.0 ** -24
    bound = 2 * K * u * (A.double().abs() @ B.double().abs()) + 2 * u * C.double().abs()
    if c_half:
        bound = bound + 2.0 ** -11 * (want.abs() + bound) + 2.0 ** -25
    assert bool(((dC.double() - want).abs() <= bound + 1e-30).all())


def test_fp16_update_of_b_itself():
    """C lies over B: the update uses B as it was before the call."""
    rng = np.random.default_rng(7)
    n = 256
    A = torch.from_numpy(rng.uniform(-1, 1, (n, n)).astype(np.float16)).cuda()
    B = torch.from_numpy(rng.uniform(-1, 1, (n, n)).astype(np.float16)).cuda()
    dA, dB = _view(A, n, 0), _view(B, n, 0)
    dC = _view(B, n, 0)
    rb.gemmex(rb.TC32, -1.0, dA, dB, 1.0, dC)      # apart
    rb.gemmex(rb.TC32, -1.0, dA, dB, 1.0, dB)      # over B
    assert torch.equal(dB, dC)


@pytest.mark.parametrize("M,N,K,lda_pad,ldb_pad", [
    (1, 1, 1, 0, 0), (128, 128, 256, 0, 0), (129, 257, 257, 0, 3), (131, 126, 63, 1, 0),
    (260, 127, 65, 0, 1), (127, 300, 320, 5, 0), (64, 64, 530, 0, 0), (300, 140, 200, 4, 4)])
@pytest.mark.parametrize("kind", ["TC32_E4M3", "TC32_SPLIT"])
def test_scaled_copies(M, N, K, lda_pad, ldb_pad, kind):
    rng = np.random.default_rng(M * N + K)
    # tiles of different size: their scales differ
    A = (rng.uniform(-1, 1, (M, K)) * np.exp2(7.0 * (np.arange(M) // 128 - 1))[:, None])
    B = (rng.uniform(-1, 1, (K, N)) * np.exp2(-9.0 * (np.arange(N) // 128))[None, :])
    A, B = np.asfortranarray(A.astype(np.float32)), np.asfortranarray(B.astype(np.float32))
    dA = _view(torch.from_numpy(A).cuda(), M + lda_pad, 0)
    dB = _view(torch.from_numpy(B).cuda(), K + ldb_pad, 0)
    dC = torch.zeros((N, M), dtype=torch.float32, device="cuda").t()
    rb.gemmex(getattr(rb.compute_type, kind), 1.0, dA, dB, 1.0, dC)
    if kind == "TC32_SPLIT":
        (Ah, Al), (Bh, Bl) = split_tiles(A, True), split_tiles(B, False)
        terms = [(Ah, Bh), (Ah, Bl), (Al, Bh)]
    else:
        terms = [rounded_operands(A, B, O.FMT_E4M3)]
    want = sum(x @ y for x, y in terms)
    mag = sum(np.abs(x) @ np.abs(y) for x, y in terms)
    # fp32 sums of K (split: 3 K) exact products
    bound = 2 * len(terms) * K * 2.0 ** -24 * mag + 2.0 ** -23 * np.abs(want) + 1e-30
    assert np.all(np.abs(dC.double().cpu().numpy() - want) <= bound)
