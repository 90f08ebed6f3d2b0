"""The work that programs built on this framework spend their time in, as measurable cases.

Every case is one call (or one short call sequence) of the public entry
points on inputs a program has in GPU memory: factorizations of one matrix in
each storage / update type, the Schur update on its own, a solve with kept
factors, the mixed-precision solve, the differentiable solve, and the batched
factorization and differentiable solve.

    listed()            the fixed cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs, plans and buffers, on the GPU
    run(state)          one pass
    work(case)          bytes and flops a pass cannot do without
    exact(case, seed)   what run() returns, computed by torch in 64 bits
"""
from __future__ import annotations

import math

import numpy as np
import torch

import remifa_b200 as rb
from remifa_b200.autograd import lu_solve_autograd
from remifa_b200.batch import BatchPlan, MatrixBatch, RhsBatch, batch_sizes, batched_lu_solve

DEV = "cuda"
OUTER = {"fp32": rb.compute_type.FP32, "fp16": rb.compute_type.TC32,
         "bf16": rb.compute_type.TC32_BF16, "e4m3": rb.compute_type.TC32_E4M3,
         "split": rb.compute_type.TC32_SPLIT}


def listed():
    return [
        # One small factorization in fp32: what a call costs where launches
        # and the dependency chain are everything.
        dict(name="rl_fp32_n200", kind="rl", n=200, outer="fp32", nb=256, alpha=1.5),
        # The plain fp32 factorization at the size the reference reports.
        dict(name="rl_fp32_n4096", kind="rl", n=4096, outer="fp32", nb=256, alpha=1.5),
        # The headline: large matrix, fp16 tensor-core trailing updates.
        dict(name="rl_fp16_n16384", kind="rl", n=16384, outer="fp16", nb=256, alpha=1.5),
        # An ordinary ragged size with bf16 updates.
        dict(name="rl_bf16_n5001", kind="rl", n=5001, outer="bf16", nb=256, alpha=1.5),
        # fp8 updates (power-of-two tile scales), the cheapest operand type.
        dict(name="rl_e4m3_n8192", kind="rl", n=8192, outer="e4m3", nb=256, alpha=1.5),
        # Left-looking on fp16 storage: half the memory, the reference's
        # fp16 wrappers.
        dict(name="ll_f16_n8192", kind="ll", n=8192, outer="fp16", nb=256, alpha=1.5),
        # A Schur update by itself, fp16 operands, ragged in every direction.
        dict(name="gemm_fp16_m6000_k500", kind="gemm", m=6000, n=7000, k=500),
        # A system with one right-hand side solved to fp64 accuracy: factor
        # in mixed precision, refine.
        dict(name="gesv_n2000", kind="gesv", n=2000, outer="fp16", solver="classic", alpha=1.5),
        # One more right-hand side with factors kept from before.
        dict(name="solve_n10007", kind="solve", n=10007, nrhs=1, trans=False),
        # The differentiable solve, forward and backward, 64 right-hand sides.
        dict(name="adjoint_n8192_rhs64", kind="adjoint", n=8192, nrhs=64, outer="fp16", alpha=2.0),
        # Ten thousand small matrices of uneven sizes 16 .. 511, factored.
        dict(name="batch_10000_n16_511", kind="batch", count=10000, lo=16, ratio=32.0,
             sizes_seed=11, outer="fp16", alpha=1.5),
        # The differentiable batched solve, forward and backward.
        dict(name="batch_grad_1024_n64_256", kind="batch_grad", count=1024, lo=64, hi=256,
             sizes_seed=12, nrhs=1, outer="fp16", iters=4, alpha=2.0),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["rl", "rl", "rl", "ll", "gemm", "gesv", "solve", "adjoint", "batch",
                       "batch_grad"])
    if kind == "rl":
        outer = rng.choice(["fp32", "fp16", "bf16", "e4m3", "split"])
        top = {"fp32": 6000, "split": 10000}.get(outer, 16384)
        return dict(kind="rl", n=_log_int(rng, 100, top), outer=outer,
                    nb=rng.choice([256, 256, 128]), alpha=rng.choice([1.05, 1.5, 4.0]))
    if kind == "ll":
        return dict(kind="ll", n=_log_int(rng, 100, 12000), outer="fp16",
                    nb=rng.choice([256, 128]), alpha=rng.choice([1.5, 4.0]))
    if kind == "gemm":
        return dict(kind="gemm", m=_log_int(rng, 100, 12000), n=_log_int(rng, 100, 12000),
                    k=_log_int(rng, 32, 2048))
    if kind == "gesv":
        return dict(kind="gesv", n=_log_int(rng, 100, 8192), outer=rng.choice(["fp16", "bf16"]),
                    solver=rng.choice(["classic", "classic", "gmres"]),
                    alpha=rng.choice([1.5, 4.0]))
    if kind == "solve":
        return dict(kind="solve", n=_log_int(rng, 100, 16384),
                    nrhs=rng.choice([1, 1, 2, 3, 8, 17, 64]), trans=rng.random() < 0.5)
    if kind == "adjoint":
        return dict(kind="adjoint", n=_log_int(rng, 200, 8000),
                    nrhs=rng.choice([1, 4, 16, 30, 64]), outer=rng.choice(["fp16", "bf16"]),
                    alpha=2.0)
    if kind == "batch":
        return dict(kind="batch", count=_log_int(rng, 100, 9000), lo=16,
                    ratio=rng.choice([4.0, 8.0, 16.0, 32.0]), sizes_seed=rng.randrange(1000),
                    outer=rng.choice(["fp16", "fp16", "fp32"]), alpha=1.5)
    hi = rng.choice([96, 160, 256, 400])
    return dict(kind="batch_grad", count=_log_int(rng, 16, 1000), lo=rng.choice([16, 32, 64]),
                hi=hi, sizes_seed=rng.randrange(1000), nrhs=rng.choice([1, 1, 2, 5]),
                outer=rng.choice(["fp16", "fp32"]), iters=rng.choice([2, 4]), alpha=2.0)


# ---- inputs -------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _dominant(n, alpha, g, dtype=torch.float32):
    """Column-major n x n: R ~ N(0,1)/sqrt(n) with row dominance alpha."""
    lda = (n + 15) // 16 * 16
    a = rb.colmajor_empty(n, n, lda, torch.float32, DEV)
    a.copy_(torch.randn(n, n, device=DEV, generator=g).t().mul_(1.0 / math.sqrt(n)))
    d = a.diagonal()
    d.copy_((a.abs().sum(1) - d.abs()) * alpha)
    if dtype == torch.float32:
        return a
    out = rb.colmajor_empty(n, n, lda, dtype, DEV)
    out.copy_(a)
    return out


def _factors(n, g):
    """A packed L\\U pair: unit lower L with small entries, U with a
    dominant diagonal, as the factorization of a dominant matrix leaves it."""
    lda = (n + 15) // 16 * 16
    f = rb.colmajor_empty(n, n, lda, torch.float32, DEV)
    f.copy_(torch.randn(n, n, device=DEV, generator=g).t().mul_(1.0 / math.sqrt(n)))
    rows = f.abs().sum(1)
    i = torch.arange(n, device=DEV)
    f.copy_(torch.where(i[:, None] > i[None, :], f / rows[None, :], f))
    f.diagonal().copy_(1.5 * rows)
    return f


def _sizes(case):
    if case["kind"] == "batch":
        return batch_sizes(case["count"], seed=case["sizes_seed"], lo=case["lo"],
                           ratio=case["ratio"])
    rng = np.random.default_rng(case["sizes_seed"])
    return rng.integers(case["lo"], case["hi"] + 1, size=case["count"]).astype(np.int32)


def _batch_data(mats, alpha, g):
    """Off-diagonal entries U[-1, 1), diagonal alpha times their expected
    absolute row sum plus one (padding rows zero)."""
    n, lda, off = mats.sizes.astype(np.int64), mats.lda.astype(np.int64), mats.offsets[:-1]
    mats.data.uniform_(-1.0, 1.0, generator=g)
    first = np.repeat(np.cumsum(n) - n, n)
    k = np.arange(int(n.sum()), dtype=np.int64) - first
    start, step, size = np.repeat(off, n), np.repeat(lda, n), np.repeat(n, n)
    diag = torch.from_numpy(start + k * (step + 1)).to(DEV)
    mats.data[diag] = torch.from_numpy((alpha * (size * 0.5 + 1.0)).astype(np.float32)).to(DEV)
    for p in range(1, mats.align):
        sel = (step - size) >= p
        if sel.any():
            pad = (start + k * step + size + p - 1)[sel]
            mats.data[torch.from_numpy(pad).to(DEV)] = 0.0
    return mats


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind in ("rl", "ll"):
        s["a"] = _dominant(case["n"], case["alpha"], g,
                           torch.float16 if kind == "ll" else torch.float32)
        s["lu"] = rb.colmajor_empty(*s["a"].shape, rb.ld(s["a"]), s["a"].dtype, DEV)
    elif kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]

        def cm(r, c, dtype):
            ld = (r + 15) // 16 * 16
            t = rb.colmajor_empty(r, c, ld, dtype, DEV)
            t.copy_(torch.randn(c, r, device=DEV, generator=g).t())
            return t
        s["a"], s["b"] = cm(m, k, torch.float16), cm(k, n, torch.float16)
        s["a"].mul_(1.0 / math.sqrt(k))
        s["c"] = cm(m, n, torch.float32)
    elif kind == "gesv":
        n = case["n"]
        s["a"] = _dominant(n, case["alpha"], g)
        s["b"] = torch.randn(n, dtype=torch.float64, device=DEV, generator=g)
    elif kind == "solve":
        n, k = case["n"], case["nrhs"]
        s["lu"] = _factors(n, g)
        s["b"] = torch.randn(k, n, dtype=torch.float64, device=DEV, generator=g).t()
        s["x"] = torch.empty(k, n, dtype=torch.float64, device=DEV).t()
    elif kind == "adjoint":
        n, k = case["n"], case["nrhs"]
        s["a"] = _dominant(n, case["alpha"], g).requires_grad_(True)
        s["b"] = torch.randn(n, k, dtype=torch.float64, device=DEV,
                             generator=g).requires_grad_(True)
        s["g"] = torch.randn(n, k, dtype=torch.float64, device=DEV, generator=g)
    elif kind == "batch":
        sizes = _sizes(case)
        s["mats"] = _batch_data(MatrixBatch(sizes, align=4), case["alpha"], g)
        s["plan"] = BatchPlan(sizes, outer=OUTER[case["outer"]])
        s["lu"] = s["mats"].like()
        s["info"] = torch.zeros(len(sizes), dtype=torch.int32, device=DEV)
    else:
        sizes, k = _sizes(case), case["nrhs"]
        s["layout"] = _batch_data(MatrixBatch(sizes, align=4), case["alpha"], g)
        s["plan"] = BatchPlan(sizes, outer=OUTER[case["outer"]])
        s["a"] = s["layout"].data.clone().requires_grad_(True)
        nb = int(sizes.sum()) * k
        s["b"] = torch.randn(nb, dtype=torch.float64, device=DEV,
                             generator=g).requires_grad_(True)
        s["g"] = torch.randn(nb, dtype=torch.float64, device=DEV, generator=g)
    return s


# ---- one pass -----------------------------------------------------------

def run(s):
    c, kind = s["case"], s["kind"]
    if kind == "rl":
        s["lu"].copy_(s["a"])
        info = rb.lu_nopiv_rl(s["lu"], nb=c["nb"], outer=OUTER[c["outer"]])
        return {"lu": s["lu"], "info": info}
    if kind == "ll":
        s["lu"].copy_(s["a"])
        info = rb.lu_nopiv_ll(s["lu"], nb=c["nb"], outer=OUTER[c["outer"]])
        return {"lu": s["lu"], "info": info}
    if kind == "gemm":
        # C -= A B in place: a program's next update goes on from this C
        return {"c": rb.gemmex(rb.TC32, -1.0, s["a"], s["b"], 1.0, s["c"])}
    if kind == "gesv":
        x, info, _, _ = rb.gesv_mixed(s["a"], s["b"], outer=OUTER[c["outer"]],
                                      solver=c["solver"])
        return {"x": x, "info": info}
    if kind == "solve":
        s["x"].copy_(s["b"])
        return {"x": rb.lu_solve(s["lu"], s["x"], trans=c["trans"])}
    if kind == "adjoint":
        x = lu_solve_autograd(s["a"], s["b"], outer=OUTER[c["outer"]])
        da, db = torch.autograd.grad(x, (s["a"], s["b"]), s["g"])
        return {"x": x.detach(), "da": da, "db": db}
    if kind == "batch":
        s["lu"].data.copy_(s["mats"].data)
        s["plan"](s["lu"], s["info"])
        return {"lu": s["lu"].data, "info": s["info"]}
    x = batched_lu_solve(s["a"], s["b"], s["layout"], s["plan"], nrhs=c["nrhs"],
                         refine_iters=c["iters"])
    da, db = torch.autograd.grad(x, (s["a"], s["b"]), s["g"])
    return {"x": x.detach(), "da": da, "db": db}


def work(case):
    kind = case["kind"]
    if kind in ("rl", "ll"):
        n = float(case["n"])
        return {"bytes": 2 * n * n * (2 if kind == "ll" else 4), "flops": 2 * n ** 3 / 3}
    if kind == "gemm":
        m, n, k = float(case["m"]), float(case["n"]), float(case["k"])
        return {"bytes": 2 * (m + n) * k + 8 * m * n, "flops": 2 * m * n * k}
    if kind == "gesv":
        n = float(case["n"])
        return {"bytes": 4 * n * n + 16 * n, "flops": 2 * n ** 3 / 3 + 4 * n * n}
    if kind == "solve":
        n, k = float(case["n"]), float(case["nrhs"])
        return {"bytes": 4 * n * n + 16 * n * k, "flops": 2 * n * n * k}
    if kind == "adjoint":
        n, k = float(case["n"]), float(case["nrhs"])
        return {"bytes": 8 * n * n + 32 * n * k, "flops": 2 * n ** 3 / 3 + 6 * n * n * k}
    n = _sizes(case).astype(np.float64)
    if kind == "batch":
        return {"bytes": float(8 * (n * n).sum()), "flops": float((2 * n ** 3 / 3).sum())}
    k = float(case["nrhs"])
    return {"bytes": float((8 * n * n + 32 * n * k).sum()),
            "flops": float((2 * n ** 3 / 3 + 6 * n * n * k).sum())}


# ---- the same in 64 bits ------------------------------------------------

def _lu64(a):
    """In-place L\\U of fp64 matrices (..., n, n) without pivoting."""
    def rec(lo, hi):
        if hi - lo <= 32:
            for j in range(lo, hi - 1):
                a[..., j + 1:hi, j] /= a[..., j, j, None]
                a[..., j + 1:hi, j + 1:hi] -= (a[..., j + 1:hi, j, None]
                                               * a[..., None, j, j + 1:hi])
            return
        mid = lo + max(32, (hi - lo) // 2 // 32 * 32)
        rec(lo, mid)
        d = a[..., lo:mid, lo:mid]
        a[..., lo:mid, mid:hi] = torch.linalg.solve_triangular(
            d, a[..., lo:mid, mid:hi], upper=False, unitriangular=True)
        a[..., mid:hi, lo:mid] = torch.linalg.solve_triangular(
            d, a[..., mid:hi, lo:mid], upper=True, left=False)
        a[..., mid:hi, mid:hi] -= a[..., mid:hi, lo:mid] @ a[..., lo:mid, mid:hi]
        rec(mid, hi)
    rec(0, a.shape[-1])
    return a


def _padded_groups(mats):
    """(matrix numbers, flat index, validity mask, padded size) for groups of
    matrices of nearly one size."""
    top = (mats.sizes.astype(np.int64) + 63) // 64 * 64
    for p in np.unique(top):
        every = np.nonzero(top == p)[0]
        per = max(1, int(4e7 // (p * p)))
        for at in range(0, len(every), per):
            i = every[at:at + per]
            n = torch.from_numpy(mats.sizes[i].astype(np.int64)).to(DEV)[:, None, None]
            lda = torch.from_numpy(mats.lda[i].astype(np.int64)).to(DEV)[:, None, None]
            off = torch.from_numpy(mats.offsets[:-1][i]).to(DEV)[:, None, None]
            r = torch.arange(int(p), device=DEV)
            ok = (r[None, :, None] < n) & (r[None, None, :] < n)
            idx = torch.where(ok, off + r[None, :, None] + r[None, None, :] * lda, 0)
            yield i, idx, ok, int(p)


def _gather(data, idx, ok, p):
    eye = torch.eye(p, dtype=torch.float64, device=DEV)
    return torch.where(ok, data[idx].double(), eye)


def exact(case, seed):
    kind = case["kind"]
    s = prepare(case, seed)
    if kind in ("rl", "ll"):
        return {"lu": _lu64(s["a"].double().contiguous()), "info": None}
    if kind == "gemm":
        return {"c": s["c"].double() - s["a"].double() @ s["b"].double()}
    if kind == "gesv":
        return {"x": torch.linalg.solve(s["a"].double(), s["b"]), "info": None}
    if kind == "solve":
        f = s["lu"].double()
        low = dict(upper=False, unitriangular=True)
        if not case["trans"]:
            y = torch.linalg.solve_triangular(f, s["b"], **low)
            return {"x": torch.linalg.solve_triangular(f, y, upper=True)}
        y = torch.linalg.solve_triangular(f.t(), s["b"], upper=False)
        return {"x": torch.linalg.solve_triangular(f.t(), y, upper=True, unitriangular=True)}
    if kind == "adjoint":
        a = s["a"].detach().double()
        x = torch.linalg.solve(a, s["b"].detach())
        db = torch.linalg.solve(a.t(), s["g"])
        return {"x": x, "da": -(db @ x.t()), "db": db}
    if kind == "batch":
        out = s["mats"].data.double()
        for _, idx, ok, p in _padded_groups(s["mats"]):
            out[idx[ok]] = _lu64(_gather(s["mats"].data, idx, ok, p))[ok]
        return {"lu": out, "info": None}
    lay, k = s["layout"], case["nrhs"]
    rhs = RhsBatch(lay.sizes, k)
    b, g = s["b"].detach(), s["g"]
    x, db = torch.zeros_like(b), torch.zeros_like(b)
    da = torch.zeros(lay.data.numel(), dtype=torch.float64, device=DEV)
    for i, idx, ok, p in _padded_groups(lay):
        n = torch.from_numpy(lay.sizes[i].astype(np.int64)).to(DEV)[:, None, None]
        off = torch.from_numpy(rhs.offsets[:-1][i]).to(DEV)[:, None, None]
        r = torch.arange(p, device=DEV)[None, :, None]
        okv = (r < n).expand(-1, -1, k)
        vi = torch.where(okv, off + r + torch.arange(k, device=DEV)[None, None, :] * n, 0)
        a = _gather(s["a"].detach(), idx, ok, p)
        xs = torch.linalg.solve(a, torch.where(okv, b[vi], 0.0))
        ds = torch.linalg.solve(a.mT, torch.where(okv, g[vi], 0.0))
        x[vi[okv]], db[vi[okv]] = xs[okv], ds[okv]
        da[idx[ok]] = -(ds @ xs.mT)[ok]
    return {"x": x, "da": da, "db": db}
