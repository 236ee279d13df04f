"""The work a user of this package has it do, as measured cases.

Kernel ridge regression and Gaussian-process models on one GPU: build the
kernel matrix in RFP (`ssfrk`), shift its diagonal, factor, solve; keep a
factor and solve with it again; refine a solve; invert; pack and unpack;
multiply; differentiate a likelihood.  Every case goes through the package's
public Python functions.

`listed()` gives the cases, `draw(rng)` another one of the same ranges,
`prepare(case, seed)` a program's state before the call, `run(state)` one
pass, `work(case)` the bytes and operations a pass cannot do without, and
`exact(case, seed)` what the pass returns, computed in 64 bits by plain torch.

The matrices are A A^T + I with A ~ N(0, 1) / sqrt(k) (n x k, k >= n / 64),
the benchmark's and the tests' distribution: condition numbers up to ~80, the
range of a regularised kernel matrix on standardised data.
"""
import math

import torch

import curfp_b200 as curfp
from curfp_b200 import autograd as AG
from curfp_b200 import precision as P

VARIANTS = [(t, u) for t in "NT" for u in "LU"]


def listed():
    return [
        # The smallest use: a few hundred training points, one target.  Every
        # launch and every host call shows.
        dict(name="krr_small", kind="krr", n=250, k=100, nrhs=1, transr="T", uplo="U"),
        # The tests' pipeline size (n = 4095, k = 128, 64 right-hand sides), odd order.
        dict(name="krr_4095", kind="krr", n=4095, k=128, nrhs=64, transr="N", uplo="L"),
        # The benchmark's headline size, default layout.
        dict(name="krr_32768", kind="krr", n=32768, k=1024, nrhs=64, transr="T", uplo="U"),
        # The plain FP32 form: FP32 FMA contractions chosen by the caller.
        dict(name="krr_fp32", kind="krr_fp32", n=8192, k=512, nrhs=16, transr="T", uplo="L"),
        # The precision form: factor, then a solve refined with FP64 residuals.
        dict(name="refined", kind="refined", n=16384, k=512, nrhs=64, transr="N", uplo="U"),
        # The inverse of a kernel matrix from its factor (leave-one-out
        # errors, posterior covariances).
        dict(name="inverse", kind="inverse", n=6001, transr="T", uplo="L"),
        # A kept factor and one new target at a time (retraining on new labels).
        dict(name="solve_one", kind="solve", n=16383, nrhs=1, transr="T", uplo="U"),
        # A kept factor and a batch of right-hand sides (posterior variances of test points).
        dict(name="solve_many", kind="solve", n=8192, nrhs=400, transr="N", uplo="L"),
        # A dense symmetric matrix to RFP and back.
        dict(name="pack", kind="pack", n=12345, transr="T", uplo="U"),
        # The kernel matrix times a vector (predictions on the training set,
        # residuals, iterative solvers).
        dict(name="multiply", kind="multiply", n=16001, cols=1, transr="N", uplo="U"),
        # The FP64 twins of the pipeline.
        dict(name="krr_fp64", kind="krr_fp64", n=3000, k=200, nrhs=10, transr="T", uplo="U"),
        # A training step: negative log marginal likelihood and its gradients
        # (n = 8192, d = 256, the tests' and the benchmark's size).
        dict(name="nll_step", kind="nll", n=8192, k=256, transr="T", uplo="U", math="bf16x3"),
    ]


# Ranges of each kind: order, and columns (right-hand sides, or columns of the
# multiplied block).
RANGES = {
    "krr": ((100, 32768), (1, 64)),
    "krr_fp32": ((500, 8192), (1, 64)),
    "refined": ((1000, 16384), (1, 64)),
    "inverse": ((200, 8192), None),
    "solve": ((300, 20000), (1, 400)),
    "pack": ((500, 20000), None),
    "multiply": ((500, 20000), (1, 64)),
    "krr_fp64": ((200, 4096), (1, 64)),
    "nll": ((500, 8192), None),
}


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(sorted(RANGES))
    (lo, hi), cols = RANGES[kind]
    n = spread(lo, hi)
    transr, uplo = rng.choice(VARIANTS)
    case = dict(kind=kind, n=n, transr=transr, uplo=uplo)
    if kind.startswith("krr") or kind == "refined":
        case["k"] = spread(max(32, n // 64 + 1), 1024)
    if kind == "nll":
        case["k"] = spread(max(16, n // 64 + 1), 512)
        case["math"] = rng.choice(["bf16x3", "fp32"])
    if kind == "multiply":
        case["cols"] = spread(*cols)
    elif cols:
        case["nrhs"] = spread(*cols)
    return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _normal(g, *shape, dtype=torch.float32):
    return torch.randn(*shape, generator=g, device="cuda", dtype=dtype)


def _features(case, g, dtype=torch.float32):
    return _normal(g, case["n"], case["k"], dtype=dtype) / math.sqrt(case["k"])


def _kernel(n, g):
    """The dense A A^T + I of a kept factor's or a packed matrix's case."""
    k = max(32, n // 32)
    A = _normal(g, n, k) / math.sqrt(k)
    K = A @ A.t()
    K.diagonal().add_(1.0)
    return K


def _rfp(M, transr, uplo):
    """LAPACK's RFP array of the lower triangle of the dense M (UPLO = U: of
    its transpose, an upper triangle), by slices."""
    n = M.shape[0]
    n1 = n - n // 2 if uplo == "L" else n // 2   # order of the leading block
    rows = n + 1 if n % 2 == 0 else n
    AR = M.new_zeros(rows, (n + 1) // 2)
    if uplo == "L":
        top = 1 if n % 2 == 0 else 0             # first row of the leading trapezoid
        AR[top:, :] = M[:, :n1].tril()
        AR[:n - n1, 1 - top:] += M[n1:, n1:].t().triu()
    else:
        U = M.t()
        AR[:n, :] = U[:, n1:].triu(-n1)
        AR[rows - n1:, :n1] += U[:n1, :n1].t().tril()
    return (AR if transr == "T" else AR.t()).reshape(-1)


def _factor(n, g):
    return torch.linalg.cholesky(_kernel(n, g))


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def prepare(case, seed):
    g = _generator(seed)
    kind, n = case["kind"], case["n"]
    size = n * (n + 1) // 2
    lay = dict(transr=case["transr"], uplo=case["uplo"])
    s = dict(kind=kind, lay=lay)
    if kind in ("krr", "krr_fp32", "refined", "krr_fp64"):
        dtype = torch.float64 if kind == "krr_fp64" else torch.float32
        s["A"] = _features(case, g, dtype)
        s["B"] = _normal(g, n, case["nrhs"], dtype=dtype)
        s["C"] = torch.empty(size, device="cuda", dtype=dtype)
        s["X"] = torch.empty_like(s["B"])
        if kind == "refined":
            s["F"] = torch.empty_like(s["C"])
    elif kind == "inverse":
        s["F"] = _rfp(_factor(n, g), **lay)
        s["C"] = torch.empty_like(s["F"])
    elif kind == "solve":
        s["F"] = _rfp(_factor(n, g), **lay)
        s["B"] = _normal(g, n, case["nrhs"])
        s["X"] = torch.empty_like(s["B"])
    elif kind == "pack":
        s["K"] = _kernel(n, g)
    elif kind == "multiply":
        s["C"] = _rfp(_kernel(n, g), **lay)
        s["B"] = _normal(g, n) if case["cols"] == 1 else _normal(g, n, case["cols"])
    else:
        s["A"] = _normal(g, n, case["k"])
        s["y"] = _normal(g, n)
        s["k"], s["math"] = case["k"], case["math"]
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def run(s):
    kind, lay = s["kind"], s["lay"]
    if kind == "krr":
        curfp.ssfrk(s["A"], s["C"], **lay)
        curfp.add_to_diagonal(s["C"], 1.0, **lay)
        curfp.spftrf(s["C"], **lay)
        s["X"].copy_(s["B"])
        curfp.spftrs(s["C"], s["X"], **lay)
        return dict(factor=s["C"], x=s["X"])
    if kind == "krr_fp32":
        P.ssfrk(s["A"], s["C"], math="fp32", **lay)
        curfp.add_to_diagonal(s["C"], 1.0, **lay)
        P.spftrf(s["C"], math="fp32", **lay)
        s["X"].copy_(s["B"])
        curfp.spftrs(s["C"], s["X"], **lay)
        return dict(factor=s["C"], x=s["X"])
    if kind == "refined":
        P.ssfrk(s["A"], s["C"], **lay)
        curfp.add_to_diagonal(s["C"], 1.0, **lay)
        s["F"].copy_(s["C"])
        P.spftrf(s["F"], **lay)
        s["X"].copy_(s["B"])
        P.spftrs_refined(s["C"], s["F"], s["X"], **lay)
        return dict(kernel=s["C"], factor=s["F"], x=s["X"])
    if kind == "inverse":
        s["C"].copy_(s["F"])
        curfp.spftri(s["C"], **lay)
        return s["C"]
    if kind == "solve":
        s["X"].copy_(s["B"])
        curfp.spftrs(s["F"], s["X"], **lay)
        return s["X"]
    if kind == "pack":
        arf = curfp.strttf(s["K"], **lay)
        return dict(arf=arf, dense=curfp.stfttr(arf, **lay))
    if kind == "multiply":
        if s["B"].ndim == 1:
            return curfp.ssfmv(s["C"], s["B"], **lay)
        return curfp.ssfmm(s["C"], s["B"], **lay)
    if kind == "krr_fp64":
        curfp.dsfrk(s["A"], s["C"], **lay)
        curfp.add_to_diagonal(s["C"], 1.0, **lay)
        curfp.dpftrf(s["C"], **lay)
        s["X"].copy_(s["B"])
        curfp.dpftrs(s["C"], s["X"], **lay)
        return dict(factor=s["C"], x=s["X"])
    X = s["A"].detach().requires_grad_(True)
    scale = torch.tensor(1.0 / s["k"], device="cuda", requires_grad=True)
    noise = torch.tensor(1.0, device="cuda", requires_grad=True)
    loss = AG.nll(X, scale, noise, s["y"], math=s["math"], **lay)
    loss.backward()
    return dict(loss=loss.detach(), x=X.grad, scale=scale.grad, noise=noise.grad)


# ---------------------------------------------------------------------------
# What a pass cannot do without, and its values in 64 bits
# ---------------------------------------------------------------------------

def work(case):
    kind, n = case["kind"], case["n"]
    size = n * (n + 1) // 2
    k, nrhs = case.get("k", 0), case.get("nrhs", 0)
    if kind in ("krr", "krr_fp32", "krr_fp64"):
        w = 8 if kind == "krr_fp64" else 4
        return dict(bytes=w * (n * k + size + 2 * n * nrhs),
                    flops=n * (n + 1) * k + n ** 3 / 3 + 2 * n * n * nrhs)
    if kind == "refined":  # one solve, one residual, one correction
        return dict(bytes=4 * (n * k + 2 * size + 2 * n * nrhs),
                    flops=n * (n + 1) * k + n ** 3 / 3 + 6 * n * n * nrhs)
    if kind == "inverse":
        return dict(bytes=4 * 2 * size, flops=2 * n ** 3 / 3)
    if kind == "solve":
        return dict(bytes=4 * (size + 2 * n * nrhs), flops=2 * n * n * nrhs)
    if kind == "pack":  # the triangle in, the array out; the array in, the square out
        return dict(bytes=4 * (3 * size + n * n), flops=0)
    if kind == "multiply":
        return dict(bytes=4 * (size + 2 * n * case["cols"]), flops=2 * n * n * case["cols"])
    # rank-k update, factor, inverse of the factor, two solves with k columns
    return dict(bytes=4 * (2 * n * k + 2 * n),
                flops=n * (n + 1) * k + 2 * n ** 3 / 3 + 2 * n * n * k)


def exact(case, seed):
    g = _generator(seed)
    kind, n = case["kind"], case["n"]
    lay = dict(transr=case["transr"], uplo=case["uplo"])
    if kind in ("krr", "krr_fp32", "refined", "krr_fp64"):
        dtype = torch.float64 if kind == "krr_fp64" else torch.float32
        A = _features(case, g, dtype).double()
        B = _normal(g, n, case["nrhs"], dtype=dtype).double()
        K = A @ A.t()
        K.diagonal().add_(1.0)
        out = dict(kernel=_rfp(K, **lay)) if kind == "refined" else {}
        L = torch.linalg.cholesky(K)
        del K
        out.update(x=torch.cholesky_solve(B, L), factor=_rfp(L, **lay))
        return out
    if kind == "inverse":
        L = _factor(n, g).double()
        return _rfp(torch.cholesky_inverse(L), **lay)
    if kind == "solve":
        L = _factor(n, g).double()
        return torch.cholesky_solve(_normal(g, n, case["nrhs"]).double(), L)
    if kind == "pack":
        K = _kernel(n, g).double()
        # the stored triangle is the one of row-major K that UPLO names
        arf = _rfp(K if lay["uplo"] == "L" else K.t(), **lay)
        return dict(arf=arf, dense=K.tril() if lay["uplo"] == "L" else K.triu())
    if kind == "multiply":
        K = _kernel(n, g).double().tril()
        B = (_normal(g, n) if case["cols"] == 1 else _normal(g, n, case["cols"])).double()
        b = B.reshape(-1, n).t()  # ssfmm takes the storage as column-major, n rows
        return (K @ b + K.tril(-1).t() @ b).t().reshape(B.shape)
    X = _normal(g, n, case["k"]).double()
    y = _normal(g, n).double()
    scale = torch.tensor(1.0 / case["k"], dtype=torch.float32).double().item()
    C = scale * (X @ X.t())
    C.diagonal().add_(1.0)
    L = torch.linalg.cholesky(C)
    del C
    a = torch.cholesky_solve(y[:, None], L)
    loss = 0.5 * torch.dot(y, a[:, 0]) + L.diagonal().log().sum()
    inv = torch.cholesky_inverse(L)
    Cbar = 0.5 * (inv - a @ a.t())
    G = Cbar @ X
    return dict(loss=loss, x=2.0 * scale * G, scale=(G * X).sum(), noise=Cbar.diagonal().sum())
