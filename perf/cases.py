"""Workloads that time the solver through its public entry points.

Each case is one call sequence of a user's program: factor and solve from
device memory, from host memory, through the two reference-shaped entry points,
differentiably, and for a batch.  Orders, conditioning, formats and right-hand
sides are those of the configurations, tests and benchmark of this repository;
``draw`` spreads over the same ranges.
"""
from __future__ import annotations

import math
import random

import torch

import cholesky_gpu_b200 as mp
from cholesky_gpu_b200 import tune

# Factor options by name.  "fp16": the plain method for well-conditioned
# systems; "fp16x2": the FP32-class factor on the tensor cores; "fp32": the
# plain FP32 factor; "growth": switching by the growth criterion over
# E4M3 / FP16 / FP16X2; "rbf": the MXFP8 ladder with its coherence threshold
# that kernel matrices are solved with.
OPTS = {
    "fp16": dict(precision="fp16"),
    "fp16x2": dict(precision="fp16x2"),
    "fp32": dict(precision="fp32"),
    "growth": dict(precision="switching", ladder=["e4m3", "fp16", "fp16x2"], eps_prime=1e-5),
    "rbf": dict(precision="switching", ladder=["mxfp8", "fp16", "fp16x2"], eps_prime=2.0,
                eps_coherence=0.0625),
}
MAX_IT = 200


def listed() -> list[dict]:
    return [
        # the smallest calls: one small system, all launches and waits
        dict(name="solve_512", kind="solve", matrix="spd", n=512, kappa=1e4, nrhs=1, block=128,
             opts="fp16", tol=1e-10),
        # the plain method at its configured size
        dict(name="solve_1024", kind="solve", matrix="spd", n=1024, kappa=1e4, nrhs=1, block=128,
             opts="fp16", tol=1e-10),
        # a middling kernel system of odd order with a few right-hand sides
        dict(name="solve_rbf_2999_x3", kind="solve", matrix="rbf", n=2999, d=784, nrhs=3, block=256,
             opts="rbf", tol=1e-10),
        # the plain FP32 factor, the arm that mixed precision is compared with
        dict(name="solve_fp32_4100_x2", kind="solve", matrix="spd", n=4100, kappa=1e4, nrhs=2,
             block=256, opts="fp32", tol=1e-10),
        # a large ill-conditioned system, switching precision
        dict(name="solve_8192", kind="solve", matrix="spd", n=8192, kappa=1e6, nrhs=1, block=256,
             opts="growth", tol=1e-10),
        # the headline: a kernel matrix with eight right-hand sides
        dict(name="solve_rbf_16384_x8", kind="solve", matrix="rbf", n=16384, d=784, nrhs=8,
             block=256, opts="rbf", tol=1e-10),
        # the same kind of system whose matrix is in page-locked host memory
        dict(name="host_6144", kind="host", matrix="spd", n=6144, kappa=1e6, nrhs=1, block=256,
             opts="growth", tol=1e-10),
        # the drop-in driver: FP64 matrix in, factor object made and freed inside
        dict(name="precond_cg_3072", kind="precond_cg", matrix="spd", n=3072, kappa=1e4, block=256,
             eps=1e-3, tol=1e-10),
        # the drop-in factorization, in place
        dict(name="switching_chol_2048", kind="switching_chol", matrix="spd", n=2048, kappa=1e2,
             block=128, eps=1e-3),
        # building the kernel matrix of image-like points
        dict(name="rbf_build_8192_d784", kind="rbf_build", n=8192, d=784),
        # one training step: solve and gradients for points, lengthscale, nugget, targets
        dict(name="rbf_train_8192_d64", kind="rbf_train", n=8192, d=64, block=256, opts="growth",
             tol=1e-12),
        # many uneven systems at once
        dict(name="batch_128_x4", kind="batch", count=128, lo=64, hi=2048, orders=8, nrhs=4,
             tol=1e-10),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["solve", "solve", "solve", "solve", "host", "precond_cg", "switching_chol",
                       "rbf_build", "rbf_train", "batch"])
    if kind in ("solve", "host"):
        name = rng.choice(["fp16", "fp16x2", "growth", "rbf", "fp32"])
        c = dict(kind=kind, matrix="rbf" if name == "rbf" else "spd")
        big = {"solve": 12000, "host": 8000}[kind]
        c["n"] = _log_int(rng, {"solve": 300, "host": 2000}[kind], 4096 if name == "fp32" else big)
        if name == "rbf":
            c["d"] = 784
        else:
            c["kappa"] = 10.0 ** rng.uniform(2, 4 if name == "fp16" else 6)
        c.update(nrhs=rng.randint(1, 8), block=128 if c["n"] < 1500 else 256, opts=name,
                 tol=1e-10)
        return c
    if kind == "precond_cg":
        return dict(kind=kind, matrix="spd", n=_log_int(rng, 500, 4096),
                    kappa=10.0 ** rng.uniform(2, 4), block=rng.choice([128, 256]), eps=1e-3,
                    tol=1e-10)
    if kind == "switching_chol":
        return dict(kind=kind, matrix="spd", n=_log_int(rng, 500, 4096), kappa=1e2,
                    block=rng.choice([128, 256]), eps=1e-3)
    if kind == "rbf_build":
        return dict(kind=kind, n=_log_int(rng, 500, 8192), d=_log_int(rng, 16, 784))
    if kind == "rbf_train":
        return dict(kind=kind, n=_log_int(rng, 1000, 8192), d=_log_int(rng, 16, 96), block=256,
                    opts="growth", tol=1e-12)
    hi = rng.choice([512, 1024, 2048])
    return dict(kind=kind, count=rng.randint(16, 128), lo=64, hi=hi, orders=rng.randint(0, 999),
                nrhs=rng.randint(1, 8), tol=1e-10)


# ---- inputs, from the seed alone --------------------------------------------

def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _spd(n: int, kappa: float, g: torch.Generator) -> torch.Tensor:
    """Q diag(sigma) Q^T with a geometric spectrum from 1 to 1/kappa and Q a
    product of cosine transforms with random signs between them (a dense
    orthogonal matrix without a QR), FP64."""
    f64 = dict(dtype=torch.float64, device="cuda")
    i = torch.arange(n, **f64)
    C = torch.cos(math.pi / n * (i + 0.5).unsqueeze(0) * i.unsqueeze(1)) * math.sqrt(2.0 / n)
    C[0] *= math.sqrt(0.5)
    s = torch.randint(0, 2, (2, n), generator=g, device="cuda").double() * 2 - 1
    Q = (C * s[0]) @ (C * s[1])
    sig = kappa ** (-i / max(n - 1, 1))
    sig = sig[torch.randperm(n, generator=g, device="cuda")]
    A = (Q * sig) @ Q.t()
    return 0.5 * (A + A.t())


def _points(n: int, d: int, g: torch.Generator, image: bool) -> torch.Tensor:
    """Image-like points in [0,1]^d, 80 % of the coordinates zero, or N(0, I)."""
    if not image:
        return torch.randn((n, d), generator=g, device="cuda")
    X = torch.rand((n, d), generator=g, device="cuda")
    return X * (torch.rand((n, d), generator=g, device="cuda") >= 0.8)


def _lengthscale(X: torch.Tensor) -> float:
    """Median pairwise distance of the first points."""
    return torch.pdist(X[:512].double()).median().item()


def _kernel(X: torch.Tensor, ell: float, nugget: float) -> torch.Tensor:
    """The kernel matrix in FP64."""
    X = X.double()
    sq = (X * X).sum(1)
    K = (X @ X.t()).mul_(2.0).sub_(sq.unsqueeze(1)).sub_(sq.unsqueeze(0)).clamp_max_(0.0)
    K.fill_diagonal_(0.0)
    K.mul_(1.0 / (2.0 * ell * ell)).exp_()
    K.diagonal().add_(nugget)
    return K


def _matrix(case: dict, g: torch.Generator) -> torch.Tensor:
    """The system's matrix in FP32, exactly symmetric."""
    if case["matrix"] == "spd":
        return _spd(case["n"], case["kappa"], g).float()
    X = _points(case["n"], case["d"], g, image=True)
    K = _kernel(X, _lengthscale(X), 1e-3).float()
    return K.tril_().add_(K.tril(-1).t())


def _rhs(n: int, nrhs: int, g: torch.Generator) -> torch.Tensor:
    B = torch.randn((n, nrhs), generator=g, device="cuda", dtype=torch.float64)
    return B[:, 0].contiguous() if nrhs == 1 else B


def _batch_orders(case: dict) -> list[int]:
    """Orders uniform in [lo, hi], the same for every seed: they are the plan."""
    r = random.Random(case["orders"])
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["count"])]


def _batch_inputs(case: dict, g: torch.Generator):
    ns = _batch_orders(case)
    kappas = [10.0 ** (2.0 + 4.0 * v)
              for v in torch.rand(case["count"], generator=g, device="cuda").tolist()]
    As = [_spd(n, k, g).float() for n, k in zip(ns, kappas)]
    return ns, As, [_rhs(n, case["nrhs"], g) for n in ns]


def prepare(case: dict, seed: int) -> dict:
    kind, g = case["kind"], _gen(seed)
    st = dict(case=case)
    if kind in ("solve", "host"):
        n = case["n"]
        st["A"] = _matrix(case, g)
        st["B"] = _rhs(n, case["nrhs"], g)
        if kind == "host":
            st["A"], st["B"] = st["A"].cpu().pin_memory(), st["B"].cpu().pin_memory()
        st["factor"] = mp.Factor(n, block_size=case["block"], **OPTS[case["opts"]])
    elif kind == "precond_cg":
        st["A"] = _matrix(case, g).double()
        st["b"] = _rhs(case["n"], 1, g)
    elif kind == "switching_chol":
        n = case["n"]
        st["A"] = _matrix(case, g)
        st["L"] = torch.empty_like(st["A"])
        st["d"], st["dt"] = (torch.empty(n, device="cuda") for _ in range(2))
    elif kind == "rbf_build":
        st["X"] = _points(case["n"], case["d"], g, image=case["d"] > 64)
        st["ell"] = _lengthscale(st["X"])
    elif kind == "rbf_train":
        n, d = case["n"], case["d"]
        st["X"] = _points(n, d, g, image=False).requires_grad_(True)
        st["ell"] = torch.tensor(0.5 * math.sqrt(d), dtype=torch.float64, requires_grad=True)
        st["nugget"] = torch.tensor(1e-2, dtype=torch.float64, requires_grad=True)
        st["y"] = _rhs(n, 1, g).requires_grad_(True)
    elif kind == "batch":
        ns, st["A"], st["B"] = _batch_inputs(case, g)
        st["batch"] = tune.TunedBatch(ns, nrhs=case["nrhs"], plan=tune.plan_for(ns, case["nrhs"]))
    return st


# ---- one pass ----------------------------------------------------------------

def run(st: dict):
    case = st["case"]
    kind = case["kind"]
    if kind == "solve":
        f = st["factor"].compute(st["A"])
        X, _ = f.pcg(st["A"], st["B"], rel_tol=case["tol"], max_it=MAX_IT)
        return X
    if kind == "host":
        X, _ = st["factor"].solve_host(st["A"], st["B"], rel_tol=case["tol"], max_it=MAX_IT)
        return X
    if kind == "precond_cg":
        x = torch.empty_like(st["b"])
        code = mp.precond_CG(st["A"], x, st["b"], case["n"], case["block"], eps_prime=case["eps"],
                             rel_tol=case["tol"], max_it=MAX_IT)
        return x, code
    if kind == "switching_chol":
        L = st["L"].copy_(st["A"])
        code = mp.switching_chol(L, case["n"], case["block"], st["d"], st["dt"], case["eps"])
        return L.t().tril(), st["d"], st["dt"], code
    if kind == "rbf_build":
        return mp.rbf_build(st["X"], st["ell"], 1e-3, fp64=False)[1]
    if kind == "rbf_train":
        x = mp.rbf_solve(st["X"], st["ell"], st["nugget"], st["y"], rel_tol=case["tol"],
                         max_it=500, block_size=case["block"], **OPTS[case["opts"]])
        loss = 0.5 * (st["y"] * x).sum()
        grads = torch.autograd.grad(loss, [st["X"], st["ell"], st["nugget"], st["y"]])
        return (loss.detach(), x.detach()) + grads
    b = st["batch"]
    b.factor(st["A"])
    Xs, _, _ = b.pcg(st["A"], st["B"], rel_tol=case["tol"], max_it=MAX_IT)
    if case["nrhs"] == 1:
        return torch.cat(Xs)
    return torch.cat([X.t() for X in Xs], dim=1)


# ---- what a pass cannot do without -------------------------------------------

def work(case: dict) -> dict:
    """Each input read and each output written once; n^3/3 for a factor, one
    pair of triangular solves and one product per right-hand side for a solve
    (flops, a multiply-add as two)."""
    kind = case["kind"]
    if kind == "batch":
        ns = [float(n) for n in _batch_orders(case)]
        return dict(bytes=sum(2.0 * n * n + 16.0 * n * case["nrhs"] for n in ns),
                    flops=sum(n ** 3 / 3.0 + 4.0 * n * n * case["nrhs"] for n in ns))
    n = float(case["n"])
    if kind == "rbf_build":
        return dict(bytes=4.0 * n * case["d"] + 2.0 * n * n, flops=1.5 * n * n * case["d"])
    if kind == "rbf_train":
        d = case["d"]
        return dict(bytes=8.0 * n * d + 40.0 * n,
                    flops=n ** 3 / 3.0 + 8.0 * n * n + 1.5 * n * n * d + 2.0 * n * n * (2 + 2 * d))
    if kind == "switching_chol":
        return dict(bytes=4.0 * n * n + 8.0 * n, flops=n ** 3 / 3.0)
    nrhs = case.get("nrhs", 1)
    elem = 8.0 if kind == "precond_cg" else 4.0
    return dict(bytes=0.5 * elem * n * n + 16.0 * n * nrhs,
                flops=n ** 3 / 3.0 + 4.0 * n * n * nrhs)


# ---- what plain torch gives in 64 bits -----------------------------------------

def _dense_solve(A: torch.Tensor, B: torch.Tensor) -> torch.Tensor:
    """Cholesky solve with one step of refinement, all in FP64."""
    L = torch.linalg.cholesky(A)
    B2 = B.reshape(A.shape[0], -1)
    X = torch.cholesky_solve(B2, L)
    X = X + torch.cholesky_solve(B2 - A @ X, L)
    return X.reshape(B.shape)


def _exact_train(case: dict, g: torch.Generator):
    n, d = case["n"], case["d"]
    X = _points(n, d, g, image=False).double().requires_grad_(True)
    ell = torch.tensor(0.5 * math.sqrt(d), dtype=torch.float64, device="cuda", requires_grad=True)
    nugget = torch.tensor(1e-2, dtype=torch.float64, device="cuda", requires_grad=True)
    y = _rhs(n, 1, g)
    with torch.enable_grad():
        sq = (X * X).sum(1)
        r2 = sq.unsqueeze(1) + sq.unsqueeze(0) - 2.0 * (X @ X.t())
        r2 = r2 * (1.0 - torch.eye(n, dtype=torch.float64, device="cuda"))
        K = torch.exp(-r2 / (2.0 * ell * ell))
        K = K + nugget * torch.eye(n, dtype=torch.float64, device="cuda")
        with torch.no_grad():
            x = _dense_solve(K, y)
        # d(y^T K^-1 y / 2) = -x^T dK x / 2
        surrogate = -0.5 * (x @ (K @ x))
        gX, gl, gn = torch.autograd.grad(surrogate, [X, ell, nugget])
    # the loss reads y directly and through x = K^-1 y: each gives x / 2
    return 0.5 * (y @ x), x, gX, gl, gn, x


def exact(case: dict, seed: int):
    kind, g = case["kind"], _gen(seed)
    if kind in ("solve", "host"):
        A = _matrix(case, g)
        X = _dense_solve(A.double(), _rhs(case["n"], case["nrhs"], g))
        return X.cpu() if kind == "host" else X
    if kind == "precond_cg":
        A = _matrix(case, g).double()
        return _dense_solve(A, _rhs(case["n"], 1, g)), None
    if kind == "switching_chol":
        A = _matrix(case, g).double()
        L = torch.linalg.cholesky(A)
        return L, A.diagonal().clone(), None, None
    if kind == "rbf_build":
        X = _points(case["n"], case["d"], g, image=case["d"] > 64)
        return _kernel(X, _lengthscale(X), 1e-3).tril_()
    if kind == "rbf_train":
        return _exact_train(case, g)
    ns, As, Bs = _batch_inputs(case, g)
    Xs = [_dense_solve(A.double(), B) for A, B in zip(As, Bs)]
    return torch.cat(Xs) if case["nrhs"] == 1 else torch.cat([X.t() for X in Xs], dim=1)
