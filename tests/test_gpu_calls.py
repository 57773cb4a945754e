"""How calls share memory, streams and threads: solves in place, objects freed
while others work, calls from several threads at once."""
import ctypes

import pytest
import torch

import cholesky_gpu_b200 as mp
from cholesky_gpu_b200 import _lib, matgen

pytestmark = pytest.mark.gpu


def _stream():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("n", [9, 512, 1000, 1024, 1025])
@pytest.mark.parametrize("nrhs", [1, 4])
@pytest.mark.parametrize("f64", [False, True])
def test_the_solution_may_overwrite_the_right_hand_side(n, nrhs, f64):
    """mpchol_pcg, mpchol_pcg_f64 and mpchol_adjoint_solve with the solution's
    buffer as the right-hand side's, on both sides of the one-launch solve's
    range.  Two solutions with relative residuals of 1e-10 at kappa = 1e2 differ
    by at most 2 * 1e-10 * 1e2."""
    lib = _lib.load()
    A = matgen.spd_matrix(n, 1e2, n).cuda()
    if f64:
        A = A.double()
    B = matgen.rhs(n, nrhs, n + 1).cuda().reshape(n, nrhs).t().contiguous()    # column-major
    f = mp.factor(A.float(), block_size=128, precision="fp16")
    solve = lib.mpchol_pcg_f64 if f64 else lib.mpchol_pcg
    po, rep = _lib.default_pcg_opts(rel_tol=1e-10), _lib.Report()
    X = torch.empty_like(B)

    def call(b, x):
        return solve(f.handle, A.data_ptr(), n, b.data_ptr(), x.data_ptr(), nrhs, ctypes.byref(po),
                     ctypes.byref(rep), _stream())
    assert call(B, X) == _lib.OK
    bar = 2e-8 * X.norm().item()
    for _ in range(50):
        b = B.clone()
        assert call(b, b) == _lib.OK and rep.converged
        assert (b - X).norm().item() <= bar
    if f64:
        for _ in range(10):
            b = B.clone()
            assert lib.mpchol_adjoint_solve(f.handle, A.data_ptr(), n, X.data_ptr(), b.data_ptr(), b.data_ptr(),
                                            nrhs, None, n, ctypes.byref(po), ctypes.byref(rep),
                                            _stream()) == _lib.OK
            assert (b - X).norm().item() <= bar


@pytest.mark.parametrize("n", [512, 1000, 1100])
def test_the_drop_in_driver_solves_in_place(n):
    A = matgen.spd_matrix(n, 1e2, n).cuda().double()
    b = matgen.rhs(n, 1, n).cuda().reshape(n)
    x = torch.empty_like(b)
    args = dict(eps_prime=1e-3, rel_tol=1e-10)
    assert mp.precond_CG(A, x, b, n, 128, **args) == 0
    for _ in range(20):
        y = b.clone()
        assert mp.precond_CG(A, y, y, n, 128, **args) == 0
        assert (y - x).norm().item() <= 2e-8 * x.norm().item()


def _threads(*work):
    """Runs each function in a thread of its own; returns what they raised."""
    import threading
    raised = []

    def guard(fn):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                fn()
        except Exception as e:      # a thread's exception does not fail the test by itself
            raised.append(e)
    ts = [threading.Thread(target=guard, args=(fn,)) for fn in work]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    return raised


def test_small_solves_of_different_orders_in_threads():
    """One-launch solves of one number of right-hand sides need shared memory by
    their order: none may bound another thread's."""
    def solver(n, turns):
        A = matgen.spd_matrix(n, 1e2, n).cuda()
        B = matgen.rhs(n, 1, n).cuda().reshape(n)
        f = mp.factor(A, block_size=128, precision="fp16")
        torch.cuda.synchronize()

        def run():
            for _ in range(turns):
                _, rep = f.pcg(A, B, rel_tol=1e-10)
                assert rep.converged and rep.rel_residual <= 1e-10
        return run
    assert _threads(solver(1000, 300), solver(64, 600), solver(500, 400), solver(9, 600)) == []


_FIRST_SOLVES = """
import threading
import torch
import cholesky_gpu_b200 as mp
from cholesky_gpu_b200 import matgen
n = 1100
A = matgen.spd_matrix(n, 1e2, n).cuda()
fs = [mp.factor(A, block_size=128, precision="fp16") for _ in range(8)]
Bs = [matgen.rhs(n, k, k).cuda().reshape(n, k) for k in (1, 2, 4, 8) * 2]
torch.cuda.synchronize()
gate, done = threading.Barrier(8), []
def first(f, B):
    with torch.cuda.stream(torch.cuda.Stream()):
        gate.wait()
        X, rep = f.pcg(A, B, rel_tol=1e-10)
        assert rep.converged
        done.append(1)
ts = [threading.Thread(target=first, args=a) for a in zip(fs, Bs)]
[t.start() for t in ts]
[t.join() for t in ts]
assert len(done) == 8, len(done)
"""


def test_the_first_solves_of_a_process_in_threads():
    """A process whose first eight solves (each number of columns twice, general
    path) start together: what the launchers look up once per device is complete
    for every one of them."""
    import subprocess
    import sys
    from .conftest import ROOT
    for _ in range(3):
        r = subprocess.run([sys.executable, "-c", _FIRST_SOLVES], cwd=ROOT, capture_output=True, text=True,
                           timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]


def test_a_pointer_to_a_batch_factor_outlives_the_next_factor_call():
    """A pointer from mpchol_batch_lower is read on a stream of its own right
    after a second factor call on another one: it holds the second factor."""
    from cholesky_gpu_b200.api import _wrap_device
    ns = [2048, 300, 1500]
    As = [matgen.spd_matrix(n, 1e2, n).cuda() for n in ns]
    bt = mp.Batch(ns, block_size=128, precision="fp16x2")
    bt.factor([4.0 * A for A in As])
    p, ld, n = ctypes.c_void_p(), ctypes.c_int(), ctypes.c_int()
    assert _lib.load().mpchol_batch_lower(bt.handle, 0, ctypes.byref(p), ctypes.byref(ld),
                                          ctypes.byref(n)) == _lib.OK
    view = _wrap_device(p.value, (n.value, ld.value), torch.float32)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s1):
        bt.factor(As)
    with torch.cuda.stream(s2):
        got = view.clone()
    torch.cuda.synchronize()
    assert torch.equal(got[:, : n.value].t().tril(), bt.lower(0))
    L = torch.linalg.cholesky(As[0].double())
    assert ((bt.lower(0) - L).norm() / L.norm()).item() < 1e-5
