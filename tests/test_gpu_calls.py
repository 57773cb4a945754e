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
    lib = _lib.load()

    def solver(n):
        A, B = matgen.spd_matrix(n, 1e2, n).cuda(), matgen.rhs(n, 1, n).cuda().reshape(n)
        X, f, side = torch.empty_like(B), mp.factor(A, block_size=128, precision="fp16"), torch.cuda.Stream()
        po, rep = _lib.default_pcg_opts(rel_tol=1e-10), _lib.Report()
        short = _lib.default_pcg_opts(rel_tol=1e-10, max_it=0, x0_precond=0)
        torch.cuda.synchronize()

        def call(o):
            return lib.mpchol_pcg(f.handle, A.data_ptr(), n, B.data_ptr(), X.data_ptr(), 1, ctypes.byref(o),
                                  ctypes.byref(rep), side.cuda_stream)

        def run():
            for _ in range(5000):                    # the launches are what meets
                st = call(short)
                assert st == _lib.PCG_MAXIT, (n, st)
            assert call(po) == _lib.OK and rep.rel_residual <= 1e-10
        return run
    assert _threads(solver(1000), solver(64), solver(500), solver(9)) == []


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


def _solved(f, A, B):
    f.compute(A)
    X, rep = f.pcg(A, B, rel_tol=1e-10)
    assert rep.converged
    return X


def test_dropping_a_factor_leaves_a_capture_in_another_thread_alone():
    """A factor object destroyed by one thread while another captures a graph in
    the thread-local mode: the capture ends well and its graph runs."""
    import threading
    n = 700
    A, B = matgen.spd_matrix(n, 1e2, n).cuda(), matgen.rhs(n, 1, n).cuda().reshape(n)
    held = [mp.Factor(n, block_size=128, precision="fp16") for _ in range(2)]
    for f in held:
        _solved(f, A, B)
    del f
    x, y = torch.ones(1000, device="cuda"), torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        y.copy_(x)
        t = threading.Thread(target=held.clear)
        t.start()
        t.join()
        y.add_(x)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, 2 * x)
    X = _solved(mp.Factor(n, block_size=128, precision="fp16"), A, B)     # no error is left behind
    assert ((A.double() @ X - B).norm() / B.norm()).item() < 2e-10


def test_factors_come_and_go_while_others_capture():
    """One thread makes and drops factor objects while two others make batches
    and factor objects that capture their graphs: every call succeeds."""
    ns = [300, 64, 700]
    As = [matgen.spd_matrix(n, 1e2, n).cuda() for n in ns]
    Bs = [matgen.rhs(n, 1, n).cuda().reshape(n) for n in ns]
    big, rhs = matgen.spd_matrix(1300, 1e2, 5).cuda(), matgen.rhs(1300, 1, 5).cuda().reshape(1300)
    torch.cuda.synchronize()

    def drops():
        for i in range(200):
            _solved(mp.Factor(ns[i % 3], block_size=128, precision="fp16"), As[i % 3], Bs[i % 3])

    def batches():
        for _ in range(15):
            bt = mp.Batch(ns, nrhs=1, block_size=128, precision="fp16")
            bt.factor(As)
            Xs, reps, st = bt.pcg(As, Bs, rel_tol=1e-10)
            assert st == _lib.OK and all(r.converged for r in reps)

    def graphs():
        for _ in range(15):
            f = mp.Factor(1300, block_size=128, precision="fp16")
            for _ in range(4):                       # the factor's graph, then the loop's
                _solved(f, big, rhs)
    assert _threads(drops, batches, graphs) == []


def test_memory_is_not_reused_before_its_last_reader():
    """The memory of a freed object serves the next one only after what still
    used it: the caller's copy through a pointer, and a factorization still
    waiting on another stream."""
    from cholesky_gpu_b200.api import _wrap_device
    n = 640
    opts = dict(block_size=128, precision="fp32")
    A1, A2 = matgen.spd_matrix(n, 1e2, 1).cuda(), 9.0 * matgen.spd_matrix(n, 1e2, 2).cuda()
    L1, L2 = mp.factor(A1, **opts).lower(), mp.factor(A2, **opts).lower()
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    f = mp.factor(A1, **opts)
    p = ctypes.c_void_p()
    assert _lib.load().mpchol_factor_lower(f.handle, ctypes.byref(p), None, None) == _lib.OK
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(40_000_000)
        got = _wrap_device(p.value, (n, n), torch.float32).clone()
        del f
    with torch.cuda.stream(other):
        h = mp.factor(A2, **opts)
    torch.cuda.synchronize()
    assert torch.equal(got.t().tril(), L1) and torch.equal(h.lower(), L2)
    del h
    for _ in range(3):
        with torch.cuda.stream(side):
            torch.cuda._sleep(40_000_000)
            f = mp.factor(A1, **opts)                # enqueued behind the wait
            del f
        with torch.cuda.stream(other):
            h = mp.factor(A2, **opts)
        torch.cuda.synchronize()
        assert torch.equal(h.lower(), L2)


def test_freed_memory_serves_the_next_solves_in_threads():
    """Objects that give out no pointer, made and freed in turn in three threads:
    each solve is that of a lone object."""
    ns = (200, 900, 513, 1100)
    mats = {n: (matgen.spd_matrix(n, 1e2, n).cuda(), matgen.rhs(n, 1, n).cuda().reshape(n)) for n in ns}
    torch.cuda.synchronize()

    def worker(order):
        def run():
            for n in order * 6:
                A, B = mats[n]
                X = _solved(mp.Factor(n, block_size=128, precision="fp16x2"), A, B)
                assert ((A.double() @ X - B).norm() / B.norm()).item() < 2e-10
        return run
    assert _threads(worker(ns), worker(ns[::-1]), worker((900, 200))) == []


def test_batches_of_different_blocks_in_threads():
    """Batches whose block sizes ask for different amounts of shared memory are
    made, factored and solved at the same time."""
    ns = [200, 64, 400]
    As = [matgen.spd_matrix(n, 1e2, n).cuda() for n in ns]
    Bs = [matgen.rhs(n, 1, n).cuda().reshape(n) for n in ns]
    torch.cuda.synchronize()

    def batches(block):
        def run():
            for _ in range(25):
                bt = mp.Batch(ns, nrhs=1, block_size=block, precision="fp16")
                bt.factor(As)                        # the launches are captured here
                assert bt.pcg(As, Bs, rel_tol=1e-10)[2] == _lib.OK
        return run
    assert _threads(batches(192), batches(64), batches(256), batches(128)) == []


@pytest.mark.parametrize("n,block", [(1, 128), (31, 128), (33, 256), (127, 128), (257, 128), (514, 256)])
def test_the_drop_in_factorization_leaves_the_upper_triangle_alone(n, block):
    """switching_chol writes L into the lower triangle of its column-major matrix
    and nothing else, whatever the memory that the library works in held before
    (a larger system's solve and factor)."""
    big = matgen.spd_matrix(600, 1e2, 1).cuda()
    _solved(mp.Factor(600, block_size=128, precision="fp16"), big, matgen.rhs(600, 1, 1).cuda().reshape(600))
    A = matgen.spd_matrix(n, 1e2, n).cuda() if n > 1 else torch.full((1, 1), 4.0, device="cuda")
    store = A.clone()                                # row j of the storage is column j
    above = torch.ones((n, n), dtype=torch.bool, device="cuda").tril(-1)   # of the storage: i < j
    store[above] = torch.arange(int(above.sum()), device="cuda", dtype=torch.float32) + 1000.0
    before = store.clone()
    d, dt = torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
    assert mp.switching_chol(store, n, block, d, dt, 1e-3) == 0
    assert torch.equal(store[above], before[above])
    L = torch.linalg.cholesky(A.double())
    got = store.t().tril().double()
    assert ((got - L).norm() / L.norm()).item() < 1e-3
    assert torch.equal(d, torch.diagonal(A))
