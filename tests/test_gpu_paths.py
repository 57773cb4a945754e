"""Edges of the device paths that a size, an alignment or a format selects."""
import numpy as np
import pytest
import torch

import cholesky_gpu_b200 as mp
from cholesky_gpu_b200 import matgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,pad,offset", [
    (37, 0, 0), (130, 2, 0), (257, 3, 1), (256, 4, 4), (515, 5, 2), (1000, 0, 0), (999, 1, 3),
])
def test_operator_copy_is_exact_for_every_alignment(n, pad, offset):
    """The copy of A's lower block columns (16-byte path, or scalar for columns
    that start elsewhere) gives the same factor bit for bit wherever A lies."""
    A = matgen.spd_matrix(n, 1e2, n).cuda()
    ref = mp.factor(A, block_size=128, precision="fp32").lower()
    lda = n + pad
    store = torch.full((n * lda + offset,), float("nan"), device="cuda")
    view = store[offset:].as_strided((n, n), (1, lda))      # column-major, leading dimension lda
    view.copy_(A)
    got = mp.factor(view, block_size=128, precision="fp32").lower()
    assert torch.equal(got, ref)
    L = np.linalg.cholesky(A.double().cpu().numpy())
    assert np.linalg.norm(got.cpu().numpy() - L) / np.linalg.norm(L) < 1e-5


def test_resources_of_a_freed_factor_serve_the_next_one():
    """Objects made and freed in turn (with other sizes between, in threads on
    streams of their own, after the cache was given back) factor as a lone one."""
    import threading
    from cholesky_gpu_b200 import _lib
    sizes = (200, 900, 513, 900)
    mats = {n: matgen.spd_matrix(n, 1e2, n).cuda() for n in set(sizes)}
    opts = dict(block_size=128, precision="fp16x2")
    _lib.load().mpchol_release_cached()
    ref = {n: mp.factor(A, **opts).lower() for n, A in mats.items()}
    torch.cuda.synchronize()
    bad = []

    def work(order):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for n in order:
                    f = mp.factor(mats[n], **opts)
                    if not torch.equal(f.lower(), ref[n]):
                        bad.append(n)
                    del f
        except Exception as e:      # a thread's exception does not fail the test by itself
            bad.append(e)
    threads = [threading.Thread(target=work, args=(o,)) for o in (sizes, sizes[::-1], sizes * 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    _lib.load().mpchol_release_cached()
    work(sizes)
    assert not bad


@pytest.mark.parametrize("n", [31, 33, 96, 128, 129, 191, 161, 193, 225, 289, 385, 545, 640, 1023, 1025, 1500])
def test_preconditioner_apply_at_block_and_super_block_edges(n):
    """z = M^-1 r through the block and super-block inverses against the FP64
    solve with the factor itself.  The inverses are exact to FP32 rounding:
    kappa(L) = 10, so 1e-5 leaves two digits."""
    A = matgen.spd_matrix(n, 1e2, n).cuda()
    f = mp.factor(A, block_size=128, precision="fp32")
    L = f.lower().double()
    R = matgen.rhs(n, 3, 5).cuda()
    Z = f.apply_precond(R)
    ref = torch.cholesky_solve(R, L)
    assert ((Z - ref).norm() / ref.norm()).item() < 1e-5


@pytest.mark.parametrize("n,nrhs", [(1025, 1), (2049, 2), (2200, 1), (3333, 1), (3200, 2), (3100, 4), (4097, 8),
                                    (9728, 1), (9601, 2)])
def test_triangular_solves_over_many_super_blocks(n, nrhs):
    """The persistent solve for each number of right-hand sides, with partial
    super-blocks and both grids, twice in a row (its slots are used again)
    against FP64.  A diagonally dominant A keeps kappa(L) below 2: the FP32
    inverses leave 1e-6, the bound has another digit."""
    g = torch.Generator().manual_seed(n)
    A = (torch.rand(n, n, generator=g) - 0.5).cuda()
    A = A + A.T
    A.diagonal().add_(2.0 * n)
    f = mp.factor(A, block_size=256, precision="fp32")
    L = f.lower().double()
    for seed in (1, 2):
        R = matgen.rhs(n, nrhs, seed).cuda()
        ref = torch.cholesky_solve(R.reshape(n, -1), L).reshape(R.shape)
        Z = f.apply_precond(R)
        assert ((Z - ref).norm() / ref.norm()).item() < 1e-5


@pytest.mark.parametrize("n,d,lower", [
    (1, 3, False), (63, 16, True), (65, 17, False), (2047, 15, True), (2305, 33, True),
])
def test_rbf_build_at_tile_edges(n, d, lower):
    """Both tile heights of the builder, ragged in rows and features: 1e-13 of
    the FP64 kernel (64 differences of FP32 values squared in FP64: d * 2^-53
    relative in the exponent, which is below 30 here), zeros above a lower build."""
    from cholesky_gpu_b200.autograd import rbf_build
    from oracle import oracle as O
    X = matgen.gaussian_points(n, d, n)
    K64, K32 = rbf_build(torch.from_numpy(X).cuda(), 2.0, 0.25, lower_only=lower)
    want, _ = O.rbf_kernel_f64(X, 2.0, 0.25)
    if lower:
        want = np.tril(want)
    got = K64.cpu().numpy()
    assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()
    assert np.array_equal(K32.cpu().numpy(), got.astype(np.float32))


@pytest.mark.parametrize("n,d", [(1, 1), (17, 128), (130, 9), (3199, 3), (3201, 8), (6401, 7), (6465, 120)])
def test_rbf_grad_contraction_at_row_tile_edges(n, d):
    """The 16-, 32- and 64-row variants against dense FP64: sums of n terms,
    relative error of a norm below 1e-13."""
    from cholesky_gpu_b200.autograd import rbf_grad_contract
    g = torch.Generator(device="cuda").manual_seed(n)
    X = torch.randn((n, d), generator=g, device="cuda")
    a, b = (torch.randn(n, generator=g, device="cuda", dtype=torch.float64) for _ in range(2))
    ell = float(d) ** 0.5
    P, s = rbf_grad_contract(X, ell, a, b)
    Xd = X.double()
    r2 = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    for k in range(d):
        r2 += (Xd[:, k].unsqueeze(1) - Xd[:, k].unsqueeze(0)) ** 2
    K = torch.exp(-r2 / (2 * ell * ell))
    Z = torch.cat([a.unsqueeze(1), b.unsqueeze(1), a.unsqueeze(1) * Xd, b.unsqueeze(1) * Xd], 1)
    want = K @ Z
    assert ((P - want).norm() / want.norm()).item() < 1e-13
    ws = (a @ ((K * r2) @ b)).item()
    scale = (a.abs() @ ((K * r2) @ b.abs())).item()
    assert abs(s.item() - ws) <= 1e-13 * max(scale, 1e-300)


@pytest.mark.parametrize("n", [1, 8, 31, 32, 40, 63, 64, 95, 128, 160, 200, 224, 255, 256])
def test_diagonal_factor_at_tile_edges(n):
    """One diagonal block of every tile count, ragged and whole, against FP64
    (kappa = 1e2: FP32 Cholesky is within n * 2^-24 * kappa^0.5 of it), with
    pivots that need no repair."""
    A = matgen.spd_matrix(n, 1e2, 3 * n) if n > 1 else torch.full((1, 1), 4.0)
    f = mp.factor(A.cuda(), block_size=256, precision="fp32")
    assert f.info().n_perturbed == 0
    L = np.linalg.cholesky(A.double().numpy())
    assert np.linalg.norm(f.lower().cpu().numpy() - L) / np.linalg.norm(L) < 1e-5


@pytest.mark.parametrize("row,value", [(0, -1.0), (7, 0.0), (8, 1e-40), (37, -2.0), (100, float("nan")),
                                       (255, float("inf"))])
def test_diagonal_factor_takes_the_full_pivot_rule_for_rare_pivots(row, value):
    """A pivot at or below its floor is repaired to max(|pivot|, floor) and
    counted; one that is not finite fails at its row.  The matrix is diagonal,
    so every pivot is known exactly."""
    d = torch.linspace(1.0, 2.0, 256)
    d[row] = value
    f = mp.factor(torch.diag(d).cuda(), block_size=256, precision="fp32", pert=0.0)
    info = f.info()
    if not np.isfinite(value) or value == 0.0:
        # a zero pivot's floor is zero here: the row below receives 0 / sqrt(0)
        # and fails
        assert info.status != 0 and info.fail_row == row + (value == 0.0)
        return
    assert info.status == 0 and info.n_perturbed == (0 if value > 0 else 1)
    stored = d.double().numpy()
    want = np.sqrt(np.where(np.arange(256) == row, np.maximum(np.abs(stored), 1e-7 * stored), stored))
    got = torch.diagonal(f.lower()).cpu().numpy()
    assert np.allclose(got, want, rtol=1e-6, atol=0.0)


@pytest.mark.parametrize("m,k,pad", [(1, 32, 0), (33, 64, 3), (127, 40, 0), (128, 256, 1), (129, 96, 4),
                                     (640, 256, 0), (1920, 17, 0), (2049, 32, 3), (2300, 256, 0)])
def test_fp32_trailing_update_sizes(m, k, pad):
    """Every kernel of the FP32 update (32-tiles, 128-tiles), ragged sizes and
    unaligned panels, against FP64: sums of k products of N(0,1) values in
    FP32, relative error of the update's norm below k * 2^-24."""
    import ctypes  # noqa: F401
    from cholesky_gpu_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(m + k)
    ld = m + pad
    P = torch.randn((k, ld), generator=g, device="cuda")       # column-major m x k, stride ld
    C = torch.randn((m, ld), generator=g, device="cuda")
    before = C.clone()
    _lib.check(_lib.load().mpchol_syrk_update(C.data_ptr(), ld, m, k, _lib.PREC_FP32, None, None,
                                              P.data_ptr(), ld, torch.cuda.current_stream().cuda_stream))
    Pd = P[:, :m].double().t()
    want = Pd @ Pd.t()
    got = (before - C)[:, :m].t().double()
    low = torch.ones((m, m), dtype=torch.bool, device="cuda").tril()
    assert ((got - want)[low].norm() / want[low].norm()).item() < max(k, 8) * 2.0 ** -24 + 2.0 ** -23
    C2 = C.clone()
    C2[:, :m].t()[low] = before[:, :m].t()[low]
    assert torch.equal(C2, before)                              # nothing else is touched


@pytest.mark.parametrize("n,nrhs,f64", [(1, 1, False), (7, 3, False), (8, 1, True), (129, 8, False),
                                        (511, 2, True), (513, 5, False), (1000, 1, False), (1017, 4, True),
                                        (1024, 8, False), (1024, 1, True), (1024, 8, True), (1025, 2, False)])
def test_small_solves_match_the_dense_solve(n, nrhs, f64):
    """The one-launch solve at the edges of its range (and the sizes that fall
    to the general path): iterations as for a general-path order, residual at
    the tolerance, solution within kappa * tolerance of the FP64 dense solve."""
    A = matgen.spd_matrix(n, 1e3, n).cuda() if n > 1 else torch.full((1, 1), 2.0, device="cuda")
    B = matgen.rhs(n, nrhs, n + 1).cuda().reshape(n, -1)
    f = mp.factor(A, block_size=128, precision="fp16")
    Ad = A.double()
    for x0 in (True, False):
        X, rep = f.pcg(Ad if f64 else A, B, rel_tol=1e-11, x0_precond=x0)
        assert rep.converged and rep.rel_residual <= 1e-11
        true = ((B - Ad @ X).norm(dim=0) / B.norm(dim=0)).max().item()
        assert true <= 2e-11
        ref = torch.linalg.solve(Ad, B)
        assert ((X - ref).norm() / ref.norm()).item() <= 1e-8
        fro, xn = Ad.norm().item(), X.norm(dim=0)
        be = ((B - Ad @ X).norm(dim=0) / (fro * xn + B.norm(dim=0))).max().item()
        assert abs(rep.backward_error - be) <= 0.5 * be + 1e-15


def test_small_solve_stops_at_its_iteration_budget_and_reports_failures():
    n = 300
    A = matgen.spd_matrix(n, 1e4, 3).cuda()
    B = matgen.rhs(n, 2, 4).cuda()
    f = mp.factor(A, block_size=128, precision="fp16")
    for budget in (0, 1, 3):
        X, rep = f.pcg(A, B, rel_tol=1e-14, max_it=budget)
        assert rep.iterations == budget and not rep.converged
    bad = -A
    with pytest.raises(mp.MpcholError) as e:
        mp.factor(bad, block_size=128, precision="fp16", diag_pert=0).pcg(A, B)
    assert e.value.status == 2
    with pytest.raises(mp.MpcholError) as e:      # an indefinite operator: p^T A p < 0
        f.pcg(bad, B)
    assert e.value.status == 6


@pytest.mark.parametrize("n,opts", [(300, {}), (1300, dict(block_size=128, precision="fp32"))])
def test_rbf_solve_reads_lower_triangles_only(n, opts):
    """The kernel matrices of a differentiable solve come from uncleared memory:
    with NaN in the blocks that the allocator hands out next, the solution and
    the gradients are those of a solve on zeroed blocks.  Tolerance: two PCG
    solves to 1e-11 at kappa below 1e4."""
    from cholesky_gpu_b200 import rbf_solve
    g = torch.Generator().manual_seed(n)
    X = torch.randn(n, 3, generator=g).cuda()
    y = torch.randn(n, generator=g, dtype=torch.float64).cuda()

    def run(fill):
        torch.cuda.empty_cache()
        held = [torch.full((n, n), fill, dtype=t, device="cuda") for t in (torch.float64, torch.float32)]
        torch.cuda.synchronize()
        del held
        Xr = X.clone().requires_grad_(True)
        x = rbf_solve(Xr, 1.0, 0.5, y, rel_tol=1e-11, **opts)
        (gX,) = torch.autograd.grad((x * y).sum(), Xr)
        return x.detach(), gX

    (x0, g0), (x1, g1) = run(0.0), run(float("nan"))
    assert ((x1 - x0).norm() / x0.norm()).item() < 1e-6
    assert ((g1 - g0).norm() / g0.norm()).item() < 1e-6


@pytest.mark.parametrize("precision,block", [("fp16x2", 128), ("fp16", 64)])
def test_batch_calls_on_different_streams(precision, block):
    """The factor call returns before the factors are complete: a second factor
    call, the status and the solve on other streams wait for it.  Orders at tile
    edges, one of two super-blocks; the true residual is FP64."""
    ns = [64, 1, 33, 130, 1100, 257]
    As = [matgen.spd_matrix(n, 1e2, n).cuda() if n > 1 else torch.full((1, 1), 3.0, device="cuda") for n in ns]
    other = [2.0 * A for A in As]
    Bs = [matgen.rhs(n, 2, n).cuda().reshape(n, 2) for n in ns]
    bt = mp.Batch(ns, nrhs=2, block_size=block, precision=precision)
    torch.cuda.synchronize()
    s1, s2, s3 = (torch.cuda.Stream() for _ in range(3))
    with torch.cuda.stream(s1):
        bt.factor(other)
    with torch.cuda.stream(s2):
        bt.factor(As)
    with torch.cuda.stream(s3):
        assert bt.info()[0] == [0] * len(ns)
        Xs, reps, _ = bt.pcg(As, Bs, rel_tol=1e-10)
    torch.cuda.synchronize()
    for A, B, X, r in zip(As, Bs, Xs, reps):
        assert r.converged
        S = torch.tril(A.double()) + torch.tril(A.double(), -1).T
        assert ((S @ X - B).norm() / B.norm()).item() < 2e-10


@pytest.mark.parametrize("n,pad", [(127, 0), (125, 2), (128, 1)])
def test_eight_column_products_of_unaligned_columns_sum_in_short_chains(n, pad):
    """A matrix of ones times vectors of one 1 among numbers t = 2^-56.  A partial
    sum that holds the 1 loses each t (or four of them) added after it, so the
    result shows how many terms share a chain: at most 16 here, and two
    roundings to 2^-53 where the parts meet."""
    from cholesky_gpu_b200 import _lib
    ld = n + pad
    A = torch.ones((n, ld), device="cuda")
    t = 2.0 ** -56
    X = torch.full((8, n), t, device="cuda", dtype=torch.float64)
    for k in range(8):
        X[k, (k * n) // 8] = 1.0
    Y = torch.empty_like(X)
    _lib.check(_lib.load().mpchol_symv(A.data_ptr(), ld, n, X.data_ptr(), Y.data_ptr(), 8,
                                       torch.cuda.current_stream().cuda_stream))
    lost = (n - 1) * t - (Y - 1.0)          # Y - 1 is exact; below 2^-46
    assert lost.abs().max().item() <= 16 * t + 2 * 2.0 ** -53
