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


@pytest.mark.parametrize("n", [31, 33, 96, 128, 129, 191, 385, 640, 1023, 1025, 1500])
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
