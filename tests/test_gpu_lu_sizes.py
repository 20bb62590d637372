"""The FP64 factorisation at the edges of its tiles, panels and thread counts: P A = L U against the product of the factors
it returns, the solve against the right-hand sides, and the batch kernels' independence of the thread count."""

import ctypes
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0**-53


def _lu(a):
    """Factors, pivots and status of column-major matrices a [n, N, N] (a[m].T is the matrix)."""
    import torch

    from dgamore_b200._lib import call

    p = lambda t: ctypes.c_void_p(t.data_ptr())
    n, N = a.shape[0], a.shape[1]
    lu = a.clone()
    piv = torch.empty((n, N), dtype=torch.int32, device="cuda")
    st = torch.zeros(n, dtype=torch.int32, device="cuda")
    call("dga_lu_batched_c128", p(lu), N, n, N * N, p(piv), p(st), ctypes.c_void_p(0))
    out = torch.empty((n, 16, N), dtype=a.dtype, device="cuda")
    k = min(16, N)
    call("dga_lu_solve_batched_c128", p(lu), p(piv), N, n, N * N, ctypes.c_void_p(0), 0, 0, 0, k, p(out), 16 * N, p(st),
         ctypes.c_void_p(0))
    torch.cuda.synchronize()
    return lu.cpu().numpy().transpose(0, 2, 1), piv.cpu().numpy(), st.cpu().numpy(), out.cpu().numpy()[:, :k]


@pytest.mark.parametrize("N", [1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 65, 96, 127, 129, 256, 257, 352, 353, 512, 513, 769, 1025])
@pytest.mark.parametrize("shift", [0.0, 3.0])
def test_factors_and_solves(N, shift):
    import torch

    g = torch.Generator(device="cuda").manual_seed(N)
    a = torch.randn((2, N, N), dtype=torch.complex128, device="cuda", generator=g)
    a += shift * torch.diag_embed(torch.randn((2, N), dtype=torch.complex128, device="cuda", generator=g))
    lu, piv, st, x = _lu(a)
    assert (st == 0).all()
    for m in range(2):
        mat = a[m].cpu().numpy().T
        L, U = np.tril(lu[m], -1) + np.eye(N), np.triu(lu[m])
        assert np.abs(L).max() <= np.sqrt(2) * (1 + 1e-9)  # |re| + |im| of a pivot is the column's largest
        perm = np.arange(N)
        for i, q in enumerate(piv[m]):
            perm[[i, q]] = perm[[q, i]]
        # backward error of an LU: a few N eps |L| |U|, elementwise (complex products: a factor of 4)
        bound = 8 * N * EPS * (np.abs(L) @ np.abs(U))
        assert (np.abs(mat[perm] - L @ U) <= bound + 1e-300).all()
        # A x = e_k to the same bound
        k = x.shape[1]
        res = mat @ x[m].T - np.eye(N)[:, :k]
        inv_perm = np.argsort(perm)
        bound = 24 * N * EPS * (np.abs(L) @ np.abs(U))[inv_perm] @ np.abs(x[m].T) + 8 * N * EPS
        assert (np.abs(res) <= bound).all()


def test_exact_ties_and_zeros():
    """A permutation matrix times constants of one modulus: ties take the first row, and a zero column is singular."""
    import torch

    N = 40
    a = torch.zeros((2, N, N), dtype=torch.complex128, device="cuda")
    a[0] = torch.triu(torch.ones((N, N), dtype=torch.complex128, device="cuda"))  # column-major: lower triangle of ones
    a[1] = torch.eye(N, dtype=torch.complex128, device="cuda")
    a[1, 17, 17] = 0.0
    lu, piv, st, _ = _lu(a)
    assert (piv[0] == np.arange(N)).all() and (piv[1] == np.arange(N)).all()
    assert st[0] == 0 and st[1] & 1


@pytest.mark.parametrize("niv", [(10, 20), (9, 33)])
def test_batch_does_not_depend_on_the_thread_count(niv):
    """A small problem next to a large one runs with the large one's thread count and gives the same bits."""
    from dgamore_b200 import synthetic
    from dgamore_b200.pipeline import LadderPass
    from dgamore_b200.serving import solve_bse_batch

    import torch

    cfgs = [dataclasses.replace(synthetic.CONFIGS["t1b"], niw=2, niv=niv[0]),
            dataclasses.replace(synthetic.CONFIGS["t2"], niw=2, niv=niv[1], niv_shell=0)]
    inps = [synthetic.make_inputs(c) for c in cfgs]
    alone, batch = [LadderPass(i) for i in inps], [LadderPass(i) for i in inps]
    for lp in alone:
        lp.pre_bse()
        lp.bse()
    for lp in batch:
        lp.pre_bse()
    solve_bse_batch(batch)
    torch.cuda.synchronize()
    for p, q in zip(alone, batch):
        assert torch.equal(p.X, q.X)
