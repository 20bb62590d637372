"""Back substitution of many right-hand sides on the tensor pipe where the last block of the matrix has one to eight rows
(one or two steps of the product over it): the dense solves and the pairing box's unit vectors."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0**-53


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _abs_lu(a):
    """|L| |U| in the rows of a (scipy's P L U)."""
    import scipy.linalg

    p, low, up = scipy.linalg.lu(a)
    return p @ (np.abs(low) @ np.abs(up))


# N % 32 = 1 .. 8, and 16, where no block is short; then both sides of the rule that gives 16 columns a CTA or a warp: N = 320
# (factors beyond L2, 16 columns) and 400, three CTAs an SM
@pytest.mark.parametrize("N,n,k", [(N, 300, N) for N in (33, 34, 35, 36, 37, 38, 39, 40, 65, 72, 200, 257, 16, 48)]
                         + [(320, 82, 16), (321, 82, 16), (321, 82, 17), (400, 28, 240), (401, 28, 240), (401, 30, 240),
                            (402, 1, 1), (416, 3, 33), (720, 21, 64), (1000, 1, 16)])
def test_dense_solve(N, n, k):
    import torch

    from dgamore_b200._lib import call

    cols = (k + 15) // 16 * 16
    g = torch.Generator(device="cuda").manual_seed(N)
    a = torch.randn((n, N, N), dtype=torch.complex128, device="cuda", generator=g)  # column-major: a[m].T
    lu, x = a.clone(), torch.full((n, cols, N), float("nan"), dtype=a.dtype, device="cuda")
    piv = torch.empty((n, N), dtype=torch.int32, device="cuda")
    st = torch.zeros(n, dtype=torch.int32, device="cuda")
    call("dga_lu_batched_c128", _p(lu), N, n, N * N, _p(piv), _p(st), ctypes.c_void_p(0))
    call("dga_lu_solve_batched_c128", _p(lu), _p(piv), N, n, N * N, ctypes.c_void_p(0), 0, 0, 0, k, _p(x), cols * N, _p(st),
         ctypes.c_void_p(0))
    assert int(st.abs().sum().item()) == 0
    mat, f, sol = a.transpose(1, 2), lu.transpose(1, 2), x[:, :k].transpose(1, 2)
    eye = torch.eye(N, dtype=a.dtype, device="cuda")
    blk = torch.arange(N, device="cuda") // 32
    diag = blk[:, None] == blk[None, :]
    low, up = torch.tril(f, -1) + eye, torch.triu(f)
    # the diagonal blocks D are multiplied by their inverses: a row block's residual is N eps |D| |D^-1| |D| |y|
    size = low.abs() @ up.abs()
    for t, side in ((low, 0), (up, 1)):
        d = t * diag
        e = t.abs() + d.abs() @ torch.linalg.inv(d).abs() @ d.abs()
        size = size + (low.abs() @ e if side else e @ up.abs())
    perm = torch.arange(N).repeat(n, 1).numpy()
    for m, pv in enumerate(piv.cpu().numpy()):
        for i, q in enumerate(pv):
            perm[m, [i, q]] = perm[m, [q, i]]
    perm = torch.from_numpy(perm).cuda()[:, :, None].expand(-1, -1, N)
    # factorisation, two substitutions and the residual itself, N eps each (complex products: a factor of 8), rows in pivot order
    res = torch.gather(mat, 1, perm) @ sol - torch.gather(eye.expand(n, N, N), 1, perm)[:, :, :k]
    size = size + torch.gather(mat, 1, perm).abs()
    assert (res.abs() <= 8 * N * EPS * (size @ sol.abs()) + 8 * N * EPS).all()


# N % 16 = 2 .. 8 up to N = 192, N % 32 = 2 .. 8 above
@pytest.mark.parametrize("n,niv,P,Q", [(1, 9, 9, 2), (1, 10, 4, 300), (1, 11, 3, 2), (1, 12, 5, 2), (1, 17, 8, 300),
                                       (1, 20, 10, 300), (1, 60, 30, 150), (1, 97, 20, 2), (1, 100, 50, 80), (1, 129, 7, 2),
                                       (2, 3, 3, 2), (2, 5, 2, 300), (2, 25, 6, 2), (3, 1, 1, 2), (3, 11, 5, 2), (3, 43, 3, 2),
                                       (4, 5, 2, 2)])
def test_pairing_box(n, niv, P, Q):
    import torch

    from dgamore_b200._lib import call, lib

    rng = np.random.default_rng(1000 * n + niv)
    n2, nv, W, w_pp, beta = n * n, 2 * niv, 3, 2, 2.0
    N, Mb, ib2 = n2 * nv, n2 * 2 * P, 0.25
    r = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    gamma, c0, uv = r(2, W, N, N), 0.1 * r(Q, W, nv, n2, n2), r(2, Q, n2, n2)
    c0 += (3.0 + rng.random((Q, W, nv, 1, 1))) * np.eye(n2)
    g3, chi = r(2, Q, W, nv, n2, n2), 0.1 * r(2, Q, W, n2, n2)
    work = np.array([(ch, q, w) for w in range(w_pp) for ch in range(2) for q in range(Q)], dtype=np.int32)
    n_items = len(work)
    dev = [torch.from_numpy(np.ascontiguousarray(t)).cuda() for t in (gamma.swapaxes(2, 3), c0, uv, g3, chi, work)]
    st = torch.zeros(n_items, dtype=torch.int32, device="cuda")
    sc = lambda b: torch.empty(int(b) // 16 + 1, dtype=torch.complex128, device="cuda")  # noqa: E731
    full = torch.full((2, Q, w_pp, Mb, Mb), float("nan"), dtype=torch.complex128, device="cuda")
    s1 = sc(lib().dga_eli_vertex_scratch_bytes(n, niv, P, n_items))
    call("dga_eli_full_vertex_c128", n, niv, W, Q, P, w_pp, beta, ib2, *[_p(t) for t in dev[:5]], _p(dev[5]), n_items,
         _p(full), _p(st), _p(s1), s1.numel() * 16, ctypes.c_void_p(0))
    assert int(st.abs().sum().item()) == 0
    fused = torch.full_like(full, float("nan"))
    X = torch.empty((2, Q, W, N, n2), dtype=torch.complex128, device="cuda")
    s2 = sc(lib().dga_bse_eli_scratch_bytes(N, n2, n_items))
    call("dga_bse_solve_sum_eli_c128", n, niv, W, Q, 2, beta, ib2, *[_p(t) for t in dev[:3]], _p(dev[5]), n_items, P, w_pp,
         _p(X), _p(fused), _p(st), _p(s2), s2.numel() * 16, ctypes.c_void_p(0))
    call("dga_eli_ladder_term_c128", _p(dev[2]), _p(dev[3]), _p(dev[4]), n, niv, W, Q, P, w_pp, _p(fused),
         ctypes.c_void_p(0))
    assert int(st.abs().sum().item()) == 0
    full, fused = full.cpu().numpy(), fused.cpu().numpy()
    assert np.isfinite(full).all() and np.isfinite(fused).all()
    box = slice(niv - P, niv + P)
    for it in sorted({0, 1, n_items // 3, n_items // 2, n_items - 2, n_items - 1}):
        ch, q, w = work[it]
        a = gamma[ch, w] * ib2 - np.repeat(np.repeat(uv[ch, q], nv, 0), nv, 1) * ib2
        for v in range(nv):
            a[v::nv, v::nv] += c0[q, w, v]
        inv = np.linalg.inv(a)
        star = inv.reshape(n2, nv, n2, nv)[:, box][..., box]  # [m, nu, m', nu']
        cb, gb = c0[q, w, box], g3[ch, q, w, box]
        ref = -np.einsum("apm,manb,bns->pasb", cb, star, cb)
        for v in range(2 * P):
            ref[:, v, :, v] += cb[v]
        z = uv[ch, q] - uv[ch, q] @ chi[ch, q, w] @ uv[ch, q]
        ladder = np.einsum("pm,amk,bks->pasb", z, gb, gb)
        ref = (beta**2 * ref + ladder).reshape(Mb, Mb)
        # the solve's error, |A^-1| (24 N eps |L| |U|) |A^-1| (numpy's own inverse: the same again), between two c0; then the
        # rounding of the products of n2 terms
        err = (np.abs(inv) @ (48 * N * EPS * _abs_lu(a)) @ np.abs(inv)).reshape(n2, nv, n2, nv)[:, box][..., box]
        bound = beta**2 * np.einsum("apm,manb,bns->pasb", np.abs(cb), err, np.abs(cb))
        size = beta**2 * np.einsum("apm,manb,bns->pasb", np.abs(cb), np.abs(star), np.abs(cb))
        zs = np.abs(uv[ch, q]) + np.abs(uv[ch, q]) @ np.abs(chi[ch, q, w]) @ np.abs(uv[ch, q])
        size += np.einsum("pm,amk,bks->pasb", zs, np.abs(gb), np.abs(gb)) + beta**2 * np.abs(cb).max()
        bound = (bound + 32 * (n2 + 1) * EPS * size).reshape(Mb, Mb)
        assert (np.abs(full[ch, q, w] - ref) <= bound).all()
        assert (np.abs(fused[ch, q, w] - ref) <= bound).all()
