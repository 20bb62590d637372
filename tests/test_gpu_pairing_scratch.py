"""Scratch of the pass with the pairing box: what the box's columns take, and not N columns whatever the box."""

import ctypes

import pytest

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("n,niv,P", [(1, 20, 1), (1, 20, 10), (1, 20, 20), (2, 15, 3), (3, 8, 4)])
def test_scratch_follows_the_box(n, niv, P):
    import torch

    from dgamore_b200._lib import DgaError, call, lib

    n2, nv, W, w_pp, Q = n * n, 2 * niv, 2, 2, 40
    N, Mb, n_items = n2 * nv, n2 * 2 * P, 2 * Q * w_pp
    g = torch.Generator(device="cuda").manual_seed(niv)
    r = lambda *s: torch.randn(s, dtype=torch.complex128, device="cuda", generator=g)  # noqa: E731
    gamma, uv = r(2, W, N, N), r(2, Q, n2, n2)
    c0 = 0.1 * r(Q, W, nv, n2, n2) + 4.0 * torch.eye(n2, dtype=torch.complex128, device="cuda")
    work = torch.tensor([(ch, q, w) for w in range(w_pp) for ch in range(2) for q in range(Q)], dtype=torch.int32, device="cuda")
    st = torch.zeros(n_items, dtype=torch.int32, device="cuda")
    need = int(lib().dga_bse_eli_box_scratch_bytes(N, n2, P, n_items))
    # fewer items than resident CTAs: one matrix, its selectors and the box's columns each
    assert need == n_items * N * (N + n2 + Mb) * 16
    assert need <= int(lib().dga_bse_eli_scratch_bytes(N, n2, n_items)) == n_items * N * (2 * N + n2) * 16

    def run(scratch_bytes):
        X = torch.zeros((2, Q, W, N, n2), dtype=torch.complex128, device="cuda")
        f = torch.zeros((2, Q, w_pp, Mb, Mb), dtype=torch.complex128, device="cuda")
        sc = torch.empty(scratch_bytes // 16, dtype=torch.complex128, device="cuda")
        call("dga_bse_solve_sum_eli_c128", n, niv, W, Q, 2, 2.0, 0.25, _p(gamma), _p(c0), _p(uv), _p(work), n_items, P, w_pp,
             _p(X), _p(f), _p(st), _p(sc), sc.numel() * 16, ctypes.c_void_p(0))
        torch.cuda.synchronize()
        assert int(st.abs().sum().item()) == 0
        return X, f

    small, large = run(need), run(int(lib().dga_bse_eli_scratch_bytes(N, n2, n_items)))
    assert torch.equal(small[0], large[0]) and torch.equal(small[1], large[1])
    with pytest.raises(DgaError):
        run(need - 16)
