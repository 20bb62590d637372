"""Pivot search of the FP64 factorisation at every thread count: LAPACK's order to the last bit, values without an order (NaN,
infinity), pivots far from one, and the error of the division by a pivot."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0**-53
SINGULAR, NONFINITE = 1, 2


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _factor(a):
    """Factors (column-major, as a), pivots and status of the matrices a[m].T."""
    import torch

    from dgamore_b200._lib import call

    n, N = a.shape[0], a.shape[1]
    lu = a.clone()
    piv = torch.empty((n, N), dtype=torch.int32, device="cuda")
    st = torch.zeros(n, dtype=torch.int32, device="cuda")
    call("dga_lu_batched_c128", _p(lu), N, n, N * N, _p(piv), _p(st), ctypes.c_void_p(0))
    torch.cuda.synchronize()
    return lu, piv, st


def _matrices(N):
    """More matrices than would leave half of the SMs' threads idle: the thread count is the one of N alone."""
    import torch

    threads = 32 if N <= 64 else 64 if N <= 192 else 128 if N <= 512 else 256
    return torch.cuda.get_device_properties(0).multi_processor_count * 256 // threads + 1


# both sides of each thread count's range, of its rows per thread (1, 2, 4, 8) and of the block width (N = 192)
@pytest.mark.parametrize("N", [33, 40, 64, 65, 128, 129, 191, 192, 193, 256, 257, 511, 512, 513])
def test_thread_counts(N):
    """The first column's entries agree to 2^-43: the largest, at a place of its own in each matrix, is the pivot."""
    import scipy.linalg
    import torch

    n = _matrices(N)
    g = torch.Generator(device="cuda").manual_seed(N)
    a = torch.randn((n, N, N), dtype=torch.complex128, device="cuda", generator=g)
    rank = torch.argsort(torch.rand((n, N), device="cuda", generator=g), dim=1)
    a[:, 0] = 1.0 + rank.to(torch.float64) * 2.0**-52
    lu, piv, st = _factor(a)
    assert int(st.abs().sum().item()) == 0
    assert torch.equal(piv[:, 0].long(), rank.argmax(dim=1))
    for m in (0, n // 2, n - 1):
        assert (scipy.linalg.lu_factor(a[m].T.cpu().numpy())[1] == piv[m].cpu().numpy()).all()
    few = _factor(a[:2])  # the same bits with the most threads a matrix can have
    assert torch.equal(few[0], lu[:2]) and torch.equal(few[1], piv[:2])
    perm = np.tile(np.arange(N), (n, 1))
    rows = np.arange(n)
    for i, q in enumerate(piv.cpu().numpy().T):
        perm[rows, i], perm[rows, q] = perm[rows, q], perm[rows, i]
    perm = torch.from_numpy(perm).cuda()
    for m0 in range(0, n, 256):  # P A = L U to N eps |L| |U| (complex products, and the check's own: a factor of 8)
        m1 = min(n, m0 + 256)
        f = lu[m0:m1].transpose(1, 2)
        low = torch.tril(f, -1) + torch.eye(N, dtype=a.dtype, device="cuda")
        up = torch.triu(f)
        rows_in_order = torch.gather(a[m0:m1].transpose(1, 2), 1, perm[m0:m1, :, None].expand(-1, -1, N))
        assert ((rows_in_order - low @ up).abs() <= 8 * N * EPS * (low.abs() @ up.abs())).all()


@pytest.mark.parametrize("N", [40, 120, 300, 600])
def test_equal_entries_take_the_first_row(N):
    """Columns whose entries all have one modulus (a Vandermonde matrix of the fourth roots of one, then random columns)."""
    import torch

    n = 3
    g = torch.Generator(device="cuda").manual_seed(N)
    a = torch.randn((n, N, N), dtype=torch.complex128, device="cuda", generator=g)
    k = torch.randint(0, 4, (n, N), device="cuda", generator=g)
    a[:, 0] = torch.tensor([1, 1j, -1, -1j], dtype=a.dtype, device="cuda")[k]
    a[1, 0, : N // 2] *= 0.5  # the first half is smaller: the first of the second half
    _, piv, st = _factor(a)
    assert int(st.abs().sum().item()) == 0
    assert piv[:, 0].tolist() == [0, N // 2, 0]


@pytest.mark.parametrize("N", [40, 120, 300, 600])
def test_values_without_an_order(N):
    """A column of NaN keeps its diagonal row and an infinity is the largest entry; a NaN ends as NONFINITE, and the other
    matrices of the batch are as they are alone."""
    import torch

    from dgamore_b200._lib import call

    n = 5
    g = torch.Generator(device="cuda").manual_seed(N)
    a = torch.randn((n, N, N), dtype=torch.complex128, device="cuda", generator=g)
    a[1, 7] = float("nan")
    a[2, 0, N - 2] = float("inf")
    a[3, N - 1, 5] = float("nan")
    good = [0, 4]
    ref, ref_piv, _ = _factor(a[good])
    lu, piv, st = _factor(a)
    assert torch.equal(lu[good], ref) and torch.equal(piv[good], ref_piv)
    assert piv[1, 7].item() == 7 and piv[2, 0].item() == N - 2
    assert ((piv >= torch.arange(N, device="cuda")) & (piv < N)).all()
    x = torch.empty((n, 16, N), dtype=a.dtype, device="cuda")
    call("dga_lu_solve_batched_c128", _p(lu), _p(piv), N, n, N * N, ctypes.c_void_p(0), 0, 0, 0, 16, _p(x), 16 * N, _p(st),
         ctypes.c_void_p(0))
    assert [st[m].item() & NONFINITE for m in (0, 1, 3, 4)] == [0, 2, 2, 0]
    assert not any(s & SINGULAR for s in st.tolist())


@pytest.mark.parametrize("N", [40, 120, 300])
@pytest.mark.parametrize("power", [59, 62, 80, 300])
def test_pivots_far_from_one(N, power):
    """Columns scaled by powers of two on both sides of the range that the short division takes (2^-60 .. 2^60): the pivots do
    not change, U's columns are scaled, and the factors stay within the backward error of an LU."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(N)
    a = torch.randn((2, N, N), dtype=torch.complex128, device="cuda", generator=g)
    e = torch.tensor([2.0**power, 2.0**-power, 1.0, 2.0 ** (power // 2)], dtype=torch.float64, device="cuda")
    scale = e[torch.arange(N, device="cuda") % 4]
    _, piv0, _ = _factor(a)
    lu, piv, st = _factor(a * scale[None, :, None])
    assert int(st.abs().sum().item()) == 0 and torch.equal(piv, piv0)
    for m in range(2):
        mat, f = a[m].T.cpu().numpy(), lu[m].T.cpu().numpy() / scale.cpu().numpy()[None, :]
        low = np.tril(lu[m].T.cpu().numpy(), -1) + np.eye(N)
        up = np.triu(f)
        perm = np.arange(N)
        for i, q in enumerate(piv[m].tolist()):
            perm[[i, q]] = perm[[q, i]]
        assert (np.abs(mat[perm] - low @ up) <= 8 * N * EPS * (np.abs(low) @ np.abs(up))).all()


@pytest.mark.parametrize("power", [0, 58, 61, 200])
def test_division_by_a_pivot(power):
    """L(2, 1) = a / d of 2 x 2 matrices against the quotient in extended precision. With u = 2^-53: |d|^2 to 2 u, its
    reciprocal to 1.5 u more, a conj(d) to sqrt(5) u and the scaling to u, or Smith's reciprocal to 5 u and the product:
    below 8 u either way."""
    import torch

    n = 50000
    rng = np.random.default_rng(power)
    z = lambda: (rng.standard_normal(n) + 1j * rng.standard_normal(n)) * 2.0 ** rng.uniform(-3, 3, n)  # noqa: E731
    d, x = z(), z()
    d[::7] = d[::7].real
    d[1::7] = 1j * d[1::7].imag
    s = np.where(np.arange(n) % 2, 2.0**power, 2.0**-power)
    d, x = d * s, x * s
    a = np.zeros((n, 2, 2), dtype=np.complex128)  # column-major
    a[:, 0, 0], a[:, 0, 1], a[:, 1, 0], a[:, 1, 1] = d, x, 1.0, 1.0
    lu, piv, _ = _factor(torch.from_numpy(a).cuda())
    swap = piv[:, 0].cpu().numpy() == 1
    assert (swap == (np.abs(x.real) + np.abs(x.imag) > np.abs(d.real) + np.abs(d.imag))).all()
    top, low = np.where(swap, x, d).astype(np.clongdouble), np.where(swap, d, x).astype(np.clongdouble)
    q = low / top
    err = np.abs(lu[:, 0, 1].cpu().numpy().astype(np.clongdouble) - q) / np.abs(q)
    assert float(err.max()) <= 8 * EPS
