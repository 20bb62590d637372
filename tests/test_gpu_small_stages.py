"""The transforms and small-matrix stages at the edges of their splits: axes of one point, prime lengths and lengths on both
sides of the direct / two-stage line; more elements than the lambda search keeps; every orbital count with frequency
counts that fill no block."""

import ctypes

import numpy as np
import pytest

from oracle import ladder as oracle

pytestmark = pytest.mark.gpu

EPS = 2.0**-53


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("nk", [(1, 1, 1), (2, 1, 1), (1, 17, 1), (16, 16, 1), (17, 13, 1), (18, 18, 1), (48, 24, 1),
                                (27, 5, 3), (31, 2, 7), (1, 1, 64), (64, 64, 1), (121, 3, 1)])
def test_plane_transform(nk):
    import torch

    from dgamore_b200._lib import call
    from dgamore_b200.pipeline import twiddles

    rng = np.random.default_rng(sum(nk))
    n, planes = int(np.prod(nk)), 5
    x = rng.standard_normal((n, planes)) + 1j * rng.standard_normal((n, planes))
    a, tw = torch.from_numpy(x).cuda(), torch.from_numpy(twiddles(nk, -1)).cuda()
    out = torch.empty_like(a)
    call("dga_dft_planes_c128", _p(a), 1, 0, planes, _p(out), 1, 0, planes, 1, planes, *nk, _p(tw), 1.0,
         ctypes.c_void_p(0))
    ref = np.fft.fftn(x.reshape(*nk, planes), axes=(0, 1, 2)).reshape(n, planes)
    # each stage is a sum of at most 32 terms here (121 = 11 x 11, the primes directly), six stages
    bound = 8 * (sum(nk) + 6) * EPS * np.abs(x).sum(axis=0)
    assert (np.abs(out.cpu().numpy() - ref) <= bound).all()


@pytest.mark.parametrize("Q,W", [(1, 1), (3, 2), (7, 9), (45, 41), (561, 61), (2111, 41)])
def test_lambda(Q, W):
    import torch

    from dgamore_b200._lib import call

    rng = np.random.default_rng(Q * W)
    beta, nk = 10.0, 4 * Q
    chi = (0.2 + rng.random((2, Q, W))) / (1 + np.arange(W)) + 1e-3j * rng.standard_normal((2, Q, W))
    chi[:, :, 0] = chi[:, :, 0].real
    count = rng.integers(1, 8, Q)
    full = np.concatenate([np.conj(chi[..., :0:-1]), chi], axis=-1)
    target = 0.7 * (count[None, :, None] * full).sum(axis=(1, 2)) / beta / nk
    c, w, t = torch.from_numpy(chi).cuda(), torch.from_numpy(count.astype(np.int64)).cuda(), torch.from_numpy(target).cuda()
    lam = torch.zeros(2, dtype=torch.float64, device="cuda")
    its, st, out = torch.zeros(2, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda"), torch.empty_like(c)
    call("dga_lambda_c128", _p(c), Q, W, 2, _p(w), _p(t), beta, float(nk), 0.1, 1e-7, 1000, _p(lam), _p(its), _p(st),
         _p(out), ctypes.c_void_p(0))
    assert int(st.item()) == 0
    for ch in range(2):
        ref = oracle.find_lambda(full[ch], target[ch], count, beta, nk)
        assert abs(lam[ch].item() - ref) <= 1e-12 * max(1.0, abs(ref))
        assert np.allclose(out[ch].cpu().numpy(), 1 / (1 / chi[ch] + ref), rtol=1e-11, atol=0)


@pytest.mark.parametrize("n", [1, 2, 3, 4])
@pytest.mark.parametrize("niv,shell", [(1, 0), (5, 2), (17, 3)])
def test_double_counting_and_assembly(n, niv, shell):
    import torch

    from dgamore_b200._lib import call, lib

    rng = np.random.default_rng(n * 100 + niv)
    n2, nv, nvf, Q, W, beta = n * n, 2 * niv, 2 * (niv + shell), 3, 2, 7.0
    r = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    up = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    chi0, u, fdc = r(Q, W, nvf, n2, n2), r(n2, n2), r(W, n2 * nvf, n2 * nvf)
    d = [up(x) for x in (chi0, u, fdc)]
    k_dc = torch.empty((Q, W, nv, n2, n2), dtype=torch.complex128, device="cuda")
    sc = torch.empty(int(lib().dga_dc_scratch_bytes(n, niv + shell, W, Q)) // 16 + 1, dtype=torch.complex128, device="cuda")
    call("dga_dc_kernel_c128", _p(d[0]), _p(d[1]), _p(d[2]), n, niv, shell, W, Q, _p(k_dc), _p(sc), sc.numel() * 16,
         ctypes.c_void_p(0))
    left = np.einsum("ij,qwvjk->qwikv", u, chi0)
    f = fdc.reshape(W, n2, nvf, n2, nvf)[..., shell : shell + nv]
    ref = np.einsum("qwpmv,wmvsu->qwups", left, f)
    size = np.einsum("qwpmv,wmvsu->qwups", np.abs(u).sum() * np.abs(chi0).max() * np.ones_like(left, dtype=float), np.abs(f))
    assert (np.abs(k_dc.cpu().numpy() - ref) <= 8 * (n2 * nvf + n2) * EPS * size).all()

    c0i, x, uv, cp = r(Q, W, nv, n2, n2), r(2, Q, W, n2 * nv, n2), r(2, Q, n2, n2), r(2, Q, W, n2, n2)
    d = [up(t) for t in (c0i, x, uv, cp)]
    K, g3 = torch.empty_like(k_dc), torch.empty((2, Q, W, nv, n2, n2), dtype=torch.complex128, device="cuda")
    call("dga_kernel_assembly_c128", *[_p(t) for t in d], _p(k_dc), n, niv, W, Q, beta, _p(K), _p(g3), ctypes.c_void_p(0))
    xm = x.reshape(2, Q, W, n2, nv, n2).transpose(0, 1, 2, 4, 3, 5)
    gamma = beta * c0i[None] @ xm
    ref = -k_dc.cpu().numpy()
    for ch, fac in ((0, 1.0), (1, 3.0)):
        t = gamma[ch] - gamma[ch] @ uv[ch][:, None, None] @ cp[ch][:, :, None]
        if ch:
            t = t - 2.0 / 3.0 * np.eye(n2)
        ref = ref + fac * uv[ch][:, None, None] @ t
    # four products of at most 16 terms each
    scale = np.abs(ref).max() + 3 * n2 * np.abs(uv).max() ** 2 * n2 * np.abs(cp).max() * n2 * np.abs(gamma).max()
    assert np.abs(g3.cpu().numpy() - gamma).max() <= 8 * n2 * EPS * beta * n2 * np.abs(c0i).max() * np.abs(x).max()
    assert np.abs(K.cpu().numpy() - ref).max() <= 64 * n2 * EPS * scale
