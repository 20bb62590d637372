"""Threads of the FP64 solves where a launch has room for fewer CTAs than it has items (the re-solve's limit, the fixed scratch,
a small batch buffer, a tuning): as many as a list of that length gets, and the same bits as the unlimited launch."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _launches(fn):
    """(threads, CTAs) of the kernels that fn launches, from a capture."""
    import torch
    from cuda.bindings import driver

    fn()  # what a first call looks up stays outside the capture
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        fn()
    raw = driver.CUgraph(g.raw_cuda_graph())
    _, _, n = driver.cuGraphGetNodes(raw)
    _, nodes, _ = driver.cuGraphGetNodes(raw, n)
    out = []
    for node in nodes:
        err, kind = driver.cuGraphNodeGetType(node)
        if kind == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            err, par = driver.cuGraphKernelNodeGetParams(node)
            assert err == driver.CUresult.CUDA_SUCCESS
            out.append((par.blockDimX, par.gridDimX))
    return out


@pytest.mark.parametrize("n,niv,Q", [(1, 20, 700), (1, 60, 400), (1, 96, 400), (2, 30, 300)])
def test_limited_launches(n, niv, Q):
    import torch

    from dgamore_b200._lib import BseProblem, BseTuning, call, lib

    rng = np.random.default_rng(niv)
    n2, nv, W, beta, ib2 = n * n, 2 * niv, 2, 2.0, 0.25
    N, n_items = n2 * nv, 4 * Q
    g = torch.Generator(device="cuda").manual_seed(niv)
    r = lambda *s: torch.randn(s, dtype=torch.complex128, device="cuda", generator=g)  # noqa: E731
    gamma, uv = r(2, W, N, N), r(2, Q, n2, n2)
    c0 = 0.1 * r(Q, W, nv, n2, n2) + 4.0 * torch.eye(n2, dtype=torch.complex128, device="cuda")
    work = np.array([(ch, q, w) for w in range(W) for ch in range(2) for q in range(Q)], dtype=np.int32)
    work = work[rng.permutation(n_items)]
    d_work = torch.from_numpy(work).cuda()
    st = torch.zeros(n_items, dtype=torch.int32, device="cuda")
    X = torch.zeros((2, Q, W, N, n2), dtype=torch.complex128, device="cuda")
    slot = (N * N + N * n2) * 16
    sc = torch.empty(int(lib().dga_bse_scratch_bytes(N, n2, n_items)) // 16 + 1, dtype=torch.complex128, device="cuda")
    s = lambda: ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)  # noqa: E731
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    head = (n, niv, W, Q, 2, beta, ib2, _p(gamma), _p(c0), _p(uv), _p(d_work))

    def plain(count=n_items):
        call("dga_bse_solve_sum_c128", *head, count, _p(X), _p(st), _p(sc), sc.numel() * 16, s())

    def check(fn, at_once):
        (threads, ctas), = _launches(fn)
        X.zero_()
        fn()
        assert torch.equal(X, ref)
        assert ctas <= at_once
        assert threads == _launches(lambda: plain(at_once))[0][0]

    plain()
    ref = X.clone()
    assert int(st.abs().sum().item()) == 0

    def resolve():
        st.fill_(4)
        call("dga_bse_resolve_fp64_c128", *head, n_items, _p(X), _p(st), sms, _p(sc), sms * slot, s())

    # the re-solve, whose status words another kernel of the capture writes: its own launch is the last one
    launches = _launches(resolve)
    X.zero_()
    resolve()
    assert torch.equal(X, ref) and launches[-1][1] <= sms
    assert launches[-1][0] == _launches(lambda: plain(sms))[0][0]

    check(lambda: call("dga_bse_solve_sum_noalloc_c128", *head, n_items, _p(X), _p(st), s()), min(n_items, (64 << 20) // slot))

    for ctas_per_sm in (1, 2):
        t = BseTuning(kernel=2, ctas_per_sm=ctas_per_sm)
        it = torch.zeros_like(st)
        check(lambda: call("dga_bse_solve_sum_tuned_c128", *head, n_items, 0, 6, 1e-10, _p(X), _p(st), _p(it), ctypes.byref(t),
                           _p(sc), sc.numel() * 16, s()), min(n_items, ctas_per_sm * sms))

    probs = (BseProblem * 1)(BseProblem(gamma_cm=gamma.data_ptr(), chi0_inv=c0.data_ptr(), uv=uv.data_ptr(), out=X.data_ptr(),
                                        n_orb=n, niv=niv, niw_half=W, n_q=Q, beta=beta, inv_beta2=ib2))
    d_probs = torch.frombuffer(bytearray(bytes(probs)), dtype=torch.uint8).cuda()
    items = torch.from_numpy(np.concatenate([np.zeros((n_items, 1), np.int32), work], axis=1)).cuda()
    padded = (slot + 255) // 256 * 256
    check(lambda: call("dga_bse_solve_sum_batch_c128", probs, _p(d_probs), 1, _p(items), n_items, 0, 6, 1e-10, _p(st), _p(it),
                       _p(sc), sms * padded, s()), sms)
