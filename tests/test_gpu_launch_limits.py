"""A launch leaves a kernel's shared-memory limit where it was: a small call between another thread's preparation and launch of
a large one does not make that launch fail."""

import ctypes

import pytest

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _s():
    import torch

    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _kernels(fn):
    """(function, dynamic shared memory) of the kernels that fn launches, from a capture."""
    import torch
    from cuda.bindings import driver

    fn()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        fn()
    raw = driver.CUgraph(g.raw_cuda_graph())
    _, _, n = driver.cuGraphGetNodes(raw)
    _, nodes, _ = driver.cuGraphGetNodes(raw, n)
    out = []
    for node in nodes:
        _, kind = driver.cuGraphNodeGetType(node)
        if kind == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            err, par = driver.cuGraphKernelNodeGetParams(node)
            assert err == driver.CUresult.CUDA_SUCCESS
            func = int(par.func)
            if func == 0:
                err, kernel = driver.cuKernelGetFunction(par.kern)
                assert err == driver.CUresult.CUDA_SUCCESS
                func = int(kernel)
            out.append((func, par.sharedMemBytes))
    return out


def _lambda(Q, W):
    import torch

    from dgamore_b200._lib import call

    chi = torch.full((1, Q, W), 0.5, dtype=torch.complex128, device="cuda")
    count = torch.ones(Q, dtype=torch.int64, device="cuda")
    target = torch.full((1,), 0.2, dtype=torch.complex128, device="cuda")
    lam = torch.zeros(1, dtype=torch.float64, device="cuda")
    its, st, out = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda"), torch.empty_like(chi)
    return lambda: call("dga_lambda_c128", _p(chi), Q, W, 1, _p(count), _p(target), 10.0, float(Q), 0.1, 1e-7, 50, _p(lam),
                        _p(its), _p(st), _p(out), _s())


def _double_counting(n, niv):
    import torch

    from dgamore_b200._lib import call, lib

    n2, nv = n * n, 2 * niv
    z = lambda *s: torch.zeros(s, dtype=torch.complex128, device="cuda")  # noqa: E731
    chi0, u, fdc, out = z(2, 2, nv, n2, n2), z(n2, n2), z(2, n2 * nv, n2 * nv), z(2, 2, nv, n2, n2)
    sc = z(int(lib().dga_dc_scratch_bytes(n, niv, 2, 2)) // 16 + 1)
    return lambda: call("dga_dc_kernel_c128", _p(chi0), _p(u), _p(fdc), n, niv, 0, 2, 2, _p(out), _p(sc), sc.numel() * 16, _s())


def _plane(nk):
    import torch

    from dgamore_b200._lib import call
    from dgamore_b200.pipeline import twiddles

    tw = torch.from_numpy(twiddles((nk, nk, 1), -1)).cuda()
    a = torch.zeros((2, nk * nk), dtype=torch.complex128, device="cuda")
    b = torch.empty_like(a)
    return lambda: call("dga_dft_planes_c128", _p(a), nk * nk, 0, 1, _p(b), nk * nk, 0, 1, 2, 1, nk, nk, 1, _p(tw), 1.0, _s())


def _factorisation(N):
    import torch

    from dgamore_b200._lib import call

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 8 * sms + 1  # one warp a matrix up to N = 64
    a = torch.eye(N, dtype=torch.complex128, device="cuda").repeat(n, 1, 1)
    piv = torch.empty((n, N), dtype=torch.int32, device="cuda")
    st = torch.zeros(n, dtype=torch.int32, device="cuda")
    return lambda: call("dga_lu_batched_c128", _p(a), N, n, N * N, _p(piv), _p(st), _s())


@pytest.mark.parametrize("make,large,small", [(_lambda, (600, 121), (5, 3)), (_double_counting, (4, 8), (1, 2)),
                                              (_plane, (64,), (4,)), (_factorisation, (64,), (8,))])
def test_a_small_call_leaves_the_limit(make, large, small):
    import torch
    from cuda.bindings import driver

    big = _kernels(make(*large))
    few = dict(_kernels(make(*small)))
    torch.cuda.synchronize()
    assert any(f in few and few[f] < smem for f, smem in big)
    for f, smem in big:
        err, limit = driver.cuFuncGetAttribute(driver.CUfunction_attribute.CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES,
                                               driver.CUfunction(f))
        assert err == driver.CUresult.CUDA_SUCCESS and limit >= smem
