"""FP64 solves on a stream that may use only some of the SMs (a CUDA green context, as a process
that partitions its GPU sets up): the persistent launches take a grid that is resident there."""
import ctypes as C

import numpy as np
import pytest

import sp2_oracle as O
import sp2b
from sp2b import _lib, modelham as M

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def share(cuda):
    """(stream, SMs) of a green context with about a quarter of the SMs."""
    drv = pytest.importorskip("cuda.bindings.driver")
    cuda.zeros(1, device="cuda")
    held = []

    def call(fn, *a):
        r = fn(*a)
        if r[0] != drv.CUresult.CUDA_SUCCESS:
            pytest.skip(f"{fn.__name__}: {r[0]}")
        return r[1] if len(r) == 2 else r[1:]
    dev = call(drv.cuDeviceGet, 0)
    sms = call(drv.cuDeviceGetDevResource, dev, drv.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM)
    groups, _, _ = call(drv.cuDevSmResourceSplitByCount, 1, sms, 0, 32)
    desc = call(drv.cuDevResourceGenerateDesc, [groups[0]], 1)
    g = call(drv.cuGreenCtxCreate, desc, dev, drv.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM)
    st = call(drv.cuGreenCtxStreamCreate, g, drv.CUstream_flags.CU_STREAM_NON_BLOCKING, 0)
    held += [g, st]
    yield int(st), groups[0].sm.smCount
    cuda.cuda.synchronize()
    drv.cuStreamDestroy(st)
    drv.cuGreenCtxDestroy(g)


@pytest.mark.parametrize("n", [100, 500, 1000])
def test_dense_solve_and_response(cuda, share, n):
    torch = cuda
    stream, sms = share
    assert 0 < sms < torch.cuda.get_device_properties(0).multi_processor_count
    h, h1 = M.two_band_1d(n, seed=n), M.random_symmetric(n, seed=n + 1)
    dh, dh1 = torch.from_numpy(h).cuda(), torch.from_numpy(h1).cuda()
    rho, rsp = torch.empty_like(dh), torch.empty_like(dh)
    torch.cuda.synchronize()
    L = _lib.lib()
    o = _lib.make_opts(device_ptrs=True, stream=stream)
    _lib.check(L.sp2b_compute_response_sp2(dh.data_ptr(), dh1.data_ptr(), rsp.data_ptr(),
                                           rho.data_ptr(), n, 0.0, 0.5, 0, 100, b"None", 1e-10, 0.0,
                                           0, None, None, C.byref(o)), "response")
    ref, ref1, _ = O.compute_response_sp2(h, h1, 0.5, 0, 100, "None", 1e-10)
    # (two orders of summation, as tests/test_gpu_f64_solve.py derives it)
    assert np.linalg.norm(rho.cpu().numpy() - ref) <= 2e-12 * np.linalg.norm(ref)
    assert np.linalg.norm(rsp.cpu().numpy() - ref1) <= 4e-12 * np.linalg.norm(ref1)
    _lib.check(L.sp2b_sp2_alg2(dh.data_ptr(), rho.data_ptr(), n, 0.0, 0.5, 0, 100, b"None", 1e-10, 0,
                               C.byref(o), None), "alg2")
    assert np.linalg.norm(rho.cpu().numpy() - ref) <= 2e-12 * np.linalg.norm(ref)
