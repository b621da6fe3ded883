"""The plans that the host makes: which kernel a call takes, and in how many parts.  The GPU tests name a shape for every route of the
GEMMs; if a retuned rule sends one of them elsewhere, the route is no longer tested and this says so."""
import ctypes as C

import pytest

import test_gemm_fp8_gpu
import test_gemm_gpu
from flagtree_b200 import _lib, ops


def _plan(fp8, m, n, k, sms=148):
    plan = (C.c_int32 * 3)()
    assert _lib.load().ftb_gemm_plan(fp8, m, n, k, sms, plan) == 0
    return tuple(plan)


@pytest.mark.parametrize("fp8,routes", [(0, test_gemm_gpu.ROUTES), (1, test_gemm_fp8_gpu.ROUTES)])
def test_gpu_tests_reach_every_route(fp8, routes):
    for route, shapes in routes.items():
        for m, n, k in shapes:
            assert _plan(fp8, m, n, k) == route, (m, n, k)
    # and there is no other one
    seen = set()
    for m in (1, 17, 40, 64, 129, 200, 300, 395, 512, 700, 1024, 2048, 4096, 8192):
        for n in range(128, 8193, 256):
            for k in (128, 512, 1024, 2304, 4096, 7168, 10240, 15616, 28672):
                seen.add(_plan(fp8, m, n, k))
    assert seen <= set(routes)


def test_plan_arguments_are_checked():
    plan = (C.c_int32 * 3)()
    lib = _lib.load()
    assert lib.ftb_gemm_plan(0, 0, 8, 8, 148, plan) == _lib.FTB_ERR_INVALID
    assert lib.ftb_gemm_plan(0, 8, 8, 8, 148, None) == _lib.FTB_ERR_INVALID


def test_paged_plan_of_few_and_many_tokens():
    assert ops._plan_paged(0, 128, 2048, 74)[0] >= 1                      # no token: nothing to divide by
    assert ops._plan_paged(3, 128, 2048, 74) == (16, False)
    assert ops._plan_paged(8, 128, 512, 74) == (8, False)
    assert ops._plan_paged(8, 128, 2048, 74)[1] and ops._plan_paged(8, 128, 2048, 74)[0] >= 9
    assert ops._plan_paged(30, 128, 2048, 74) == (2, True)
    assert ops._plan_paged(73, 128, 2048, 74) == (1, True)
    assert ops._plan_paged(128, 128, 2048, 74) == (1, True)
    assert ops._plan_paged(5, 16, 0, 74)[0] == 1
