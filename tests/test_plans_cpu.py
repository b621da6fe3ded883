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


@pytest.mark.parametrize("fp8,routes", [(0, test_gemm_gpu.ROUTES), (2, test_gemm_fp8_gpu.ROUTES)])
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


def test_gpu_tests_reach_the_halved_tiles():
    for route, shapes in test_gemm_fp8_gpu.ROUTES_HALVED.items():
        for m, n, k in shapes:
            assert _plan(2, m, n, k) == route, (m, n, k)
            assert _plan(1, m, n, k)[1:] == route[1:]                     # the same parts of K


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


@pytest.mark.parametrize("fp8", [0, 1])
def test_misaligned_split_workspace_is_refused(fp8):
    """Refused on the host, before anything is launched: the kernels write the partial results 16 bytes at a time."""
    lib = _lib.load()
    a = _lib.SparseMlaArgs()
    a.q = a.kv = a.indices = a.out = a.lse = 4096
    a.s_q, a.h, a.s_kv, a.topk = 4, 16, 1000, 256
    a.q_stride_token, a.q_stride_head, a.kv_stride_row, a.idx_stride_token = 16 * 576, 576, 576, 256
    a.out_stride_token, a.out_stride_head, a.lse_stride_token = 16 * 512, 512, 16
    a.sm_scale, a.n_splits = 0.05, 4
    if fp8:
        a.kv_is_fp8, a.page_size, a.q_per_seq, a.block_table_stride = 1, 64, 1, 16
        a.kv_scale = a.block_table = a.context_lens = 4096
    a.workspace, a.workspace_bytes = 4096 + 8, lib.ftb_sparse_mla_workspace_bytes(4, 16, 4)
    assert lib.ftb_sparse_mla_fwd(C.byref(a), None) == _lib.FTB_ERR_INVALID
    assert "aligned" in _lib.last_error()


def test_few_tokens_with_lists_of_more_than_three_tiles_are_cut_in_parts():
    """The parts are not for speed alone: every one has a weight of exactly 1."""
    for h in (16, 32, 64, 128):
        for s_q in (1, 2, 5, 8):
            assert [ops._plan_splits(s_q, h, topk, 74) for topk in (1, 128, 384)] == [1, 1, 1]
            for topk in (385, 512, 640, 768):
                assert ops._plan_splits(s_q, h, topk, 74) == -(-topk // 128)
        assert ops._plan_splits(16, h, 768, 74) >= 3
    assert ops._plan_splits(0, 128, 2048, 74) >= 1                        # no token: nothing to divide by


def test_whole_paged_tokens_take_a_table_where_it_is_the_faster_form():
    assert ops._table_is_faster(1, 128, 2048) and ops._table_is_faster(20, 64, 1024) and ops._table_is_faster(10, 16, 2048)
    assert not ops._table_is_faster(21, 64, 2048) and not ops._table_is_faster(11, 128, 2048) and not ops._table_is_faster(1, 128, 1023)
    assert not ops._table_is_faster(1, 16, 1024) and not ops._table_is_faster(0, 128, 0)
    assert not ops._table_is_faster(10, 128, 1 << 20)                     # 11 GB of scratch


def test_scratch_that_the_entry_points_allocate_is_what_the_library_asks_for():
    """The entry points work the sizes out themselves; the library refuses less."""
    lib = _lib.load()
    for s_q, h, n in ((1, 1, 2), (3, 128, 16), (300, 64, 2), (7, 17, 64)):
        assert ops._parts_bytes(s_q, h, n) == lib.ftb_sparse_mla_workspace_bytes(s_q, h, n)
    for pages in (1, 37, 4096):
        assert ops._cand_bytes(pages) == lib.ftb_kv_cache_write_workspace_bytes(pages)
