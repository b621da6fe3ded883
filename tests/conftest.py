import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

GOLDEN_DIR = os.path.join(ROOT, "tests", "golden")

# Parity tolerances stated by the benchmark contract: bf16 output max-abs error and LSE
# relative error against the fp32 oracle.
OUT_ATOL = 2e-2
LSE_RTOL = 1e-3


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")


@pytest.fixture(scope="session")
def golden_dir():
    return GOLDEN_DIR


def paged_algo(args, sm_scale, page_size, algo, splits):
    """The paged form through the C ABI, with a kernel and a number of parts of the caller's choice."""
    import ctypes as C

    import torch

    from flagtree_b200 import _lib
    q, cache, scale, table, lens, idx = args
    b, n_q, h, _ = q.shape
    topk = idx.shape[2]
    lib = _lib.load()
    out = torch.empty(b, n_q, h, 512, dtype=torch.bfloat16, device=q.device)
    lse = torch.empty(b, n_q, h, dtype=torch.float32, device=q.device)
    status = torch.zeros(1, dtype=torch.int32, device=q.device)
    a = _lib.SparseMlaArgs(q.data_ptr(), cache.data_ptr(), idx.data_ptr(), out.data_ptr(), lse.data_ptr(), b * n_q, h, cache.shape[0] * page_size,
                           topk, h * 576, 576, 576, topk, h * 512, 512, h, sm_scale, 0, algo, status.data_ptr(), 1, scale.data_ptr(),
                           table.data_ptr(), lens.data_ptr(), page_size, n_q, table.stride(0))
    ws = torch.empty(max(1, lib.ftb_sparse_mla_workspace_bytes(b * n_q, h, splits)), dtype=torch.uint8, device=q.device)
    a.n_splits, a.workspace, a.workspace_bytes = splits, ws.data_ptr(), ws.numel()
    assert lib.ftb_sparse_mla_fwd(C.byref(a), C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0, _lib.last_error()
    torch.cuda.synchronize()
    assert status.item() == 0
    return out, lse
