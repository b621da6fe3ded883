"""GPU parity of the block-scaled FP8 GEMM against the CPU oracle (dequantise, fp32 product).  Tolerance:
the reference's fp8 GEMM tests use rtol = atol = 1e-2 on fp16 outputs
(third_party/mthreads/python/test/sqmma/base_cases/test_batch_fp8.py:54-57); the inputs here are exact e4m3
values, so the only error is fp32 accumulation order and the bf16 rounding of the output."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from flagtree_b200 import matmul_fp8_blockscaled
    from flagtree_b200 import workloads as W
from oracle.gemm_rs_ref import gemm_rs_fp8_ref

DEV = "cuda:0"


@pytest.mark.parametrize("m,n,k", [(128, 128, 128), (128, 256, 512), (256, 384, 1024), (200, 128, 256), (1024, 8192, 3584)])
def test_fp8_blockscaled_matches_oracle(m, n, k):
    g = torch.Generator().manual_seed(m + n + k)
    a8, a_s = W.quantize_block_e4m3(torch.randn(m, k, generator=g), 1, 128)
    b8, b_s = W.quantize_block_e4m3(torch.randn(k, n, generator=g), 128, 128)
    c = matmul_fp8_blockscaled(a8.to(DEV), a_s.to(DEV), b8.to(DEV), b_s.to(DEV))
    torch.cuda.synchronize()
    ref = gemm_rs_fp8_ref([a8], [a_s], [b8], [b_s])[0]
    err = (c.float().cpu() - ref).abs().max().item()
    scale = ref.abs().max().item()
    print(f"[fp8 {m}x{n}x{k}] max-abs err {err:.3e} (max |C| {scale:.3e})")
    assert err <= 2 ** -8 * scale


def test_weight_kept_as_n_by_k_gives_the_same_bits():
    """B passed as the transposed view of an [N, K] weight (the K-major operand of the tensor cores) must give the
    result of the [K, N] row-major call bit for bit: the same products are summed in the same order."""
    c = W.gemm_cfg5(tp=1, rank=0, m=384, n=512, k_total=640)
    a, b, a_s, b_s = c.a.to(DEV), c.b.to(DEV), c.a_scale.to(DEV), c.b_scale.to(DEV)
    ref = matmul_fp8_blockscaled(a, a_s, b, b_s)
    w = b.t().contiguous()                      # [N, K]
    got = matmul_fp8_blockscaled(a, a_s, w.t(), b_s)
    assert torch.equal(ref, got)


def test_fp8_unit_scales_equal_plain_product():
    g = torch.Generator().manual_seed(3)
    a = torch.randint(-8, 9, (256, 256), generator=g).float()
    b = torch.randint(-8, 9, (256, 256), generator=g).float()
    a8, b8 = a.to(torch.float8_e4m3fn).view(torch.uint8), b.to(torch.float8_e4m3fn).view(torch.uint8)
    ones_a, ones_b = torch.ones(256, 2), torch.ones(2, 2)
    c = matmul_fp8_blockscaled(a8.to(DEV), ones_a.to(DEV), b8.to(DEV), ones_b.to(DEV)).float().cpu()
    assert torch.equal(c, (a @ b).bfloat16().float())      # small integers: every partial sum is exact


# Tiles of one CTA with K in 1, 4 and 8 parts and tiles of a pair (the other choices are further down), most with a remainder
# in M and, for the pairs, an N that ends in the middle of a 256-column tile.  The sums of the parts of K are added in fp32,
# so the bound is the same as for one part: the bf16 rounding of the result.
@pytest.mark.parametrize("m,n,k", [(1, 128, 128), (7, 128, 256), (64, 1024, 7168), (130, 512, 2048), (60, 2048, 1024), (33, 3968, 4096),
                                   (129, 8192, 256), (520, 4224, 640), (1025, 8064, 128), (2049, 4224, 384)])
@pytest.mark.parametrize("nk", [False, True])
def test_fp8_tile_shapes_and_parts_of_k(m, n, k, nk):
    _check_fp8(m, n, k, nk)


# Single tiles take two K blocks per wait: odd counts in one part and in unequal parts (7 and 13 in four), and CTAs with two tiles
# (19 200 columns, 150 tiles), whose second one begins in the middle of such a pair of stages.
@pytest.mark.parametrize("m,n,k", [(64, 1024, 384), (50, 512, 896), (33, 3968, 1664), (64, 19200, 384), (128, 19200, 640)])
def test_fp8_odd_counts_of_k_blocks(m, n, k):
    _check_fp8(m, n, k, False)


def _check_fp8(m, n, k, nk):
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    a8, a_s = W.quantize_block_e4m3(torch.randn(m, k, generator=g, device=DEV), 1, 128)
    b8, b_s = W.quantize_block_e4m3(torch.randn(k, n, generator=g, device=DEV), 128, 128)
    b = b8.t().contiguous().t() if nk else b8
    c = matmul_fp8_blockscaled(a8, a_s, b, b_s).double()
    deq_a = a8.view(torch.float8_e4m3fn).double().view(m, k // 128, 128) * a_s.double()[..., None]
    deq_b = b8.view(torch.float8_e4m3fn).double().view(k // 128, 128, n // 128, 128) * b_s.double()[:, None, :, None]
    ref = deq_a.view(m, k) @ deq_b.view(k, n)
    # 2^-8 of the value for the bf16 result, 2^-17 of the largest value for sums in fp32 in any order
    assert ((c - ref).abs() <= 2 ** -8 * ref.abs() + 2 ** -17 * ref.abs().max()).all()


# One shape or two per route of the dispatch on 148 SMs: (columns of a tile, CTAs that share it, parts of K).
ROUTES = {(64, 1, 1): [(60, 2048, 1024), (130, 512, 1024)], (64, 1, 4): [(64, 2048, 7168)], (128, 1, 1): [(128, 9600, 384)], (128, 1, 2): [(40, 8192, 7168)],
          (128, 1, 4): [(33, 3968, 4096)], (128, 1, 8): [(64, 1024, 7168)],
          (256, 2, 1): [(1025, 2176, 384), (1030, 3200, 1664)], (256, 2, 2): [(142, 4608, 13824), (162, 4224, 10240), (395, 2304, 15616)]}


# Where few single tiles are halved to 64 columns: both sides of that line, some with an odd count of K blocks.
ROUTES_HALVED = {(64, 1, 1): [(60, 2048, 1024), (1, 128, 384), (128, 9472, 384), (257, 3072, 640)], (64, 1, 4): [(64, 2048, 7168), (100, 1920, 3456)],
                 (128, 1, 1): [(128, 9600, 384)], (128, 1, 4): [(33, 3968, 4096)], (128, 1, 8): [(64, 1920, 7168)]}


@pytest.mark.parametrize("m,n,k", [s for shapes in ROUTES_HALVED.values() for s in shapes])
@pytest.mark.parametrize("nk", [False, True])
def test_fp8_every_route_of_halved_tiles(m, n, k, nk):
    _check_fp8(m, n, k, nk)


@pytest.mark.parametrize("m,n,k", [(64, 1024, 1024), (64, 2048, 7168), (100, 9472, 384), (128, 9600, 384), (64, 1920, 7168)])
def test_fp8_same_bits_in_both_layouts(m, n, k):
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    a8, a_s = W.quantize_block_e4m3(torch.randn(m, k, generator=g, device=DEV), 1, 128)
    b8, b_s = W.quantize_block_e4m3(torch.randn(k, n, generator=g, device=DEV), 128, 128)
    assert torch.equal(matmul_fp8_blockscaled(a8, a_s, b8, b_s), matmul_fp8_blockscaled(a8, a_s, b8.t().contiguous().t(), b_s))


@pytest.mark.parametrize("m,n,k", [s for shapes in ROUTES.values() for s in shapes])
@pytest.mark.parametrize("nk", [False, True])
def test_fp8_every_route(m, n, k, nk):
    """The result, and the same with K in one part: a row then has the bits that it has in a product of many rows."""
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    a8, a_s = W.quantize_block_e4m3(torch.randn(m + 2048, k, generator=g, device=DEV), 1, 128)
    b8, b_s = W.quantize_block_e4m3(torch.randn(k, n, generator=g, device=DEV), 128, 128)
    b = b8.t().contiguous().t() if nk else b8
    deq_a = a8[:m].view(torch.float8_e4m3fn).double().view(m, k // 128, 128) * a_s[:m].double()[..., None]
    deq_b = b8.view(torch.float8_e4m3fn).double().view(k // 128, 128, n // 128, 128) * b_s.double()[:, None, :, None]
    ref = deq_a.view(m, k) @ deq_b.view(k, n)
    whole = matmul_fp8_blockscaled(a8[:m], a_s[:m], b, b_s, whole_k=True)
    for c in (matmul_fp8_blockscaled(a8[:m], a_s[:m], b, b_s), whole):
        # 2^-8 of the value for the bf16 result, 2^-16 of the largest value for sums in fp32 in any order
        assert ((c.double() - ref).abs() <= 2 ** -8 * ref.abs() + 2 ** -16 * ref.abs().max()).all()
    assert torch.equal(whole, matmul_fp8_blockscaled(a8, a_s, b, b_s, whole_k=True)[:m])
