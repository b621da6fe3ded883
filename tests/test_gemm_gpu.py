"""GPU parity of the tcgen05 GEMM (through the C ABI) against the fp32 CPU product, following the
reference's matmul test idiom (python/test/unit/operators/test_matmul.py:187-199: golden = torch.matmul
of the same inputs).  bf16 output: relative error bound 2^-8 of the row-block magnitude."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from flagtree_b200 import matmul, spec
    from flagtree_b200 import workloads as W

DEV = "cuda:0"


def _check(a, b, name=""):
    c = matmul(a.to(DEV), b.to(DEV))
    torch.cuda.synchronize()
    ref = a.float() @ b.float()
    err = (c.float().cpu() - ref).abs().max().item()
    scale = ref.abs().max().item()
    print(f"[{name}] max-abs err {err:.3e} (max |C| {scale:.3e})")
    assert err <= 2 ** -8 * scale + 1e-30, (name, err, scale)
    return c


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (128, 256, 512), (256, 512, 128), (384, 768, 320),
                                   (200, 264, 72), (1, 8, 8), (130, 1000, 1096), (1024, 256, 2304)])
def test_matmul_shapes(m, n, k):
    g = torch.Generator().manual_seed(m * 7 + n * 3 + k)
    a = torch.randn(m, k, generator=g).bfloat16()
    b = torch.randn(k, n, generator=g).bfloat16()
    _check(a, b, f"{m}x{n}x{k}")


@pytest.mark.parametrize("m,n,k", [(1, 512, 512), (50, 7168, 2304), (64, 9472, 128), (127, 8, 520), (129, 4160, 2304), (512, 512, 1024),
                                   (40, 4104, 584), (8, 136, 64), (300, 6152, 1000), (17, 2048, 72)])
def test_products_with_few_tiles(m, n, k):
    """Shapes that leave most SMs idle at 128 x 256: narrow tiles (64 columns, a last one of 8), K in one, two and four
    parts with K tails and parts of unequal length, one to four row blocks, row counts that are not a multiple of eight; and the
    persistent kernel just above the line (300 x 6152)."""
    g = torch.Generator().manual_seed(m + n + k)
    a = torch.randn(m, k, generator=g).bfloat16()
    b = torch.randn(k, n, generator=g).bfloat16()
    c = _check(a, b, f"{m}x{n}x{k}")
    assert torch.equal(c, matmul(a.to(DEV), b.to(DEV)))


@pytest.mark.parametrize("k", [64, 192, 448, 832, 1096])
@pytest.mark.parametrize("m,n", [(50, 1024), (128, 9472)])
def test_narrow_tiles_with_odd_counts_of_k_blocks(m, n, k):
    """The narrow tiles take two K blocks per wait: counts of 1, 3, 7, 13 and 18 (the last one short), in one part and split unequally."""
    g = torch.Generator().manual_seed(m + n + k)
    _check(torch.randn(m, k, generator=g).bfloat16(), torch.randn(k, n, generator=g).bfloat16(), f"{m}x{n}x{k}")


@pytest.mark.parametrize("m,n,k", [(4096, 4864, 256), (2048, 9992, 128), (3072, 2560, 192)])
def test_leftover_tiles_run_as_half_width_steps(m, n, k):
    """Shapes whose tile count leaves a few tiles after the whole waves of a 148-SM GPU: 304 = 4 x 74 + 8 pair
    tiles; 320 = 4 x 74 + 24 with a last column block of 8 columns; 120 = 74 + 46 (too many left to halve).  The
    leftover runs as 128-column halves where that helps, and every element must still be the product."""
    g = torch.Generator().manual_seed(m + n + k)
    a = torch.randn(m, k, generator=g).bfloat16()
    b = torch.randn(k, n, generator=g).bfloat16()
    c = _check(a, b, f"{m}x{n}x{k}")
    assert torch.equal(c, matmul(a.to(DEV), b.to(DEV)))


def test_matmul_powers_of_two_exact():
    """Inputs 2^randint(-3,0) as in test_matmul.py:164-176; K=64 keeps every fp32 partial sum exact,
    so the result must equal the fp32 product rounded to bf16 bit for bit."""
    g = torch.Generator().manual_seed(0)
    a = (2.0 ** torch.randint(-3, 1, (256, 64), generator=g)).bfloat16()
    b = (2.0 ** torch.randint(-3, 1, (64, 512), generator=g)).bfloat16()
    c = matmul(a.to(DEV), b.to(DEV)).cpu()
    assert torch.equal(c, (a.float() @ b.float()).bfloat16())


def test_cfg4_per_rank_product():
    case = W.gemm_cfg4(tp=8, rank=3)
    _check(case.a, case.b, case.name)


def test_strided_and_transposed_inputs_are_copied_like_the_reference():
    g = torch.Generator().manual_seed(5)
    a = torch.randn(96, 300, generator=g).bfloat16().to(DEV)
    b = torch.randn(512, 96, generator=g).bfloat16().to(DEV)
    c = matmul(a.t()[:256], b.t())          # both operands column-major views
    ref = a.t()[:256].float().cpu() @ b.t().float().cpu()
    assert (c.float().cpu() - ref).abs().max().item() <= 2 ** -8 * ref.abs().max().item()


def test_spec_hook_writes_into_caller_buffer():
    g = torch.Generator().manual_seed(9)
    a = torch.randn(256, 128, generator=g).bfloat16().to(DEV)
    b = torch.randn(128, 512, generator=g).bfloat16().to(DEV)
    c = torch.zeros(256, 512, dtype=torch.bfloat16, device=DEV)
    handled = spec.matmul_kernel(None, a, b, c, 256, 512, 128, torch.float32, None, True, torch.bfloat16)
    assert handled is True
    assert torch.equal(c, matmul(a, b))
    # unsupported dtype -> None, the reference's own kernel would run
    assert spec.matmul_kernel(None, a.half(), b.half(), c, 256, 512, 128, None, None, True, torch.float16) is None


def test_determinism():
    g = torch.Generator().manual_seed(1)
    a = torch.randn(1024, 2304, generator=g).bfloat16().to(DEV)
    b = torch.randn(2304, 1792, generator=g).bfloat16().to(DEV)
    assert torch.equal(matmul(a, b), matmul(a, b))


# One shape or two per route of the dispatch on 148 SMs, with tails in M, N and K: (columns of a tile, CTAs that share it, parts of K).
ROUTES = {(64, 1, 1): [(50, 7168, 2304), (129, 4160, 200)], (64, 1, 2): [(40, 4104, 584), (33, 4096, 2304)], (64, 1, 4): [(17, 2048, 2304), (129, 512, 1096)],
          (128, 1, 1): [(300, 6136, 1000), (512, 4096, 2304)], (256, 1, 1): [(50, 20488, 584), (128, 19456, 136)], (256, 2, 1): [(700, 6152, 328)]}


@pytest.mark.parametrize("m,n,k", [s for shapes in ROUTES.values() for s in shapes])
def test_every_route(m, n, k):
    """The result, and the same with K in one part: a row then has the bits that it has in a product of many rows."""
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    a = torch.randn(m, k, generator=g, device=DEV).bfloat16()
    b = torch.randn(k, n, generator=g, device=DEV).bfloat16()
    ref = a.double() @ b.double()
    many = torch.cat([a, torch.randn(2048, k, generator=g, device=DEV).bfloat16()])
    whole = matmul(a, b, whole_k=True)
    for c in (matmul(a, b), whole):
        # 2^-8 of the value for the bf16 result, 2^-16 of the largest value for sums in fp32 in any order
        assert ((c.double() - ref).abs() <= 2 ** -8 * ref.abs() + 2 ** -16 * ref.abs().max()).all()
    assert torch.equal(whole, matmul(many, b, whole_k=True)[:m])
