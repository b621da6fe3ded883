"""GPU parity of the top-k index producer (through the C ABI) against its CPU restatement: index lists must be
identical, including ties (lower position wins), signed zeros, infinities, lengths shorter than topk, empty rows
and rows longer than one pass of the block; and its output must drive the sparse MLA forward."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from flagtree_b200 import sparse_mla_fwd, topk_indices
from oracle.sparse_mla_ref import sparse_mla_fwd_ref, topk_indices_ref

DEV = "cuda:0"


@pytest.mark.parametrize("s_kv,topk", [(1, 1), (37, 5), (512, 512), (513, 64), (1024, 1000), (4096, 2048), (32768, 2048),
                                       (70000, 2048)])
def test_random_scores_match_exactly(s_kv, topk):
    g = torch.Generator().manual_seed(s_kv + topk)
    sc = torch.randn(9, s_kv, generator=g)
    got = topk_indices(sc.to(DEV), topk).cpu()
    assert torch.equal(got, topk_indices_ref(sc, topk))


def test_ties_zeros_infinities_and_lengths():
    g = torch.Generator().manual_seed(3)
    s_q, s_kv, topk = 12, 1500, 300
    sc = torch.randint(-3, 4, (s_q, s_kv), generator=g).float()          # seven distinct values: ties everywhere
    sc[0, ::7] = -0.0
    sc[1, 5] = float("inf")
    sc[1, 9] = -float("inf")
    sc[2] = 1.0                                                            # a constant row: the first topk positions
    lengths = torch.tensor([1500, 1500, 1500, 0, 1, 299, 300, 301, 777, 1500, 1024, 513], dtype=torch.int32)
    got = topk_indices(sc.to(DEV), topk, lengths.to(DEV)).cpu()
    want = topk_indices_ref(sc, topk, lengths)
    assert torch.equal(got, want)
    assert torch.equal(got[2], torch.arange(topk, dtype=torch.int32))
    assert (got[3] == -1).all() and got[4, 0] == 0 and (got[4, 1:] == -1).all()
    assert (got[5, :299] == torch.arange(299)).all() and got[5, 299] == -1


def test_many_rows_with_causal_lengths_and_a_strided_view():
    """More rows than SMs (the persistent kernel takes several rows per CTA), ragged lengths, ties from rounding the
    scores to bf16, and a view whose rows are not contiguous."""
    g = torch.Generator().manual_seed(11)
    s_q, s_kv, topk = 700, 8192, 512
    wide = torch.randn(s_q, s_kv + 64, generator=g).bfloat16().float()
    sc = wide[:, :s_kv]
    lengths = torch.randint(0, s_kv + 1, (s_q,), generator=g).int()
    lengths[:4] = torch.tensor([0, 1, s_kv, 512])
    got = topk_indices(wide.to(DEV)[:, :s_kv], topk, lengths.to(DEV)).cpu()
    assert torch.equal(got, topk_indices_ref(sc, topk, lengths))


def test_long_rows_with_few_distinct_values_and_a_misleading_sample():
    """Rows long enough for the sampled bracket: few distinct values (crowded bins, ties across many threads), a
    constant row, a sorted row, and a row whose sampled positions hold values unlike the rest (the bracket is
    rejected and the whole key range is searched)."""
    g = torch.Generator().manual_seed(21)
    s_kv, topk = 32768, 2048
    rows = [torch.randint(-3, 4, (s_kv,), generator=g).float(),
            torch.full((s_kv,), 2.5),
            torch.arange(s_kv).float(),
            -torch.arange(s_kv).float(),
            torch.randn(s_kv, generator=g).mul(1e-30),                  # denormal-range keys
            torch.randn(s_kv, generator=g)]
    odd = torch.randn(s_kv, generator=g)
    sample_at = (torch.arange(256) * s_kv >> 8) + (torch.arange(256) & 15)
    odd[sample_at] = 1e6
    rows.append(odd)
    low = torch.randn(s_kv, generator=g)
    low[sample_at] = -1e6
    rows.append(low)
    sc = torch.stack(rows)
    lengths = torch.tensor([s_kv, s_kv, s_kv, s_kv, s_kv, 4096, s_kv, s_kv], dtype=torch.int32)
    for k in (topk, 1, 32767):
        got = topk_indices(sc.to(DEV), k, lengths.to(DEV)).cpu()
        assert torch.equal(got, topk_indices_ref(sc, k, lengths)), k


def test_causal_lengths_feed_the_forward():
    """The producer's output as the `indices` of the forward: causal lengths, scores = q.k of head 0."""
    g = torch.Generator().manual_seed(8)
    s_q, h, s_kv, topk = 64, 16, 640, 128
    q = torch.randn(s_q, h, 576, generator=g).bfloat16()
    kv = torch.randn(s_kv, 576, generator=g).bfloat16()
    scores = q[:, 0].float() @ kv.float().T
    lengths = (torch.arange(s_q) * 10 + 1).int()
    idx = topk_indices(scores.to(DEV), topk, lengths.to(DEV))
    assert torch.equal(idx.cpu(), topk_indices_ref(scores, topk, lengths))
    out, lse = sparse_mla_fwd(q.to(DEV), kv.to(DEV), idx, 0.05, check=True)
    ref_out, ref_lse = sparse_mla_fwd_ref(q, kv, idx.cpu(), 0.05)
    assert (out.float().cpu() - ref_out).abs().max().item() <= 2e-2
    assert ((lse.cpu() - ref_lse).abs() / ref_lse.abs().clamp(min=1)).max().item() <= 1e-3


@pytest.mark.parametrize("s_kv", [4095, 4097, 32767, 32768, 32769, 33791, 50001, 65535, 65536, 65537])
def test_edges_of_the_row_kernels(s_kv):
    """Lengths around what the registers and the shared memory hold, rows that are not 16-byte aligned (odd strides),
    rows of two values (more ties than the candidate list holds), rows that rise or fall (the candidates of a row sit in
    few warps), a sample unlike the rest, NaN patterns, and more rows than SMs for the ragged case."""
    g = torch.Generator().manual_seed(s_kv)
    odd = torch.randn(s_kv, generator=g)
    odd[(torch.arange(256) * s_kv >> 8) + (torch.arange(256) & 15)] = -1e6
    nan = torch.randn(s_kv, generator=g)
    nan[3::1000] = float("nan")
    nan[5::1000] = -float("nan")
    rows = [torch.randn(s_kv, generator=g), torch.randint(0, 2, (s_kv,), generator=g).float(), torch.full((s_kv,), -0.0),
            torch.arange(s_kv).float(), -torch.arange(s_kv).float(), odd, nan, torch.randn(s_kv, generator=g).bfloat16().float()]
    sc = torch.stack(rows * (20 if s_kv == 32769 else 1))
    lengths = torch.full((sc.shape[0],), s_kv, dtype=torch.int32)
    lengths[-1] = max(1, s_kv - 777)
    for k in (2048, 1, s_kv - 1):
        got = topk_indices(sc.to(DEV), k, lengths.to(DEV)).cpu()
        assert torch.equal(got, topk_indices_ref(sc, k, lengths)), k


@pytest.mark.parametrize("s_q,s_kv", [(300, 33), (7, 1000), (160, 5119), (3, 5121), (150, 6656), (149, 6657), (5, 20001), (150, 32765), (300, 40003)])
def test_ties_and_lengths_on_every_kernel(s_q, s_kv):
    """Rows of few values, rows padded with -inf, rows that are short in a long matrix and rows that do not start on a 16-byte boundary, at
    sizes either side of the lines between the kernels."""
    g = torch.Generator().manual_seed(s_kv)
    sc = torch.randn(s_q, s_kv, generator=g)
    sc[::3] = (sc[::3] * 4).round()
    sc[1::3] = torch.where(torch.arange(s_kv) < s_kv // 20, sc[1::3], float("-inf"))
    lengths = torch.randint(0, s_kv + 1, (s_q,), generator=g).int()
    lengths[::2] = torch.minimum(lengths[::2], torch.randint(1, 6000, (lengths[::2].numel(),), generator=g).int())
    lengths[:3] = torch.tensor([s_kv, 0, 1])
    wide = torch.zeros(s_q, s_kv + 5)
    wide[:, 1:s_kv + 1] = sc
    for k in (min(512, s_kv), min(2048, s_kv)):
        ref = topk_indices_ref(sc, k, lengths)
        assert torch.equal(topk_indices(sc.to(DEV), k, lengths.to(DEV)).cpu(), ref)
        assert torch.equal(topk_indices(wide.to(DEV)[:, 1:s_kv + 1], k, lengths.to(DEV)).cpu(), ref)


@pytest.mark.parametrize("rows,s_kv,topk", [(3, 511, 100), (3, 512, 100), (3, 513, 512), (2, 4096, 64), (2, 4097, 64), (5, 8192, 2048),
                                            (5, 8193, 2048), (2, 65536, 2048), (2, 65536, 30000), (3, 32768, 16384), (200, 5001, 512),
                                            (200, 3000, 2999), (150, 12001, 5000), (900, 24577, 65), (160, 65535, 1)])
@pytest.mark.parametrize("values", ["plain", "crowded", "negative"])
def test_lists_of_candidates(rows, s_kv, topk, values):
    """Both sides of every rule of the dispatch and of the list: rows that are their own sample, that fit the list as a whole, that fill an
    SM or share one; keys whose bound is a value that fills much of the row; bounds below zero; an unaligned view; short and empty rows."""
    g = torch.Generator().manual_seed(rows + s_kv + topk)
    wide = torch.randn(rows, s_kv + 3, generator=g)
    if values == "crowded":
        wide = wide.clamp(-0.5, 0.5).mul(4).round()
    elif values == "negative":
        wide = -wide.abs() - 1e-30
    lengths = torch.full((rows,), s_kv, dtype=torch.int32)
    if rows >= 5:
        lengths[1:5] = torch.tensor([0, min(topk, s_kv), min(topk + 1, s_kv), s_kv // 3])
    got = topk_indices(wide.to(DEV)[:, 1:1 + s_kv], topk, lengths.to(DEV)).cpu()
    assert torch.equal(got, topk_indices_ref(wide[:, 1:1 + s_kv], topk, lengths))


@pytest.mark.parametrize("rows,s_kv,topk", [(2, 2048, 512), (2, 2049, 512), (150, 1024, 300), (150, 1025, 300), (150, 4096, 2400), (150, 4097, 2400),
                                            (150, 32768, 16384), (4, 20000, 9000), (4, 20000, 10000), (900, 24577, 2049)])
@pytest.mark.parametrize("values", ["plain", "huge"])
def test_whole_rows_and_long_lists(rows, s_kv, topk, values):
    """Both sides of the lines between rows taken whole and rows swept, and lists that fill an SM; scores among which an interval of the
    search ends in an infinity or is wider than the largest float."""
    g = torch.Generator().manual_seed(rows + s_kv + topk + 1)
    sc = torch.randn(rows, s_kv, generator=g) * (2e38 if values == "huge" else 1.0)
    assert torch.equal(topk_indices(sc.to(DEV), topk).cpu(), topk_indices_ref(sc, topk))


@pytest.mark.parametrize("rows,s_kv,topk", [(3, 1000, 333), (150, 1000, 100), (150, 4096, 1300), (150, 4097, 1300), (150, 2048, 682), (1, 4096, 50)])
@pytest.mark.parametrize("values", [1, 2, 10])
def test_short_rows_of_few_values(rows, s_kv, topk, values):
    """Rows whose k-th largest key is one of many equal ones, whole and swept, either side of the length up to which the radix select finishes them."""
    g = torch.Generator().manual_seed(rows + s_kv + topk + values)
    sc = torch.randint(0, values, (rows, s_kv), generator=g).float() - 0.3 * (values // 2)
    assert torch.equal(topk_indices(sc.to(DEV), topk).cpu(), topk_indices_ref(sc, topk))


@pytest.mark.parametrize("top", [0.0, 1e6, -1e6])
def test_sample_that_misleads(top):
    """The sampled positions hold values unlike the rest: a bound that is too high, or a list that overflows, sends the row to the radix select."""
    g = torch.Generator().manual_seed(31)
    s_kv, t = 40000, torch.arange(512)
    at = t * s_kv // 512 + ((((t * 0x9E3779B1) & 0xFFFFFFFF) >> 16) * (s_kv // 512) >> 16)
    sc = torch.randn(4, s_kv, generator=g)
    sc[:, at] = top
    sc[1] = sc[1].abs()
    sc[2] = -sc[2].abs()
    got = topk_indices(sc.to(DEV), 2048).cpu()
    assert torch.equal(got, topk_indices_ref(sc, 2048))
