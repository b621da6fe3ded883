"""GPU parity of the few-heads kernel (algo 2: one CTA per token, the gathered rows on the rows of the MMA, scores
transposed) against the CPU oracle, through the C ABI: every head count up to 32, ragged and padded index lists,
tokens that select nothing, a running maximum that moves on every tile, bad indices, and agreement with the
kernel for many heads on the same inputs."""
import pytest
import torch

from conftest import paged_algo

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from flagtree_b200 import sparse_mla_fwd
    from flagtree_b200 import workloads as W
from oracle.sparse_mla_ref import sparse_mla_fwd_ref

DEV = "cuda:0"


def _check(q, kv, idx, sm_scale, name):
    out, lse = sparse_mla_fwd(q.to(DEV), kv.to(DEV), idx.to(DEV), sm_scale, check=True, algo=2)
    ref_out, ref_lse = sparse_mla_fwd_ref(q, kv, idx, sm_scale)
    err = (out.float().cpu() - ref_out).abs().max().item()
    fin = torch.isfinite(ref_lse)
    assert torch.equal(torch.isfinite(lse.cpu()), fin), name
    lerr = ((lse.cpu()[fin] - ref_lse[fin]).abs() / ref_lse[fin].abs().clamp(min=1)).max().item() if fin.any() else 0.0
    print(f"[{name}] out max-abs err {err:.3e}  lse rel err {lerr:.3e}")
    assert err <= 2e-2 and lerr <= 1e-3, (name, err, lerr)
    return out, lse


@pytest.mark.parametrize("h", [1, 8, 16, 17, 24, 32])
@pytest.mark.parametrize("topk", [1, 100, 128, 129, 640])
def test_head_counts_and_ragged_topk(h, topk):
    g = torch.Generator().manual_seed(100 * h + topk)
    s_q, s_kv = 7, 900
    q = torch.randn(s_q, h, 576, generator=g).bfloat16()
    kv = torch.randn(s_kv, 576, generator=g).bfloat16()
    idx = torch.stack([torch.randperm(s_kv, generator=g)[:topk] for _ in range(s_q)]).int()
    _check(q, kv, idx, 576 ** -0.5, f"h{h}_topk{topk}")


def test_padding_inside_the_list_and_tokens_that_select_nothing():
    g = torch.Generator().manual_seed(5)
    s_q, h, s_kv, topk = 9, 16, 500, 300
    q = torch.randn(s_q, h, 576, generator=g).bfloat16()
    kv = torch.randn(s_kv, 576, generator=g).bfloat16()
    idx = torch.stack([torch.randperm(s_kv, generator=g)[:topk] for _ in range(s_q)]).int()
    idx[0] = -1                                  # nothing selected: out 0, lse -inf
    idx[1, 1:] = -1                              # one row
    idx[2, ::2] = -1                             # holes
    idx[3, :200] = -1                            # a whole first tile masked
    idx[4, 128:256] = -1                         # a whole middle tile masked
    out, lse = _check(q, kv, idx, 0.07, "padding")
    assert (out[0] == 0).all() and torch.isinf(lse[0]).all()


def test_running_maximum_moves_on_every_tile():
    """Keys ordered so that every tile of 128 holds a larger score than all tiles before it: the accumulator is
    rescaled on every tile, for every head."""
    g = torch.Generator().manual_seed(9)
    h, s_kv = 16, 1024
    kv = torch.randn(s_kv, 576, generator=g).bfloat16()
    q = torch.randn(3, h, 576, generator=g).bfloat16()
    scores = q[0, 0].float() @ kv.float().T
    order = scores.argsort()                     # ascending for head 0 of token 0
    idx = order[None, :].repeat(3, 1).int()
    idx[1] = order.flip(0).int()                 # descending: the maximum never moves after the first tile
    _check(q, kv, idx, 0.3, "stepped")


def test_bad_indices_are_reported_and_never_read():
    g = torch.Generator().manual_seed(2)
    q = torch.randn(2, 16, 576, generator=g).bfloat16().to(DEV)
    kv = torch.randn(64, 576, generator=g).bfloat16().to(DEV)
    idx = torch.randint(0, 64, (2, 40), generator=g).int()
    idx[1, 3] = 64
    with pytest.raises(RuntimeError):
        sparse_mla_fwd(q, kv, idx.to(DEV), 0.1, check=True, algo=2)
    idx[1, 3] = -7
    with pytest.raises(RuntimeError):
        sparse_mla_fwd(q, kv, idx.to(DEV), 0.1, check=True, algo=2)


def test_agrees_with_the_default_kernel_on_the_cpu_runnable_case():
    c = W.mla_cfg1()                             # S_q 128, h 16, topk 256, S_kv 4096
    q, kv, idx = c.q.to(DEV), c.kv.to(DEV), c.indices.to(DEV)
    o_few, l_few = sparse_mla_fwd(q, kv, idx, c.sm_scale, check=True, algo=2)
    o_def, l_def = sparse_mla_fwd(q, kv, idx, c.sm_scale, check=True)
    assert (o_few.float() - o_def.float()).abs().max().item() <= 2e-2
    assert ((l_few - l_def).abs() / l_def.abs().clamp(min=1)).max().item() <= 1e-3
    _check(c.q, c.kv, c.indices, c.sm_scale, c.name)


def test_more_than_32_heads_are_refused():
    q = torch.zeros(1, 33, 576, dtype=torch.bfloat16, device=DEV)
    kv = torch.zeros(8, 576, dtype=torch.bfloat16, device=DEV)
    idx = torch.zeros(1, 4, dtype=torch.int32, device=DEV)
    with pytest.raises((RuntimeError, ValueError)):
        sparse_mla_fwd(q, kv, idx, 0.1, algo=2)


@pytest.mark.parametrize("h,s_q,topk", [(16, 160, 200), (32, 40, 1000), (64, 9, 64), (100, 5, 700), (128, 60, 130), (32, 40, 600), (64, 160, 100), (16, 5, 2000),
                                         (64, 20, 1500)])
@pytest.mark.parametrize("steps", [False, True])
def test_bits_of_a_head_do_not_depend_on_the_heads_of_the_call(h, s_q, topk, steps):
    """The kernel for few heads, its groups of 64 and the pairs for many add in the same order: equal bits, also where maxima move in either
    half of a tile of the pairs (`steps`), where whole tiles are masked, and for tokens that select nothing."""
    g = torch.Generator().manual_seed(h + s_q + topk)
    s_kv = 1500
    q = torch.randn(s_q, h, 576, generator=g).bfloat16().to(DEV)
    kv = torch.randn(s_kv, 576, generator=g)
    if steps:
        kv *= torch.linspace(0.1, 20.0, s_kv)[:, None]
    kv = kv.bfloat16().to(DEV)
    idx = torch.stack([torch.randperm(s_kv, generator=g)[:topk] for _ in range(s_q)]).int().sort(dim=1).values
    idx[1, :] = -1
    idx[2, :64] = -1
    idx[3, 1::2] = -1
    idx[4, 40:] = -1
    idx = idx.to(DEV)
    reps = 1 + (400 + s_q - 1) // s_q                       # so many tokens that all heads of a call with more than 64 go to the pairs
    many, lse_many = sparse_mla_fwd(q.repeat(reps, 128 // h + 1, 1)[:, :128].contiguous(), kv, idx.repeat(reps, 1), 0.05, check=True, num_splits=1)
    out, lse = sparse_mla_fwd(q, kv, idx, 0.05, check=True, num_splits=1)
    assert torch.equal(out, many[:s_q, :h]) and torch.equal(lse, lse_many[:s_q, :h])


@pytest.mark.parametrize("h", [1, 16, 32, 64, 100, 128])
@pytest.mark.parametrize("batch,n_q,topk,page", [(3, 2, 300, 64), (160, 1, 65, 16), (2, 1, 64, 64), (5, 3, 1000, 7)])
def test_paged_rows_converted_in_the_gather(h, batch, n_q, topk, page):
    """e4m3 pages: whole tokens have the bits of the two-pass form (the same values, multiplied and added in the same order), parts of them its
    values; contexts shorter than the lists, padding inside a list, entries past the context, pages of odd sizes, several items per CTA."""
    from flagtree_b200 import sparse_mla_fwd_paged
    c = W.mla_cfg3(batch=batch, n_q=n_q, h=h, topk=topk, len_lo=30, len_hi=1500, page_size=page)
    c.indices[0, 0, 3::5] = -1
    c.indices[1, 0, :] = -1
    c.indices[-1, -1, 7] = 1 << 20                           # past the context: padding
    args = [t.to(DEV) for t in (c.q, c.kv_cache, c.kv_scale, c.block_table, c.context_lens, c.indices)]
    out, lse = sparse_mla_fwd_paged(*args, c.sm_scale, page_size=page, check=True, num_splits=1)
    ref_out, ref_lse = sparse_mla_fwd_paged(*args, c.sm_scale, page_size=page, check=True, num_splits=1, two_pass=True)
    assert torch.equal(out, ref_out) and torch.equal(lse, ref_lse)
    for kw in (dict(), dict(num_splits=3), dict(num_splits=1, two_pass=False)):
        o, l = sparse_mla_fwd_paged(*args, c.sm_scale, page_size=page, check=True, **kw)
        fin = torch.isfinite(ref_lse)
        assert torch.equal(torch.isfinite(l), fin)
        # P and the result are rounded to bf16 (2^-9 each) from another reference maximum and with sums in another order
        assert (o.float() - ref_out.float()).abs().max().item() <= 2 ** -7 * max(1.0, ref_out.abs().max().item())
        assert ((l[fin] - ref_lse[fin]).abs() <= 1e-5 * ref_lse[fin].abs().clamp(min=1)).all()


@pytest.mark.parametrize("h", [16, 64, 128])
@pytest.mark.parametrize("batch,topk,splits", [(3, 2048, 16), (2, 512, 8), (5, 300, 3), (4, 130, 1), (1, 1000, 40)])
def test_paged_parts_have_the_weights_of_the_one_cta_kernel(h, batch, topk, splits):
    """Parts of a token, and whole tokens of algo 0, take the true maximum tile by tile, in as many parts as the one-CTA kernel (algo 1) makes:
    the same weights in bf16.  Only the fp32 sums of the weights are added in another order (64 additions a tile, 2^-24 each, and as many tiles), which
    moves a result across a rounding boundary of bf16 in far less than one element of a hundred, and then to its neighbour (where the parts cancel:
    by their weights' 4e-6 of what they add up)."""
    c = W.mla_cfg3(batch=batch, n_q=1, h=h, topk=topk, len_lo=600, len_hi=4000)
    args = [t.to(DEV) for t in (c.q, c.kv_cache, c.kv_scale, c.block_table, c.context_lens, c.indices)]
    out, lse = paged_algo(args, c.sm_scale, c.page_size, 0, splits)
    ref_out, ref_lse = paged_algo(args, c.sm_scale, c.page_size, 1, splits)
    o, r = out.float(), ref_out.float()
    assert ((o - r).abs() <= 2 ** -7 * r.abs() + 2e-5 * r.abs().max()).all()
    assert (o != r).float().mean().item() < 0.01
    assert ((lse - ref_lse).abs() <= 2e-6 * ref_lse.abs().clamp(min=1)).all()


@pytest.mark.parametrize("h,topk,splits", [(16, 700, 4), (128, 300, 2), (64, 60, 3)])
def test_paged_parts_of_algo_5_take_the_true_maximum_too(h, topk, splits):
    """The lazy maximum is for whole tokens: scores that grow along the list, by less than its slack of 2^8 a tile, would show it in parts."""
    c = W.mla_cfg3(batch=3, n_q=1, h=h, topk=topk, len_lo=800, len_hi=2000)
    c.kv_scale.mul_(torch.linspace(0.5, 4.0, c.kv_scale.numel()))
    args = [t.to(DEV) for t in (c.q, c.kv_cache, c.kv_scale, c.block_table, c.context_lens, c.indices.sort(dim=2).values)]
    ref = paged_algo(args, c.sm_scale, c.page_size, 0, splits)
    got = paged_algo(args, c.sm_scale, c.page_size, 5, splits)
    assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])
