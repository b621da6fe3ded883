"""Query batches longer than one launch of the persistent sparse-MLA kernels walks through.

A launch gives every CTA of the kernel for few heads, and every CTA pair of the kernel for many, at most 64 items (tokens, or parts of
tokens of 64 heads); a longer batch becomes several launches over consecutive token ranges, each with its own offsets into q,
indices, out and lse, and for the paged form into the sequences.  Long prefill is the normal case for sparse attention, so the range
arithmetic gets tests of its own: a little more than one launch takes, compared token by token with a code path that has
no notion of token ranges and, on a sample of tokens from both ranges, with the CPU oracle.  Causal top-k with -1 padding, so the first
tokens of the batch are short and the rest full.
"""
import pytest
import torch

from conftest import LSE_RTOL, OUT_ATOL

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from flagtree_b200 import sparse_mla_fwd, sparse_mla_fwd_paged
    from flagtree_b200 import workloads as W
from oracle.sparse_mla_ref import sparse_mla_fwd_ref

DEV = "cuda:0"
SMS = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 148
ITEMS = 64                                       # per CTA, or pair of CTAs, and launch


@pytest.mark.parametrize("h,per_launch", [(128, SMS // 2 * ITEMS), (16, SMS * ITEMS)])
def test_more_tokens_than_one_launch_takes(h, per_launch):
    s_q = per_launch + 200
    c = W.mla_cfg2(device=DEV, s_q=s_q, s_kv=2048, h=h, topk=128)
    out, lse = sparse_mla_fwd(c.q, c.kv, c.indices, c.sm_scale, check=True)
    ref_out, ref_lse = sparse_mla_fwd(c.q, c.kv, c.indices, c.sm_scale, check=True, algo=1)
    torch.cuda.synchronize()
    # every token against the per-token kernel (both are within OUT_ATOL of the oracle, so 2 x between them)
    d_out = (out.float() - ref_out.float()).abs().amax(dim=(1, 2))
    fin = torch.isfinite(ref_lse)
    assert torch.equal(torch.isfinite(lse), fin)
    d_lse = ((lse - ref_lse).abs() / ref_lse.abs().clamp(min=1.0)).masked_fill(~fin, 0.0).amax(dim=1)
    worst = int(d_out.argmax())
    assert d_out.max().item() <= 2 * OUT_ATOL, f"token {worst}: out differs by {d_out.max().item():.4f}"
    assert d_lse.max().item() <= 2 * LSE_RTOL, f"token {int(d_lse.argmax())}: lse differs by {d_lse.max().item():.2e}"
    # a sample from both token ranges against the oracle
    sample = torch.tensor([0, 1, 63, 64, 2047, per_launch - 1, per_launch, per_launch + 1, per_launch + 64, s_q - 1])
    o_ref, l_ref = sparse_mla_fwd_ref(c.q[sample].cpu(), c.kv.cpu(), c.indices[sample].cpu(), c.sm_scale)
    e_out = (out[sample].float().cpu() - o_ref).abs().max().item()
    e_lse = ((lse[sample].cpu() - l_ref).abs() / l_ref.abs().clamp(min=1.0)).max().item()
    assert e_out <= OUT_ATOL and e_lse <= LSE_RTOL, f"vs oracle: out {e_out:.4f}, lse {e_lse:.2e}"


@pytest.mark.parametrize("h,batch,topk,splits", [(16, 16, 64, None), (128, 8, 64, None), (128, 40, 2048, 16)])
def test_more_paged_tokens_than_one_launch_takes(h, batch, topk, splits):
    """Every sequence has pages and a length of its own, and the launch boundary lies inside one: a token of a later launch that took the
    table of another sequence would differ.  The two-pass form resolves the rows of all tokens in one launch."""
    per_launch = SMS * ITEMS // ((splits or 1) * -(-h // 64))
    n_q = per_launch // batch + 2
    if per_launch % n_q == 0:
        n_q += 1
    assert batch * n_q > per_launch and per_launch % n_q != 0
    c = W.mla_cfg3(device=DEV, batch=batch, n_q=n_q, h=h, topk=topk, len_lo=100, len_hi=3000)
    args = (c.q, c.kv_cache, c.kv_scale, c.block_table, c.context_lens, c.indices, c.sm_scale)
    out, lse = sparse_mla_fwd_paged(*args, page_size=c.page_size, check=True, num_splits=splits)
    ref_out, ref_lse = sparse_mla_fwd_paged(*args, page_size=c.page_size, check=True, num_splits=1, two_pass=True)
    if splits is None:
        assert torch.equal(out, ref_out) and torch.equal(lse, ref_lse)       # whole tokens: the same values in the same order
    else:
        # weights and results are rounded to bf16 (2^-9 each) from other reference maxima
        assert (out.float() - ref_out.float()).abs().max().item() <= 2 ** -7 * max(1.0, ref_out.abs().max().item())
        assert ((lse - ref_lse).abs() <= 1e-5 * ref_lse.abs().clamp(min=1)).all()
