"""Decode where its forms change: kv heads per CTA, several groups of heads, the slots of unused splits, and the merge of two rows per
warp."""
import pytest
import torch

from flashck_b200 import _lib, ops
from flashck_b200.utils.inputs import make_paged_cache, normal_tensor
from tests.helpers import assert_lse_close, assert_o_close

pytestmark = pytest.mark.gpu


def _reference(q, c, lens):
    b, n, hq, d = q.shape
    o, lse = torch.zeros(b, n, hq, d, dtype=torch.float64), torch.full((b, hq, n), float("-inf"), dtype=torch.float64)
    for i, m in enumerate(lens):
        if m == 0:
            continue
        pages = c.block_table[i, :-(-m // c.k.shape[1])].long()
        k, v = (x[pages].flatten(0, 1)[:m].double().repeat_interleave(hq // x.shape[2], 1) for x in (c.k, c.v))
        x = torch.einsum("qhd,khd->hqk", q[i].double(), k) * d ** -0.5
        if n > 1:
            x = x.masked_fill(torch.arange(m) > torch.arange(n)[:, None] + (m - n), float("-inf"))
        lse[i] = torch.logsumexp(x, -1)
        o[i] = torch.einsum("hqk,khd->qhd", torch.softmax(x, -1), v)
    return o, lse


# one tile, one tile per CTA and fewer, several; an empty sequence; more sequences than CTAs share out
@pytest.mark.parametrize("lens", [[1], [16], [500], [3000], [17, 0, 900], [40] * 90, [33] * 170])
@pytest.mark.parametrize("hq,hkv,d", [(32, 8, 128), (16, 16, 128), (12, 12, 64), (8, 2, 128)])
@pytest.mark.parametrize("tokens,splits", [(1, 0), (1, 128), (4, 7)])
def test_heads_and_unused_splits(lens, hq, hkv, d, tokens, splits):
    if min(lens) == 1 and tokens > 1:
        lens = [tokens]
    c = make_paged_cache(lens, hkv, d, d, 16, torch.bfloat16, seed=3)
    q = normal_tensor((len(lens), tokens, hq, d), torch.bfloat16, 4)
    dev = {"seqlen_k": c.seqlen_k.cuda(), "block_table": c.block_table.cuda(), "causal": tokens > 1}
    S = splits or ops.default_num_splits(len(lens), rows_per_kv_head=tokens * hq // hkv)
    work = (torch.full((len(lens), hq, S, tokens), float("nan"), device="cuda"),
            torch.full((len(lens), hq, S, tokens, d), float("nan"), device="cuda"))
    for heads in (0, 4):
        _lib.set_instance_param(2, "heads_per_cta", heads)
        try:
            lse_acc, o_acc = ops.fmha_fwd_splitkv(q.cuda(), c.k.cuda(), c.v.cuda(), workspace=work, combine=False, **dev)
        finally:
            _lib.set_instance_param(2, "heads_per_cta", 0)
        assert not torch.isnan(lse_acc).any()  # every slot is written, those without keys with -inf
        o, lse = ops.fmha_fwd_splitkv_combine(lse_acc, o_acc, torch.bfloat16, return_lse=True)
        o_ref, lse_ref = _reference(q, c, lens)
        assert_o_close(o, o_ref)
        assert_lse_close(lse, lse_ref)
        for t in work:
            t.fill_(float("nan"))


# two rows per warp: an odd number of rows, slots of empty splits full of NaN, rows without any split beside rows with all
@pytest.mark.parametrize("S", [1, 2, 3, 4, 5, 15, 16])
@pytest.mark.parametrize("rows,hq,dv", [(1, 1, 128), (3, 5, 128), (7, 3, 64), (33, 4, 68), (1, 3, 4)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_merge_of_two_rows_per_warp(S, rows, hq, dv, dtype):
    g = torch.Generator().manual_seed(S * 100 + rows)
    lse_acc = torch.randn((2, hq, S, rows), generator=g)
    o_acc = torch.randn((2, hq, S, rows, dv), generator=g)
    used = torch.randint(0, S + 1, (2, hq, 1, rows), generator=g)
    used.view(-1)[0] = 0
    empty = torch.arange(S)[None, None, :, None] >= used
    lse_acc[empty] = float("-inf")
    o_acc[empty] = float("nan")
    o, lse = ops.fmha_fwd_splitkv_combine(lse_acc.cuda(), o_acc.cuda(), dtype, return_lse=True)
    w = torch.softmax(lse_acc.double(), 2).nan_to_num()[..., None]
    ref = (w * o_acc.double().masked_fill(empty[..., None], 0.0)).sum(2).permute(0, 2, 1, 3)
    assert_o_close(o, ref)
    assert_lse_close(lse, torch.logsumexp(lse_acc.double(), 2))
    if dtype == torch.float32:  # 16 products and sums in fp32, weights of expf (2 ulp) and one division
        assert (o.cpu().double() - ref).abs().max() < 2e-6 * 5
