"""The merge of split partials at the sizes where its number of warps per row changes."""
import pytest
import torch

from flashck_b200 import ops

pytestmark = pytest.mark.gpu


# (batch, heads, rows): below and above the row counts up to which a row gets 16, 8 and 4 warps (148, 296 and 592 rows on
# 148 SMs); the split counts are the ones at which each form starts, one row of 32 weights per warp overflows, and a few odd ones
@pytest.mark.parametrize("bhr", [(1, 3, 1), (2, 12, 4), (1, 37, 4), (1, 149, 1), (8, 37, 1), (1, 297, 1), (1, 296, 2), (1, 593, 1)])
@pytest.mark.parametrize("S", [8, 9, 16, 17, 32, 33, 75, 128, 129, 515])
@pytest.mark.parametrize("dv", [64, 128, 256, 20])
def test_combine_over_row_and_split_counts(bhr, S, dv):
    b, h, r = bhr
    g = torch.Generator(device="cuda").manual_seed(b * 1000 + h * 10 + S)
    lse_acc = torch.randn((b, h, S, r), generator=g, device="cuda") * 3
    o_acc = torch.randn((b, h, S, r, dv), generator=g, device="cuda")
    empty = torch.rand((b, h, S, r), generator=g, device="cuda") < 0.4  # splits without keys: their partials are never used
    empty[:, 0] |= (torch.arange(S, device="cuda") >= (S + 1) // 2)[None, :, None]
    empty[0, h - 1, :, 0] = True  # a row no split saw a key of
    lse_acc[empty] = float("-inf")
    o_acc[empty] = float("nan")
    w = torch.softmax(lse_acc.double(), 2).nan_to_num(0.0)
    o64 = torch.where(empty[..., None], 0.0, o_acc.double())
    ref = (w[..., None] * o64).sum(2).permute(0, 2, 1, 3)
    size = (w[..., None] * o64.abs()).sum(2).permute(0, 2, 1, 3)
    lse64 = torch.logsumexp(lse_acc.double(), 2)
    o, lse = ops.fmha_fwd_splitkv_combine(lse_acc, o_acc, torch.float32, return_lse=True)
    # S fp32 additions, and weights off by the rounding of an exponent below 32 and a few units of expf and the division
    assert bool(((o.double() - ref).abs() <= (S + 48) * 2.0 ** -24 * size).all())
    dead = torch.isinf(lse64)
    assert torch.equal(torch.isinf(lse), dead)
    assert bool(((lse.double() - lse64).abs()[~dead] <= 1e-5).all())
    half = ops.fmha_fwd_splitkv_combine(lse_acc, o_acc, torch.bfloat16)
    assert torch.equal(half, o.to(torch.bfloat16))
