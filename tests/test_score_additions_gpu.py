"""Logits soft cap, ALiBi and bias of the tcgen05 softmax where its forms change: scores inside and outside half a cap (the
polynomial and the quotient form of tanh, chosen per warp and tile), tiles left of the diagonal and on it, rows and keys that
no tile divides, bias rows at odd addresses."""
import pytest
import torch

from flashck_b200 import _lib, ops
from tests.helpers import assert_lse_close, assert_o_close

pytestmark = pytest.mark.gpu


def _reference(q, k, v, causal, window, cap, slopes, bias):
    b, n, hq, d = q.shape
    m, group = k.shape[1], hq // k.shape[2]
    kk, vv = (t.double().repeat_interleave(group, 2) for t in (k, v))
    x = torch.einsum("bqhd,bkhd->bhqk", q.double(), kk) * d ** -0.5
    if cap > 0:
        x = cap * torch.tanh(x / cap)
    i, j = torch.arange(n, device=q.device)[:, None] + (m - n), torch.arange(m, device=q.device)
    if slopes is not None:
        x = x - slopes.double()[:, :, None, None] * (i - j).abs()
    if bias is not None:
        x = x + bias.double()
    if causal:
        x = x.masked_fill(j > i, float("-inf"))
    if window >= 0:
        x = x.masked_fill(j < i - window, float("-inf"))
    lse = torch.logsumexp(x, -1)
    return torch.einsum("bhqk,bkhd->bqhd", torch.softmax(x, -1), vv).float(), lse.float()


# size of the queries: all scores near 0; the largest a little inside / outside half the cap; most of them far outside
@pytest.mark.parametrize("size", [0.01, 1.0, 2.6, 4.0, 40.0])
@pytest.mark.parametrize("d,n,m", [(128, 128, 128), (128, 257, 389), (64, 127, 640), (128, 1, 129), (64, 300, 300)])
@pytest.mark.parametrize("add", ["cap", "cap+alibi", "alibi", "cap+bias", "bias"])
@pytest.mark.parametrize("causal,window", [(True, -1), (True, 100), (False, -1)])
def test_score_additions(size, d, n, m, add, causal, window):
    g = torch.Generator(device="cuda").manual_seed(n + m)
    q, k, v = (torch.randn((2, s, h, d), generator=g, device="cuda") for s, h in ((n, 6), (m, 2), (m, 2)))
    q = (q * size).to(torch.bfloat16)
    k, v = k.bfloat16(), v.bfloat16()
    cap = 20.0 if "cap" in add else 0.0
    slopes = (2.0 ** -torch.arange(1, 7, device="cuda").float())[None] if "alibi" in add else None
    bias = torch.randn((1, 6, n, m), generator=g, device="cuda").bfloat16() if "bias" in add else None
    if bias is not None:
        bias[:, :, :, m // 2] = float("-inf")  # a key that the bias hides
    o, lse = ops.fmha_fwd(q, k, v, causal=causal, window_size=(window, 0) if window >= 0 else (-1, -1), logits_soft_cap=cap,
                          alibi_slopes=slopes, bias=bias, return_lse=True)
    assert bias is not None and d == 64 or _lib.get_instance_param(0, "last_instance") == 1
    o_ref, lse_ref = _reference(q, k, v, causal, window, cap, slopes, bias)
    assert_o_close(o, o_ref)
    assert_lse_close(lse, lse_ref)


# The polynomial holds for |score| <= cap / 2 whichever sign the scale has; scores here reach three caps and more.
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("add", ["cap", "cap+alibi", "cap+bias"])
@pytest.mark.parametrize("packed", [False, True])
def test_soft_cap_with_a_negative_scale(d, add, packed):
    n, m, cap, scale = 300, 300, 20.0, -d ** -0.5
    g = torch.Generator(device="cuda").manual_seed(d)
    q, k, v = (torch.randn((2, s, h, d), generator=g, device="cuda").bfloat16() for s, h in ((n, 6), (m, 2), (m, 2)))
    q = q * 20
    slopes = (2.0 ** -torch.arange(1, 7, device="cuda").float())[None] if "alibi" in add else None
    bias = torch.randn((1, 6, n, m), generator=g, device="cuda").bfloat16() if "bias" in add else None
    more = dict(causal=True, scale=scale, logits_soft_cap=cap, alibi_slopes=slopes, return_lse=True)
    if packed:
        cu = torch.tensor([0, n, 2 * n], device="cuda")
        if bias is not None:  # (packed: one plane over the packed totals)
            more["bias"] = torch.nn.functional.pad(torch.cat([bias, bias], 2), (0, m))
            more["bias"][:, :, n:, m:] = bias
        o, lse = ops.fmha_fwd_var_len(q.flatten(0, 1), k.flatten(0, 1), v.flatten(0, 1), cu, cu, n, **more)
        o, lse = o.view(2, n, 6, d), lse.view(6, 2, n).transpose(0, 1)
    else:
        o, lse = ops.fmha_fwd(q, k, v, bias=bias, **more)
    o_ref, lse_ref = _reference(-q, k, v, True, -1, cap, slopes, bias)
    assert_o_close(o, o_ref)
    assert_lse_close(lse, lse_ref)
