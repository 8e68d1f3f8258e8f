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


# What a row computes depends on nothing but the row and the keys it sees: not on the form that the other scores of its warp
# or its tile ask for.  Changed here: keys that are masked for a row, other rows, the packed sequence behind.
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("add", ["cap", "cap+alibi", "cap+bias"])
def test_capped_rows_are_independent(d, add):
    n, cap, cut = 300, 20.0, 203
    g = torch.Generator(device="cuda").manual_seed(d)
    q, k, v = (torch.randn((1, n, h, d), generator=g, device="cuda").bfloat16() for h in (6, 2, 2))
    slopes = (2.0 ** -torch.arange(1, 7, device="cuda").float())[None] if "alibi" in add else None
    bias = torch.randn((1, 6, n, n), generator=g, device="cuda").bfloat16() if "bias" in add else None
    more = dict(causal=True, logits_soft_cap=cap, alibi_slopes=slopes, return_lse=True)
    o, lse = ops.fmha_fwd(q, k, v, bias=bias, **more)
    # later tokens whose scores lie far beyond the cap, as queries and as keys
    q2, k2 = q.clone(), k.clone()
    q2[:, cut:] *= 30
    k2[:, cut:] *= 30
    o2, lse2 = ops.fmha_fwd(q2, k2, v, bias=bias, **more)
    assert torch.equal(o2[:, :cut], o[:, :cut]) and torch.equal(lse2[:, :, :cut], lse[:, :, :cut])
    # single rows in the middle of the warps
    q3 = q.clone()
    q3[:, 7::16] *= 30
    same = torch.arange(n, device="cuda") % 16 != 7
    o3, lse3 = ops.fmha_fwd(q3, k, v, bias=bias, **more)
    assert torch.equal(o3[:, same], o[:, same]) and torch.equal(lse3[:, :, same], lse[:, :, same])
    if bias is None:  # two packed sequences, the second one changed
        cu = torch.tensor([0, cut, n], device="cuda")
        a, la = ops.fmha_fwd_var_len(q[0], k[0], v[0], cu, cu, cut, **more)
        b, lb = ops.fmha_fwd_var_len(q2[0], k2[0], v[0], cu, cu, cut, **more)
        assert torch.equal(a[:cut], b[:cut]) and torch.equal(la[:, :cut], lb[:, :cut])


# One key per sequence and one channel in use: the LSE of a row is its capped score, and the score is exact before the cap.
# Queries of all sizes from 1e-3 to 4 caps stand side by side in a warp, or each size in warps of its own; the caps reach both
# ends of the range in which the polynomial's coefficients hold powers of scale / cap.
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("scale", [0.0884, 1.0, -0.0884])
@pytest.mark.parametrize("cap", [1e-5, 0.05, 1.0, 20.0, 900.0, 2e3, 1e4, 1e5, 1e6, 1e9])
@pytest.mark.parametrize("mixed", [False, True])
def test_capped_score_in_fp32(d, scale, cap, mixed):
    n = 512
    x = torch.logspace(-3, 0.6, n, dtype=torch.float64, device="cuda") * (cap / scale)
    x[::2] *= -1
    if mixed:
        x = x[torch.randperm(n, generator=torch.Generator().manual_seed(3)).cuda()]
    q = torch.zeros((1, n, 2, d), dtype=torch.bfloat16, device="cuda")
    q[0, :, :, 0] = x.bfloat16()[:, None]
    k = torch.zeros((1, 1, 2, d), dtype=torch.bfloat16, device="cuda")
    k[0, 0, :, 0] = 1.0
    _, lse = ops.fmha_fwd(q, k, k, scale=scale, logits_soft_cap=cap, return_lse=True)
    s32 = float(torch.tensor(scale)), float(torch.tensor(cap))
    ref = s32[1] * torch.tanh(q[0, :, :, 0].double().T * s32[0] / s32[1])
    # polynomial: 3e-8 of its own and about 8 roundings; quotient: 2^-22 of its exponential, twice that at most in 1 - e with
    # e <= 1 / e, the roundings of the exponent (<= 8 * 2^-24 of a term below 0.6) and of the division; then the LSE's two
    rel = ((lse[0].double() - ref) / ref).abs().max()
    assert float(rel) <= 24 * 2.0 ** -24, float(rel)
