"""The hdim-128 prefill kernel's work list: every query row of every sequence is computed once, whichever way the list is made."""
import pytest
import torch

from flashck_b200 import _lib, ops
from flashck_b200.utils.inputs import to_seqstarts, uniform_seqlens
from tests.helpers import assert_lse_close, assert_o_close

pytestmark = pytest.mark.gpu


def _reference(q, k, v, nq, nk, causal, window=-1, bias=None):
    o, lse, group = torch.empty(q.shape, device=q.device), torch.empty((q.shape[1], q.shape[0]), device=q.device), q.shape[1] // k.shape[1]
    a = c = 0
    for n, m in zip(nq, nk):
        kk, vv = (t[c:c + m].float().repeat_interleave(group, 1) for t in (k, v))
        x = torch.einsum("qhd,khd->hqk", q[a:a + n].float(), kk) * q.shape[2] ** -0.5
        if bias is not None:  # over the packed totals
            x += bias[0, :, a:a + n, c:c + m].float()
        if causal:
            x.masked_fill_(torch.arange(m, device=q.device) > torch.arange(n, device=q.device)[:, None] + (m - n), float("-inf"))
        if window >= 0:
            x.masked_fill_(torch.arange(m, device=q.device) < torch.arange(n, device=q.device)[:, None] + (m - n - window), float("-inf"))
        lse[:, a:a + n] = torch.logsumexp(x, -1)
        o[a:a + n] = torch.einsum("hqk,khd->qhd", torch.softmax(x, -1), vv)
        a, c = a + n, c + m
    return o, lse


# batch, longest query, heads: a handful of items; lists dealt by load (2-16 rounds); 511 - 513 row blocks, the edge of the
# sorted table; one block per sequence at the largest batch; more than 16 rounds in snake order; far more row blocks than
# the table holds
@pytest.mark.parametrize("batch,lo,hi,hq,hkv", [
    (1, 1, 1, 8, 8), (3, 1, 700, 8, 2), (37, 1, 900, 8, 2), (37, 1, 900, 12, 4), (256, 1, 128, 4, 2),
    (256, 129, 256, 2, 1), (171, 257, 384, 2, 1), (170, 257, 384, 6, 2), (64, 900, 1000, 12, 4), (64, 900, 1000, 12, 2), (250, 300, 500, 8, 2),
])
@pytest.mark.parametrize("causal,more", [(True, 0), (False, 0), (True, 1500)])
def test_every_row_once(batch, lo, hi, hq, hkv, causal, more):
    if more and batch > 40:
        pytest.skip("(the mask and the list do not depend on both)")
    nq = uniform_seqlens(batch, lo, hi, batch + hi)
    nk = [n + e for n, e in zip(nq, uniform_seqlens(batch, 0, more, 3))] if more else nq
    g = torch.Generator(device="cuda").manual_seed(batch)
    q, k, v = (torch.randn((sum(n), h, 128), generator=g, device="cuda").bfloat16() for n, h in ((nq, hq), (nk, hkv), (nk, hkv)))
    cu_q, cu_k = to_seqstarts(nq).cuda(), to_seqstarts(nk).cuda()
    o, lse = ops.fmha_fwd_var_len(q, k, v, cu_q, cu_k, max(nq), causal=causal, return_lse=True)
    assert _lib.device_status() == 0
    o_ref, lse_ref = _reference(q, k, v, nq, nk, causal)
    assert_o_close(o, o_ref)
    assert_lse_close(lse, lse_ref)


# Sequence starts whose unused tail holds zeros: the sequence behind the last valid one ends before it begins.  It has no rows,
# and the others are computed as if it were not there, whichever form the list takes (one item per SM at most; sorted; by level).
@pytest.mark.parametrize("nq,hq,hkv,d", [([300, 400], 4, 2, 128), ([300, 900, 1], 64, 8, 128), ([700] * 120, 8, 2, 128), ([300, 400], 3, 1, 128),
                                         ([300, 900, 1], 64, 8, 64)])
@pytest.mark.parametrize("bias", [False, True])
def test_starts_with_a_zero_tail(nq, hq, hkv, d, bias):
    if bias and (d == 64 or sum(nq) > 2000):
        pytest.skip("(the list of the bias instances: the short ones)")
    g = torch.Generator(device="cuda").manual_seed(len(nq))
    q, k, v = (torch.randn((sum(nq), h, d), generator=g, device="cuda").bfloat16() for h in (hq, hkv, hkv))
    more = {"causal": True, "return_lse": True}
    if bias:
        more["bias"] = torch.randn((1, hq, sum(nq), sum(nq)), generator=g, device="cuda").bfloat16()
    cu = to_seqstarts(nq).cuda()
    padded = torch.cat([cu, torch.zeros(5, dtype=cu.dtype, device="cuda")])
    o, lse = ops.fmha_fwd_var_len(q, k, v, padded, padded, max(nq), **more)
    assert _lib.device_status() == 0
    o_ref, lse_ref = ops.fmha_fwd_var_len(q, k, v, cu, cu, max(nq), **more)
    assert torch.equal(o, o_ref) and torch.equal(lse, lse_ref)


# Equal lengths, whose order is known in closed form: several rounds of items, batches above 2, paired and unpaired heads, even
# and odd numbers of row tiles (unpaired and odd: a last block of one tile), with the orders by block (mask or bias) and by
# sequence (neither).
@pytest.mark.parametrize("batch,n,hq,hkv", [(5, 700, 32, 8), (5, 600, 24, 8), (7, 900, 24, 8), (3, 1200, 32, 32), (4, 1100, 40, 8),
                                            (21, 129, 16, 2), (160, 100, 3, 1)])
@pytest.mark.parametrize("causal,window", [(False, -1), (True, -1), (True, 200)])
@pytest.mark.parametrize("bias", [None, 0, 1])
def test_equal_lengths(batch, n, hq, hkv, causal, window, bias):
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v = (torch.randn((batch, n, h, 128), generator=g, device="cuda").bfloat16() for h in (hq, hkv, hkv))
    b = torch.randn((1, hq if bias else 1, n, n), generator=g, device="cuda").bfloat16() if bias is not None else None
    o, lse = ops.fmha_fwd(q, k, v, causal=causal, window_size=(window, 0) if window >= 0 else (-1, -1), bias=b, return_lse=True)
    assert _lib.device_status() == 0 and _lib.get_instance_param(0, "last_instance") == 1
    for i in range(batch):
        o_ref, lse_ref = _reference(q[i], k[i], v[i], [n], [n], causal, window, b)
        assert_o_close(o[i], o_ref)
        assert_lse_close(lse[i], lse_ref)


# a bias over packed sequences with more items than SMs (the list of the bias instances by level)
@pytest.mark.parametrize("hq,hkv", [(32, 8), (40, 8)])
@pytest.mark.parametrize("causal", [False, True])
def test_packed_bias_over_several_rounds(hq, hkv, causal):
    nq = [300, 650, 1, 411]
    g = torch.Generator(device="cuda").manual_seed(hq)
    q, k, v = (torch.randn((sum(nq), h, 128), generator=g, device="cuda").bfloat16() for h in (hq, hkv, hkv))
    b = torch.randn((1, hq, sum(nq), sum(nq)), generator=g, device="cuda").bfloat16()
    cu = to_seqstarts(nq).cuda()
    o, lse = ops.fmha_fwd_var_len(q, k, v, cu, cu, max(nq), causal=causal, bias=b, return_lse=True)
    assert _lib.device_status() == 0 and _lib.get_instance_param(0, "last_instance") == 1
    o_ref, lse_ref = _reference(q, k, v, nq, nq, causal, bias=b)
    assert_o_close(o, o_ref)
    assert_lse_close(lse, lse_ref)


# The longest list a CTA can hold (1024 items), sorted and dealt, and one sequence more: that call leaves for the general instance.
@pytest.mark.parametrize("over", [0, 1])
def test_longest_list(over):
    sms, heads = torch.cuda.get_device_properties(0).multi_processor_count, 1023
    batch = sms * 1024 // heads + over
    nq = [1 + i % 2 for i in range(batch)]
    nk = [n + i % 3 for i, n in enumerate(nq)]
    g = torch.Generator(device="cuda").manual_seed(batch)
    q, k, v = (torch.randn((sum(n), heads, 128), generator=g, device="cuda").bfloat16() for n in (nq, nk, nk))
    o, lse = ops.fmha_fwd_var_len(q, k, v, to_seqstarts(nq).cuda(), to_seqstarts(nk).cuda(), max(nq), causal=True, return_lse=True)
    assert _lib.get_instance_param(0, "last_instance") == 1 - over
    assert _lib.device_status() == 0
    o_ref, lse_ref = _reference(q, k, v, nq, nk, True)
    assert_o_close(o, o_ref)
    assert_lse_close(lse, lse_ref)
