"""A bias tensor through shared memory (whole rows of 16-byte pieces) against the form that fetches it in the softmax threads, which
the same values in a buffer that starts one element later take: the arithmetic is the same, so the bits are."""
import pytest
import torch

from flashck_b200 import _lib, ops
from tests.helpers import assert_lse_close, assert_o_close

pytestmark = pytest.mark.gpu


def _shifted(t):
    """The same contiguous tensor at an address that is no multiple of 16."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    buf[1:] = t.flatten()
    return buf[1:].view(t.shape)


# rows around the tile's edges; one box, boxes that the row ends in, several tiles; pairs of heads and pairs of row tiles
@pytest.mark.parametrize("n", [1, 127, 130, 300])
@pytest.mark.parametrize("m", [64, 72, 136, 264, 640])
@pytest.mark.parametrize("rank", [0, 1, 2])
@pytest.mark.parametrize("mask", ["none", "causal", "window"])
@pytest.mark.parametrize("hq,hkv,dtype", [(4, 2, torch.bfloat16), (3, 3, torch.float16)])
def test_same_bits(n, m, rank, mask, hq, hkv, dtype):
    g = torch.Generator(device="cuda").manual_seed(n + m)
    q, k, v = (torch.randn((2, s, h, 128), generator=g, device="cuda").to(dtype) for s, h in ((n, hq), (m, hkv), (m, hkv)))
    bias = torch.randn((2 if rank == 2 else 1, hq if rank else 1, n, m), generator=g, device="cuda").to(dtype)
    bias[:, :, :, m // 2] = float("-inf")  # a key that the bias hides
    kw = {"causal": mask != "none", "window_size": (40, 0) if mask == "window" else (-1, -1), "return_lse": True}
    o, lse = ops.fmha_fwd(q, k, v, bias=bias, **kw)
    assert _lib.get_instance_param(0, "last_instance") == 1
    o2, lse2 = ops.fmha_fwd(q, k, v, bias=_shifted(bias), **kw)
    assert torch.equal(o, o2) and torch.equal(lse, lse2)
    x = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double().repeat_interleave(hq // hkv, 2)) * 128 ** -0.5 + bias.double()
    i, j = torch.arange(n, device="cuda")[:, None] + (m - n), torch.arange(m, device="cuda")
    if mask != "none":
        x = x.masked_fill(j > i, float("-inf"))
    if mask == "window":
        x = x.masked_fill(j < i - 40, float("-inf"))
    ref = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(x, -1).nan_to_num(), v.double().repeat_interleave(hq // hkv, 2))
    assert_o_close(o, ref)
    assert_lse_close(lse, torch.logsumexp(x, -1))


# a soft cap in front of the bias, several items per SM (the rings run on from item to item), and what the bias leaves of a row:
# the type's lowest value, everything hidden, infinities
@pytest.mark.parametrize("cap", [0.0, 20.0])
@pytest.mark.parametrize("kind", ["values", "lowest", "hidden row", "inf"])
def test_many_items(cap, kind):
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn((3, s, h, 128), generator=g, device="cuda").bfloat16() for s, h in ((1000, 16), (520, 8), (520, 8)))
    bias = torch.randn((1, 16, 1000, 520), generator=g, device="cuda").bfloat16()
    if kind == "lowest":
        bias[..., ::3] = torch.finfo(torch.bfloat16).min
    if kind == "hidden row":
        bias[:, :, 77::100] = float("-inf")
    if kind == "inf":
        bias[:, 1, 500, 7] = float("inf")
    o, lse = ops.fmha_fwd(q, k, v, bias=bias, logits_soft_cap=cap, return_lse=True)
    o2, lse2 = ops.fmha_fwd(q, k, v, bias=_shifted(bias), logits_soft_cap=cap, return_lse=True)
    assert torch.equal(o.view(torch.int16), o2.view(torch.int16)) and torch.equal(lse.view(torch.int32), lse2.view(torch.int32))
