"""The split forms of the tcgen05 kernel where O is rescaled: a row's maximum that grows by more than 2^8 from tile to tile, for every
row or for one row of a warp, with duplicated rows (up to 64 per kv head) and without, masked and unmasked."""
import pytest
import torch

from flashck_b200 import ops
from tests.helpers import assert_lse_close, assert_o_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,hq,hkv", [(5, 8, 2), (16, 8, 2), (17, 8, 2), (32, 8, 2), (8, 32, 2)])
@pytest.mark.parametrize("jump", [6.0, 9.0, 40.0])
@pytest.mark.parametrize("rows", ["all", "one"])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_growing_maximum(tokens, hq, hkv, jump, rows, causal, dtype):
    n, d, lens = 1500, 128, [1500, 700]
    g = torch.Generator(device="cuda").manual_seed(tokens)
    q, k, v = (torch.randn((2, s, h, d), generator=g, device="cuda").to(dtype) for s, h in ((tokens, hq), (n, hkv), (n, hkv)))
    k[..., 0] = torch.arange(n, device="cuda").div(128, rounding_mode="floor")[None, :, None] * (jump * d ** 0.5 / 16 / 1.4427)
    q[..., 0] = 16.0
    if rows == "one":  # packed rows: tokens outside, the heads of a group inside
        flat = torch.arange(tokens * hq, device="cuda").view(tokens, hq)
        q[:, flat % 32 != 5, 0] = 0.0
    o, lse = ops.fmha_fwd_splitkv(q, k, v, seqlen_k=torch.tensor(lens, dtype=torch.int32, device="cuda"), causal=causal, return_lse=True)
    for b, m in enumerate(lens):
        kk, vv = (t[b, :m].double().repeat_interleave(hq // hkv, 1) for t in (k, v))
        x = torch.einsum("qhd,khd->hqk", q[b].double(), kk) * d ** -0.5
        if causal:
            x = x.masked_fill(torch.arange(m, device="cuda") > torch.arange(tokens, device="cuda")[:, None] + (m - tokens), float("-inf"))
        assert_o_close(o[b], torch.einsum("hqk,khd->qhd", torch.softmax(x, -1), vv))
        assert_lse_close(lse[b], torch.logsumexp(x, -1))
