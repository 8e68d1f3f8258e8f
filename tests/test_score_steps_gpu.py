"""The step of the softmax with score additions, which has one copy for masked and unmasked tiles: ALiBi, a logits soft cap or both, where
tiles begin and end, with rows whose maximum grows by more than 2^8 from tile to tile (O is rescaled)."""
import pytest
import torch

from flashck_b200 import _lib, ops
from tests.helpers import assert_lse_close, assert_o_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(1, 1), (96, 97), (128, 128), (129, 225), (200, 128), (300, 640)])
@pytest.mark.parametrize("left,right", [(-1, -1), (-1, 0), (31, 0), (40, 33), (150, -1), (300, 0)])
@pytest.mark.parametrize("add", ["alibi", "cap", "alibi+cap"])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("grow", [False, True])
@pytest.mark.parametrize("hq,hkv,dtype", [(4, 2, torch.bfloat16), (3, 3, torch.float16)])
def test_steps(n, m, left, right, add, d, grow, hq, hkv, dtype):
    g = torch.Generator(device="cuda").manual_seed(n + m)
    q, k, v = (torch.randn((2, s, h, d), generator=g, device="cuda").to(dtype) for s, h in ((n, hq), (m, hkv), (m, hkv)))
    if grow:  # for one row of a warp, and under the cap: up to 5 tiles, 9 in base 2 from one to the next
        k[..., 0] = torch.arange(m, device="cuda").div(128, rounding_mode="floor")[None, :, None] * (9.0 * d ** 0.5 / 16 / 1.4427)
        q[..., 0] = 0.0
        q[:, 5::32, :, 0] = 16.0
    cap = 60.0 if "cap" in add else 0.0
    slopes = 2.0 ** (-8.0 * torch.arange(1, hq + 1, device="cuda", dtype=torch.float32) / hq).view(1, hq) if "alibi" in add else None
    o, lse = ops.fmha_fwd(q, k, v, window_size=(left, right), alibi_slopes=slopes, logits_soft_cap=cap, return_lse=True)
    assert _lib.get_instance_param(0, "last_instance") == 1
    kk, vv = (t.double().repeat_interleave(hq // hkv, 2) for t in (k, v))
    x = torch.einsum("bqhd,bkhd->bhqk", q.double(), kk) * d ** -0.5
    if cap:
        x = cap * torch.tanh(x / cap)
    i, j = torch.arange(n, device="cuda")[:, None] + (m - n), torch.arange(m, device="cuda")
    if slopes is not None:
        x = x - slopes[0, :, None, None].double() * (i - j).abs()
    if right >= 0:
        x = x.masked_fill(j > i + right, float("-inf"))
    if left >= 0:
        x = x.masked_fill(j < i - left, float("-inf"))
    assert_o_close(o, torch.einsum("bhqk,bkhd->bqhd", torch.softmax(x, -1).nan_to_num(), vv))
    assert_lse_close(lse, torch.logsumexp(x, -1))
