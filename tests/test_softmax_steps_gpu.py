"""The step of the tcgen05 softmax where its code forms change: a hidden score in the tile or none, the 32-column groups of a
masked tile, and the rescale of O when a row's maximum grows by more than 2^8."""
import pytest
import torch

from flashck_b200 import _lib, ops
from tests.helpers import assert_lse_close, assert_o_close

pytestmark = pytest.mark.gpu


def _reference(q, k, v, left, right):
    """Row i sees the keys [i + m - n - left, i + m - n + right] (-1: no bound)."""
    n, m, group = q.shape[1], k.shape[1], q.shape[2] // k.shape[2]
    kk, vv = (t.double().repeat_interleave(group, 2) for t in (k, v))
    x = torch.einsum("bqhd,bkhd->bhqk", q.double(), kk) * q.shape[3] ** -0.5
    i, j = torch.arange(n, device=q.device)[:, None] + (m - n), torch.arange(m, device=q.device)
    if right >= 0:
        x = x.masked_fill(j > i + right, float("-inf"))
    if left >= 0:
        x = x.masked_fill(j < i - left, float("-inf"))
    lse = torch.logsumexp(x, -1)
    return torch.einsum("bhqk,bkhd->bqhd", torch.softmax(x, -1).nan_to_num(), vv).float(), lse.float()


def _inputs(n, m, hq, hkv, d, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn((2, s, h, d), generator=g, device="cuda").bfloat16() for s, h in ((n, hq), (m, hkv), (m, hkv)))


# key counts around the groups' and the tile's edges; more and fewer queries than keys; bands inside a group and across some
@pytest.mark.parametrize("n,m", [(1, 1), (33, 31), (97, 96), (128, 129), (130, 160), (129, 225), (200, 128), (300, 257)])
@pytest.mark.parametrize("left,right", [(-1, -1), (-1, 0), (0, 0), (31, 0), (40, 33), (-1, 64), (150, -1)])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("hq,hkv", [(4, 2), (3, 3)])
def test_masked_tiles(n, m, left, right, d, hq, hkv):
    q, k, v = _inputs(n, m, hq, hkv, d, n + m)
    o, lse = ops.fmha_fwd(q, k, v, window_size=(left, right), return_lse=True)
    assert _lib.get_instance_param(0, "last_instance") == 1
    o_ref, lse_ref = _reference(q, k, v, left, right)
    assert_o_close(o, o_ref)
    assert_lse_close(lse, lse_ref)


# scores (base 2) that grow by `jump` from tile to tile, for every row or for one row of a warp
@pytest.mark.parametrize("jump", [6.0, 9.0, 40.0])
@pytest.mark.parametrize("rows", ["all", "one"])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("left", [-1, 200])
def test_growing_maximum(jump, rows, d, left):
    n = m = 640
    q, k, v = _inputs(n, m, 4, 2, d, 7)
    k[..., 0] = torch.arange(m, device="cuda").div(128, rounding_mode="floor")[None, :, None] * (jump * d ** 0.5 / 16 / 1.4427)
    q[..., 0] = 16.0
    if rows == "one":
        q[:, torch.arange(n, device="cuda") % 32 != 5, :, 0] = 0.0
    o, lse = ops.fmha_fwd(q, k, v, causal=True, window_size=(left, 0), return_lse=True)
    assert _lib.get_instance_param(0, "last_instance") == 1
    o_ref, lse_ref = _reference(q, k, v, left, 0)
    assert_o_close(o, o_ref)
    assert_lse_close(lse, lse_ref)


# 8-bit operands: the steps without a hidden score are a range worked out ahead, and O is rescaled under the exponentials.  P is
# rounded to 3 (E4M3) or 2 (E5M2) bits behind the leading one: an element of O is off by at most half a unit in the last place of
# every P, 2^-4 or 2^-3 of the attention over |V|, and by the rounding of O to bf16 (2^-9 of it).
@pytest.mark.parametrize("dtype,ulp", [(torch.float8_e4m3fn, 2.0 ** -4), (torch.float8_e5m2, 2.0 ** -3)])
@pytest.mark.parametrize("n,m", [(1, 1), (97, 96), (128, 129), (129, 225), (200, 128), (300, 640)])
@pytest.mark.parametrize("left,right", [(-1, -1), (-1, 0), (0, 0), (31, 0), (40, 33), (-1, 64), (150, -1), (300, 0)])
@pytest.mark.parametrize("grow", [False, True])
def test_eight_bit_steps(dtype, ulp, n, m, left, right, grow):
    q, k, v = _inputs(n, m, 4, 2, 128, n + m)
    if grow:  # the maximum rises from tile to tile, for one row of a warp
        k[..., 0] = torch.arange(m, device="cuda").div(128, rounding_mode="floor")[None, :, None] * 2.0
        q[..., 0] = 0.0
        q[:, 5::32, :, 0] = 8.0
    q8, k8, v8 = (x.to(dtype) for x in (q, k, v))
    o, lse = ops.fmha_fwd_fp8(q8, k8, v8, scale_p=256.0, scale_o=1 / 256.0, window_size=(left, right), out_dtype=torch.bfloat16,
                              return_lse=True)
    assert _lib.get_instance_param(0, "last_instance") == 1
    qd, kd, vd = (x.float() for x in (q8, k8, v8))
    o_ref, lse_ref = _reference(qd, kd, vd, left, right)
    bound = _reference(qd, kd, vd.abs(), left, right)[0] * ulp + o_ref.abs() * 2.0 ** -9
    # (a P below the smallest normal number keeps fewer bits: 2^-7 / 256 of the largest P and key, E5M2 far less)
    bound += m * 2.0 ** -10 / 256 * vd.abs().max() + 1e-6
    assert ((o.float() - o_ref).abs() <= bound).all()
    assert_lse_close(lse, lse_ref)
