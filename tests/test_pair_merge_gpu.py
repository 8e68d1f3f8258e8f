"""The merge of two rows per warp at the most splits it takes, with more rows than the forms of several warps per row are for (592 on 148
SMs) and two rows of a warp that use different numbers of splits."""
import pytest
import torch

from flashck_b200 import ops
from tests.helpers import assert_lse_close, assert_o_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [9, 15, 16])
@pytest.mark.parametrize("rows,hq,dv", [(101, 7, 128), (1, 2401, 64), (1300, 2, 68)])
@pytest.mark.parametrize("use", ["none beside all", "one beside all", "any"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_many_rows(S, rows, hq, dv, use, dtype):
    g = torch.Generator().manual_seed(S + rows)
    lse_acc = torch.randn((1, hq, S, rows), generator=g)
    o_acc = torch.randn((1, hq, S, rows, dv), generator=g)
    item = torch.arange(hq * rows).view(1, hq, 1, rows)  # (a warp takes the rows 2 i and 2 i + 1)
    used = torch.randint(0, S + 1, (1, hq, 1, rows), generator=g) if use == "any" else \
        torch.where(item % 2 == 0, 0 if use == "none beside all" else 1, S)
    empty = torch.arange(S)[None, None, :, None] >= used
    lse_acc[empty] = float("-inf")
    o_acc[empty] = float("nan")
    o, lse = ops.fmha_fwd_splitkv_combine(lse_acc.cuda(), o_acc.cuda(), dtype, return_lse=True)
    w = torch.softmax(lse_acc.double(), 2).nan_to_num()[..., None]
    assert_o_close(o, (w * o_acc.double().masked_fill(empty[..., None], 0.0)).sum(2).permute(0, 2, 1, 3))
    assert_lse_close(lse, torch.logsumexp(lse_acc.double(), 2))
