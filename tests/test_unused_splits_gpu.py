"""The slots of splits that a sequence does not use, for one and for many sequences, deep and shallow workspaces, packed queries of
unequal lengths among them: all are marked with -inf, and the slots of other sequences stay what their partials are."""
import pytest
import torch

from flashck_b200 import ops
from flashck_b200.utils.inputs import make_paged_cache, normal_tensor, to_seqstarts, uniform_seqlens
from tests.helpers import assert_lse_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 3, 60, 100, 300])
@pytest.mark.parametrize("splits", [2, 9, 128])
@pytest.mark.parametrize("tokens", ["one", "four", "packed"])
@pytest.mark.parametrize("hq,hkv,d", [(8, 2, 128), (5, 5, 64)])
def test_every_slot_is_written(batch, splits, tokens, hq, hkv, d):
    keys = uniform_seqlens(batch, 4, 400, 7)
    keys[batch // 2] = 4
    new = uniform_seqlens(batch, 0, 4, 8) if tokens == "packed" else [1 if tokens == "one" else 4] * batch
    new[0] = max(new[0], 1)
    c = make_paged_cache(keys, hkv, d, d, 16, torch.bfloat16, seed=3)
    q, kw = normal_tensor((sum(new), hq, d), torch.bfloat16, 4).cuda(), {}
    shape = (1, hq, splits, sum(new))
    if tokens == "packed":
        kw = {"cu_seqlens_q": to_seqstarts(new).cuda(), "max_seqlen_q": max(new)}
    else:
        q, shape = q.view(batch, new[0], hq, d), (batch, hq, splits, new[0])
    guard = 64  # (floats in front of and behind the LSEs)
    buf = torch.full((shape[0] * shape[1] * shape[2] * shape[3] + 2 * guard,), float("nan"), device="cuda")
    lse_acc = buf[guard:-guard].view(shape)
    o_acc = torch.full(shape + (d,), float("nan"), device="cuda")
    args = (q, c.k.cuda(), c.v.cuda())
    kw |= {"seqlen_k": c.seqlen_k.cuda(), "block_table": c.block_table.cuda(), "causal": tokens != "one"}
    ops.fmha_fwd_splitkv(*args, workspace=(lse_acc, o_acc), combine=False, **kw)
    assert torch.isnan(buf[:guard]).all() and torch.isnan(buf[-guard:]).all()
    assert not torch.isnan(lse_acc).any()
    # a split is in use by all heads of a row or by none, the ones in use come first, and each of them has its partial
    used = lse_acc != float("-inf")
    assert (used == used[:, :1]).all() and (used[:, :, 1:] <= used[:, :, :-1]).all() and used[:, :, 0].all()
    assert not torch.isnan(o_acc[used]).any()
    # one split per sequence needs no marks: the same rows but for the order of the sums
    o, lse = ops.fmha_fwd_splitkv_combine(lse_acc, o_acc, torch.float32, varlen=tokens == "packed", return_lse=True)
    one = ops.fmha_fwd_splitkv(*args, num_splits=1, return_lse=True, **kw)
    assert_lse_close(lse, one[1])
    # (P is rounded to bf16 on either side, and the one side's O as well)
    assert (o - one[0].float()).abs().max() <= 2.0 ** -9 * (2 * c.v.abs().max().float() + o.abs().max())
