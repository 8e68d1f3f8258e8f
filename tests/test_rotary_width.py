"""``rotary_dim`` of ``fmha_fwd_append_kv``: None is the width of the tables, a number is taken as it is, and one that does not fit is
refused before anything is written, through the compiled binding and through Python."""
import pytest
import torch

from flashck_b200 import ops
from flashck_b200.ops import fmha
from flashck_b200.utils.enums import RopeEnum
from flashck_b200.utils.inputs import make_paged_cache, normal_tensor, rotary_cos_sin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("rope", [RopeEnum.INTERLEAVED, RopeEnum.HALF_ROTATED])
@pytest.mark.parametrize("rotary_dim", [-128, -4, -2, -1, 0, 7, 130, 1 << 40, -(1 << 40)])
def test_a_width_that_does_not_fit_is_refused(monkeypatch, native, rope, rotary_dim):
    if not native:
        monkeypatch.setattr(fmha, "_NATIVE", False)
    c = make_paged_cache([40, 33], 2, 128, 128, 16, torch.bfloat16, seed=5)
    q, kn, vn = (normal_tensor((2, 4, h, 128), torch.bfloat16, h).cuda() for h in (8, 2, 2))
    k, v, q0 = c.k.cuda(), c.v.cuda(), q.clone()
    cos, sin = (t.cuda() for t in rotary_cos_sin(64, 128, torch.bfloat16))
    with pytest.raises(RuntimeError, match=r"rotary_dim must be even and in \(0, hdim_q\]"):
        ops.fmha_fwd_append_kv(q, k, v, kn, vn, c.seqlen_k.cuda() - 4, cos, sin, rope=rope, rotary_dim=rotary_dim,
                               block_table=c.block_table.cuda())
    assert torch.equal(q, q0) and torch.equal(k.cpu(), c.k) and torch.equal(v.cpu(), c.v)
