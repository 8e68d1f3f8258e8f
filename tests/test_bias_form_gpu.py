"""Which form a bias tensor takes into the tcgen05 kernel: whole rows of 16-byte pieces by TMA through shared memory, everything else by
the softmax threads."""
import pytest
import torch

from flashck_b200 import _lib, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,shift,packed,by_tma", [
    (130, 64, 0, False, 1), (1, 264, 0, False, 1), (130, 64, 8, False, 1), (130, 640, 1, False, 0), (130, 640, 4, False, 0),
    (130, 63, 0, False, 0), (130, 56, 0, False, 0), (130, 66, 0, False, 0), (130, 257, 0, False, 0), (128, 128, 0, True, 0),
])
@pytest.mark.parametrize("window", [(-1, -1), (40, 0)])
def test_form(n, m, shift, packed, by_tma, window):
    q, k, v = (torch.zeros((1, s, 2, 128), dtype=torch.bfloat16, device="cuda") for s in (n, m, m))
    buf = torch.zeros(2 * n * m + shift, dtype=torch.bfloat16, device="cuda")
    bias = buf[shift:].view(1, 2, n, m)
    if packed:
        cu = torch.tensor([0, n], device="cuda")
        ops.fmha_fwd_var_len(q[0], k[0], v[0], cu, cu, n, window_size=window, bias=bias)
    else:
        ops.fmha_fwd(q, k, v, window_size=window, bias=bias)
    assert _lib.get_instance_param(0, "last_instance") == 1
    assert _lib.get_instance_param(0, "last_bias_form") == by_tma
