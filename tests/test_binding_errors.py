"""Errors of the compiled binding reach Python as exceptions, whatever their message prints and whoever throws them."""
import os
import subprocess
import sys

import pytest
import torch

from flashck_b200 import flash_ck, ops
from flashck_b200.ops import fmha

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# (tensors without memory or device: the sizes are refused before anything is read; a process of its own, which may end)
_SIZES = """
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from flashck_b200 import flash_ck
with FakeTensorMode():
    q, k = (torch.zeros(1, 8, 2, d, dtype=torch.bfloat16, device="cuda") for d in (64, 32))
    try:
        flash_ck.fmha_fwd(q, k, k)
    except RuntimeError as e:
        print(str(e).splitlines()[0])
"""


def test_a_message_with_sizes():
    r = subprocess.run([sys.executable, "-c", _SIZES], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "inconsistent shapes q[1, 8, 2, 64] k[1, 8, 2, 32]" in r.stdout, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("native", [True, False])
def test_out_of_memory(monkeypatch, native):
    """A workspace larger than the card (8192 rows of 64 heads in 1024 splits: 277 GB) is the allocator's own error."""
    if not native:
        monkeypatch.setattr(fmha, "_NATIVE", False)
    assert fmha._native() is (flash_ck if native else False)
    q, k = (torch.zeros(1, n, h, 128, dtype=torch.bfloat16, device="cuda") for n, h in ((8192, 64), (16, 8)))
    with pytest.raises(torch.OutOfMemoryError):
        ops.fmha_fwd_splitkv(q, k, k, num_splits=1024)
