"""Which compiled binding the calls of ``ops`` go through: one that is older than the package, cannot be loaded or is not there."""
import sys
import types
import warnings

import pytest
import torch

import flashck_b200
from flashck_b200 import _lib, ops
from flashck_b200.ops import fmha
from flashck_b200.utils import flags


@pytest.fixture
def binding(monkeypatch):
    """Puts another module (or None: importing it fails) in the binding's place."""
    def put(module):
        monkeypatch.setattr(fmha, "_NATIVE", None)
        monkeypatch.delattr(flashck_b200, "flash_ck", raising=False)
        monkeypatch.setitem(sys.modules, "flashck_b200.flash_ck", module)
        if module is not None:
            monkeypatch.setattr(flashck_b200, "flash_ck", module, raising=False)
    return put


def _call():
    x = torch.zeros(1, 8, 2, 64, dtype=torch.bfloat16)
    ops.fmha_fwd(x, x, x)


@pytest.mark.parametrize("kept", [0, 3])
def test_older_binding(binding, kept):
    stub = types.ModuleType("flashck_b200.flash_ck")  # built before some of the calls were there
    for name in fmha._NATIVE_CALLS[:kept]:
        setattr(stub, name, None)
    binding(stub)
    with pytest.warns(RuntimeWarning, match="older sources"), pytest.raises(ValueError, match="must be a CUDA tensor"):
        _call()
    with warnings.catch_warnings():  # said once
        warnings.simplefilter("error")
        assert fmha._native() is False


def test_binding_that_does_not_load(binding, monkeypatch):
    binding(None)
    monkeypatch.setattr(fmha.glob, "glob", lambda pattern: ["flash_ck.so"])
    with pytest.warns(RuntimeWarning, match="cannot be loaded"), pytest.raises(ValueError, match="must be a CUDA tensor"):
        _call()


@pytest.mark.parametrize("log", [False, True])
def test_binding_not_built(binding, monkeypatch, capfd, log):
    binding(None)
    monkeypatch.setattr(fmha.glob, "glob", lambda pattern: [])
    monkeypatch.setattr(flags.flag("FC_TUNING_LOG"), "value", log)
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert fmha._native() is False
    assert ("has not been built" in capfd.readouterr().err) == log


def test_arguments_are_checked_before_the_library_is_missed(binding, monkeypatch):
    binding(None)
    monkeypatch.setattr(_lib, "LIB_PATH", "/nonexistent/libflashck_b200.so")
    monkeypatch.setattr(_lib, "_LIB", None)
    with pytest.raises(ValueError, match="must be a CUDA tensor"):
        _call()
    assert fmha._NATIVE is None  # looked for again once the library is there
