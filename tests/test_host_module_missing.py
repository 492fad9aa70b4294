"""The layers work without the native host side of the forward, which needs g++, torch's headers and a matching torch."""
import os
import sys
import warnings

import pytest
import torch

from bitween_b200 import QuantizedLinear
from bitween_b200.csrc import build as build_module
from bitween_b200.kernels import _lib


PATH = _lib.HOST_LIB_PATH


def _fails(*args, **kwargs):
    raise RuntimeError("no compiler")


@pytest.fixture(params=["absent", "half written"])
def without_host_module(request, monkeypatch, tmp_path):
    path = tmp_path / "_host_forward.so"
    if request.param == "half written":
        path.write_bytes(b"\x7fELF")
    monkeypatch.setattr(_lib, "HOST_LIB_PATH", str(path))
    monkeypatch.setattr(build_module, "build_host", _fails)
    monkeypatch.setattr(_lib, "_host", None)


def test_reported_once_and_no_call_is_taken(without_host_module):
    with pytest.warns(UserWarning, match="native host side"):
        forward = _lib.host_forward()
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert _lib.host_forward() is forward
    assert forward(torch.zeros(1, 32), None, None, None, None, 4, 32) is None


def test_the_cuda_library_is_built_without_it(monkeypatch, capfd):
    monkeypatch.setattr(build_module, "build_host", _fails)
    assert build_module.build() == build_module.LIB and os.path.exists(build_module.LIB)
    assert "no compiler" in capfd.readouterr().err


def test_the_module_is_named_for_its_python_and_torch():
    assert sys.implementation.cache_tag in PATH and torch.__version__ in PATH and os.path.exists(PATH)


@pytest.mark.gpu
def test_forward_without_it(without_host_module):
    torch.manual_seed(0)
    ql = QuantizedLinear.from_float(torch.nn.Linear(1024, 48).to("cuda"), 4, 128)
    x = torch.randn(5, 1024, device="cuda").half()
    with pytest.warns(UserWarning, match="native host side"), torch.no_grad():
        y = ql(x)
    _lib._host = None
    _lib.HOST_LIB_PATH = PATH
    with torch.no_grad():
        assert torch.equal(y, ql(x)) and _lib._host is not _lib._takes_no_call
