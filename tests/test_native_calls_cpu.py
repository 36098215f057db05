"""Without a native host path for the running torch, calls take the Python code: nothing that ran before stops running."""
import warnings

import pytest
import torch

from aitemplate_b200 import _lib
from aitemplate_b200 import kernels as K


@pytest.fixture(autouse=True)
def fresh(monkeypatch):
    monkeypatch.setattr(K, "_calls", None)
    monkeypatch.setattr(_lib, "_calls", None)


def _refuses_host_tensors():
    with pytest.raises(ValueError, match="CUDA tensors"):
        K.softmax(torch.zeros(3, 4))
    with pytest.raises(ValueError, match="CUDA tensors"):
        K.gemm_rcr(torch.zeros(3, 4), torch.zeros(5, 4))


def test_the_built_one_is_for_this_torch():
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert _lib.load_calls().softmax(torch.zeros(3, 4), 1) is None  # (not on the GPU)
    assert torch.__version__ in _lib.calls_path().name


def test_another_torch(monkeypatch):
    monkeypatch.setattr(torch.version, "git_version", "0123456789abcdef")
    with pytest.warns(RuntimeWarning, match="aitemplate_b200.build"):
        _refuses_host_tensors()
    with warnings.catch_warnings():
        warnings.simplefilter("error")  # once
        _refuses_host_tensors()


def test_a_file_that_does_not_load(monkeypatch, tmp_path):
    broken = tmp_path / "torch_calls.so"
    broken.write_bytes(b"not a library")
    monkeypatch.setattr(_lib, "calls_path", lambda: broken)
    with pytest.warns(RuntimeWarning, match="cannot be loaded"):
        _refuses_host_tensors()


def test_no_library_at_all(monkeypatch, tmp_path):
    monkeypatch.setattr(_lib, "LIB_PATH", tmp_path / "libb200ait.so")
    monkeypatch.setattr(_lib, "_lib", None)
    _refuses_host_tensors()
