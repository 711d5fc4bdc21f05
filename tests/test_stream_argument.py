"""The stream that a call without one runs on (CPU): the legacy stream where no
torch runs CUDA work, also while another thread is still importing torch."""
import sys
import types

import pytest

from ftd_b200 import herk


def partial_torch(cuda):
    t = types.ModuleType("torch")
    if cuda:
        t.cuda = types.ModuleType("torch.cuda")
    return t


@pytest.mark.parametrize("cuda", [False, True])
def test_half_imported_torch(monkeypatch, cuda):
    monkeypatch.setitem(sys.modules, "torch", partial_torch(cuda))
    assert herk._stream(None) == 0


def test_no_torch(monkeypatch):
    monkeypatch.delitem(sys.modules, "torch", raising=False)
    assert herk._stream(None) == 0
    assert "torch" not in sys.modules


def test_given_streams():
    assert herk._stream(77) == 77
    assert herk._stream(types.SimpleNamespace(cuda_stream=5)) == 5
