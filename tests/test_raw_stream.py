"""The stream handle handed to the library (no GPU needed)."""
import types

import pytest
import torch

from kvmix_b200 import ops


@pytest.mark.parametrize("present", [(), ("_cuda_getDevice",), ("_cuda_getCurrentRawStream",)])
def test_torch_without_the_raw_stream_functions(monkeypatch, present):
    """Where torch lacks one of the two undocumented functions, the stream comes from torch.cuda.current_stream()."""
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: types.SimpleNamespace(cuda_stream=1234))
    assert ops._stream_getter(types.SimpleNamespace(**{n: (lambda *a: 5) for n in present}))() == 1234


def test_raw_stream_of_the_current_device():
    c = types.SimpleNamespace(_cuda_getCurrentRawStream=lambda d: 100 + d, _cuda_getDevice=lambda: 3)
    assert ops._stream_getter(c)() == 103
