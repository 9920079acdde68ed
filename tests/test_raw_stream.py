"""The stream handle handed to the library (no GPU needed)."""
import types

import pytest
import torch

from kvmix_b200 import ops


@pytest.mark.parametrize("missing", ["_raw_stream", "_device"])
def test_torch_without_the_raw_stream_functions(monkeypatch, missing):
    """Where torch lacks one of the two undocumented functions, the stream comes from torch.cuda.current_stream()."""
    monkeypatch.setattr(ops, missing, None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: types.SimpleNamespace(cuda_stream=1234))
    assert ops.raw_stream() == 1234
