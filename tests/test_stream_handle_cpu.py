"""The handle of the current stream, with and without torch's raw-handle function
(a stand-in module: no GPU needed)."""
import types

import pytest

from gpg import lib as gpglib


class _Stream:
    def __init__(self, handle):
        self.cuda_stream = handle


def _module(raw):
    c = types.SimpleNamespace()
    if raw:
        c._cuda_getCurrentRawStream = lambda index: 100 + index
    return types.SimpleNamespace(_C=c, cuda=types.SimpleNamespace(current_stream=lambda index: _Stream(100 + index)))


@pytest.mark.parametrize("raw", [True, False])
def test_current_stream(monkeypatch, raw):
    monkeypatch.setattr(gpglib, "_torch", _module(raw))
    assert gpglib.stream_ptr(None, 3) == 103
    assert gpglib.stream_ptr(_Stream(7), 3) == 7
