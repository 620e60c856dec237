"""raise_on_error_words also reads the error word of the batch attention kernels, which live in no workspace (a fake of the C call
reports the expired wait: no GPU)."""
import ctypes
import types

import pytest


@pytest.fixture
def fake(lib_built, monkeypatch):
    from minit_b200 import _lib
    state = {0: 0, 1: 0}
    current = []

    class Device:
        def __init__(self, index):
            self.index = index

        def __enter__(self):
            current.append(self.index)

        def __exit__(self, *exc):
            current.pop()

    def call(word, clear):
        ptr = ctypes.cast(word, ctypes.POINTER(ctypes.c_uint32))
        ptr[0] = state[current[-1]]
        if clear:
            state[current[-1]] = 0
        return 0

    monkeypatch.setattr(_lib, "lib", types.SimpleNamespace(mt_attention_error=call, mt_strerror=_lib.lib.mt_strerror))
    monkeypatch.setattr(_lib, "_workspaces", {})
    monkeypatch.setattr(_lib, "attention_devices", {0, 1})
    monkeypatch.setattr(_lib.torch.cuda, "device", Device)
    monkeypatch.setattr(_lib.torch.cuda, "current_stream", lambda *a: types.SimpleNamespace(synchronize=lambda: None))
    return _lib, state


def test_an_expired_attention_wait_raises_and_is_cleared(fake):
    _lib, state = fake
    _lib.raise_on_error_words()
    state[1] = 8
    with pytest.raises(_lib.MinitError) as info:
        _lib.raise_on_error_words(clear=False)
    assert info.value.status == _lib.ERR_PEER_TIMEOUT and info.value.words == [((1, "attention"), 8)]
    with pytest.raises(_lib.MinitError):
        _lib.raise_on_error_words()
    _lib.raise_on_error_words()


@pytest.mark.gpu
def test_calls_are_watched_and_leave_the_word_clear(lib_built):
    import torch
    from minit_b200 import _lib, decoder as D
    q = torch.randn((1, 1, 8, 64), device="cuda:0").half()
    kv = torch.randn((1, 40, 2, 64), device="cuda:0").half()
    D.attention(q, kv, kv, 39)
    assert 0 in _lib.attention_devices and _lib.attention_error_word(0, clear=False) == 0
    _lib.raise_on_error_words()
    assert _lib.lib.mt_attention_error(None, 0) == -1
