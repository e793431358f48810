"""What `persistent_gru.check_status` makes of the status words (no GPU: the extension is a stand-in)."""
import types

import pytest


def test_status_words_become_errors(monkeypatch):
    from tensorflow_allreduce_b200 import _lib
    from tensorflow_allreduce_b200.ops import persistent_gru as pg

    codes = {0: 0, 1: 0}

    def take(device):
        code, codes[device] = codes[device], 0
        return code

    monkeypatch.setattr(_lib, "ext", lambda: types.SimpleNamespace(gru_devices=lambda: [0, 1], gru_take_status=take))
    pg.check_status()
    codes[1] = 1
    pg.check_status("cuda:0")
    with pytest.raises(RuntimeError, match="persistent GRU kernel timed out on cuda:1"):
        pg.check_status()
    pg.check_status()                                 # taken
    codes[0] = 8
    with pytest.raises(RuntimeError, match="row convolution timed out on cuda:0"):
        pg.check_status("cuda")
