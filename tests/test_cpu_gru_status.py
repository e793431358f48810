"""The host side of the persistent GRU layers without a GPU: what `persistent_gru.check_status` makes of the status words (the extension is a
stand-in), the size of the memory through which blocks exchange."""
import ctypes
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


def test_scratch_holds_what_the_kernels_address(native_lib):
    # Restated from the kernel: [direction][owner block][member of the group][slot][pack of three][row] words of 16 bytes behind the ring of
    # [direction][slot][member][K tile of 32][batch 16 or 32][32] words and 1 KiB of counters.
    for nd in (1, 2):
        for H in range(128, 1025, 128):
            for B in range(1, 33):
                blocks, nb, need = H // 16, 16 if B <= 16 else 32, 0
                ring = nd * 2 * (3 * H + 256) * 32 * 4
                for backward in (False, True):
                    small = B <= 16
                    C = (4 if H <= (256 if small else 512) else 8) if backward else (1 if H <= (512 if small else 256) else 2)
                    rows, kq = (16, 3 * H // C) if backward else (48, H // C)
                    assert nd * 2 * C * -(-kq // 32) * nb * 32 * 4 <= ring
                    need = max(need, nd * blocks * C * 2 * -(-B // 3) * rows * 16)
                assert native_lib.bc_gru_scratch_bytes(7, B, H, nd) == 1024 + ring + need


def test_partial_sums_of_the_backward_pass_fit_behind_its_ring(native_lib):
    # Restated from gru_backward.cu: groups of C blocks, a ring of [direction][slot][member][tile of 32 units][batch 16 or 32][32] words, behind it
    # [direction][owner block][source, without the owner][slot][pack of three][row] words of 16 bytes.
    for nd in (1, 2):
        for H in range(128, 1025, 128):
            for B in range(1, 33):
                nb = 16 if B <= 16 else 32
                C = 4 if nb == 32 and H <= 256 else 8
                ring = nd * 2 * C * -(-H // C // 32) * nb * 32 * 4
                sums = nd * (H // 16) * (C - 1) * 2 * -(-B // 3) * 16 * 16
                assert 1024 + ring + sums <= native_lib.bc_gru_scratch_bytes(7, B, H, nd)


def test_alignment_is_refused_before_a_launch(native_lib):
    # The kernels read factors and exchange memory 32 bytes at a time. Nothing is dereferenced: without a GPU an aligned call ends at the device.
    from tensorflow_allreduce_b200 import _lib

    p = lambda at: ctypes.c_void_p(at)
    base = 1 << 20
    for fac, scratch in ((base + 16, base), (base, base + 16), (base + 4, base)):
        with pytest.raises(Exception, match="invalid argument"):
            _lib.check(native_lib.bc_gru_backward_factors(3, 2, 128, 1, p(base), p(base), p(fac), p(base), p(base), p(base), p(scratch), p(base), 1.0,
                                                          p(None)), "backward")
        with pytest.raises(Exception, match="invalid argument"):
            _lib.check(native_lib.bc_gru_forward_factors(3, 2, 128, 1, p(base), p(base), p(base), p(base), p(base), p(base), p(fac), p(scratch), p(base),
                                                         1.0, p(None)), "forward")
