"""Host logic of the flush's form choice (no GPU): windows measured on a B200 with both kernels go to the faster one."""
import ctypes

import pytest

from blocksvibe_b200 import _lib


def flush_form(LO, W, R1, NN, KW, cols, sms=148):
    v = ctypes.c_int(-1)
    _lib.call("b3d_moments_flush_form", LO, W, R1, NN, KW, cols, sms, ctypes.addressof(v))
    return v.value


@pytest.mark.parametrize("LO,W,R1,NN,KW,cols,mma", [      # microseconds, tensor cores / CUDA cores
    (10, 10, 13, 81, 6, 500, 1),                          # 39 / 100
    (10, 10, 13, 81, 6, 12500, 0),                        # 190 / 101
    (10, 10, 13, 81, 6, 16000, 0),                        # 240 / 98
    (18, 40, 4, 81, 2, 500, 1),                           # 29 / 85
    (18, 40, 4, 81, 2, 16000, 0),                         # 200 / 87
    (30, 20, 7, 81, 2, 12500, 0),                         # 183 / 119
    (46, 40, 4, 81, 2, 16000, 0),                         # 356 / 191
    (46, 72, 28, 81, 6, 16000, 1),                        # 1136 / 2902
    (46, 72, 28, 81, 6, 170000, 1),                       # 11800 / 18000
    (38, 40, 12, 41, 2, 12500, 1),                        # 280 / 370
    (38, 40, 12, 41, 2, 593400, 0),                       # 13100 / 9000
    (38, 48, 16, 49, 6, 300000, 0),                       # 10600 / 8400
    (10, 10, 6, 11, 2, 1800, 0),                          # 43 / 42
    (46, 8, 28, 81, 6, 170000, 0),                        # the second window of an order of 80
    (42, 40, 32, 41, 12, 100, 0),                         # integers too long for one tile
])
def test_measured_windows(LO, W, R1, NN, KW, cols, mma):
    assert flush_form(LO, W, R1, NN, KW, cols) == mma


def test_follows_the_number_of_multiprocessors():
    assert flush_form(30, 20, 7, 81, 2, 12500, 600) == 1 and flush_form(30, 20, 7, 81, 2, 2000, 148) == 1
    with pytest.raises(_lib.B3DError):
        flush_form(30, 20, 33, 81, 2, 12500)
