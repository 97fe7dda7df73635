"""The pole step's form of a run (Recursion.uses_mma, no GPU): shapes measured on a B200 with both forms go to the faster one."""
from types import SimpleNamespace

import pytest

from blocksvibe_b200 import _lib, build, recursion as RC


def uses_mma(L, S, B, pole="auto"):
    rec = object.__new__(RC.Recursion)
    rec.L, rec.pole, rec.plan = L, pole, SimpleNamespace(Smax=S)
    return rec.uses_mma(B)


@pytest.mark.parametrize("L,S,B,mma", [          # ms of 3000 tasks (1500 from S = 6 on), CUDA cores / tensor cores
    (26, 2, 32, False),                          # 0.190 / 0.224
    (34, 2, 32, False),                          # 0.254 / 0.294
    (38, 2, 16, False),                          # 0.166 / 0.177
    (34, 5, 6, True),                            # a task of six lambda orders: 18.4 ms against 28
    (34, 5, 1, False),                           # one lambda order: five columns
    (26, 3, 42, True),                           # seven tasks of three structures
    (14, 5, 6, True),                            # 0.216 / 0.187
    (14, 6, 10, True),                           # 0.302 / 0.222
    (18, 3, 10, False),                          # 0.125 / 0.130
    (10, 6, 10, True),                           # 0.206 / 0.189
    (6, 7, 9, False),                            # 0.172 / 0.178
    (26, 8, 2, True),                            # 0.312 / 0.236
    (22, 8, 2, True),                            # 0.249 / 0.214
    (42, 5, 6, True),                            # 1.18 times
    (42, 8, 4, False),                           # 1.157 / 1.218
    (46, 7, 4, False),                           # 0.941 / 1.118
    (46, 6, 10, True),
    (34, 1, 64, False),                          # no tensor-core form for S = 1
])
def test_measured_shapes(L, S, B, mma):
    assert uses_mma(L, S, B) == mma


def test_fill_and_overrides():
    assert RC.pole_mma_speedup(34, 5, 7) < 0.6 * RC.pole_mma_speedup(34, 5, 6)       # a second, nearly empty chunk
    assert RC.pole_mma_speedup(34, 5, 3) < RC.pole_mma_speedup(34, 5, 4)
    assert uses_mma(34, 5, 1, "mma") and not uses_mma(34, 5, 6, "cuda")
    assert set(RC.POLE_SPEEDUP) == set(build.LIMBS)
    assert all(len(r) == 7 for rows in RC.POLE_SPEEDUP.values() for r in rows)
    assert all(_lib.lib().b3d_supported_limbs(L) for L in RC.POLE_SPEEDUP)
