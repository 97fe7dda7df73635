"""The work that the bench's tensor roofline of the pole step counts, against the geometry in csrc/pole_mma.cuh: entries in chunks
of 16 digits (U), NCH chunks an entry, two chunks a K step."""
import os
import re

import pytest

from blocksvibe_b200 import roofline as RL

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "blocksvibe_b200", "csrc")


def test_source_geometry_is_the_one_counted():
    with open(os.path.join(CSRC, "pole_mma.cuh")) as f:
        src = re.sub(r"\s+", " ", f.read())
    assert "int U = 16 * ((D + 15) / 16);" in src and "int NCH = U / 16;" in src and "int D = 4 * L;" in src
    assert "int steps(int S) { return (S * G::NCH + 1) / 2; }" in src


@pytest.mark.parametrize("L,S,steps", [(34, 5, 23), (26, 5, 18), (10, 5, 8), (10, 2, 3), (46, 8, 48), (6, 1, 1)])
def test_issued_macs(L, S, steps):
    assert RL.pole_mma_steps(L, S) == steps
    lev, B = {"t_slot": [0] * 10}, 6
    cols = S * B
    nc = 16 if cols <= 16 else 32
    issued, useful = RL.pole_mma_issued(lev, S * S * B, S, L)
    chunks = -(-cols // nc)
    assert issued == 2 * 10 * chunks * S * steps * RL.pole_mma_geometry(L)[1] * 128 * nc * 32
    assert useful == 2 * 10 * S * S * cols * (4 * L) ** 2
    assert issued <= RL.pole_mma_macs(lev, S * S * B, S, L)[0]
