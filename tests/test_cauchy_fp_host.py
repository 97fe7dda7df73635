"""Host restatement of the Cauchy step's double-precision quotient digits (csrc/cauchy_fp.cuh): the digit steps with
correctly rounded fused multiply-adds give truncated quotients exactly, for every digit width at the ends of its
range of divisors, and no intermediate leaves the range in which doubles hold integers exactly.  CPU only."""
import random
from fractions import Fraction

import pytest

MG = 6755399441055744                                     # 1.5 2^52


def rne(x):
    """a rational rounded to a double (ties to even), as a Fraction"""
    return Fraction(float(x))                             # Fraction -> float is correctly rounded


def quotient(X, d, W, ND):
    """sum_j q_j 2^(W j) after the final correction, for a signed dividend of ND digits"""
    sx = -1 if X < 0 else 1
    digits = [(abs(X) >> (W * (ND - 1 - j))) & ((1 << W) - 1) for j in range(ND)]
    inv = Fraction(1.0 / abs(d)) * (1 if d > 0 else -1)
    r, acc = 0, 0
    for v in digits:
        c = r * (1 << W) + sx * v
        assert abs(c) <= 1 << 53
        qp = rne(c * inv + MG)
        assert 1 << 52 <= qp < 1 << 53 and qp.denominator == 1
        q = int(qp) - MG
        r = c - q * d
        assert abs(r) < abs(d)
        acc = (acc << W) + q
    s = sx * (1 if d > 0 else -1)
    if r and (r < 0) != (sx < 0):
        acc -= s
    return acc


def trunc(X, d):
    q = abs(X) // abs(d)
    return q if (X < 0) == (d < 0) else -q


@pytest.mark.parametrize("W,ds", [(46, (1, 2, 3, 127, 128, 246, 247)), (45, (248, 255, 256, 479, 480)),
                                  (43, (481, 1023, 1024, 1899, 1900)), (37, (1901, 32767, 32768, 65534, 65535))])
@pytest.mark.parametrize("L", [6, 34])
def test_quotient_digits_are_exact(L, W, ds):
    rng = random.Random(W * 100 + L)
    bits = 32 * L - 2
    ND = -(-32 * (L + 1) // W)
    for d in ds:
        xs = [0, 1, (1 << bits) - 1, 1 << (bits - 1), d, d - 1, d + 1]
        xs += [rng.getrandbits(bits) for _ in range(8)]
        xs += [(rng.getrandbits(bits) // d) * d + e for e in (-1, 0, 1)]
        for x in xs:
            for X in (abs(x) << 32, -(abs(x) << 32)):
                for dd in (d, -d):
                    assert quotient(X, dd, W, ND) == trunc(X, dd), (L, W, d, x)
