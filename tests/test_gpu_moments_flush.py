"""The staged moments' flush on the CUDA cores (b3d_moments_flush) against exact integer sums: per order k the result lies
within half a unit in its last place, plus the truncation of the terms (W units of 2^(E_k - 32 (Lout + 2)), E_k the
exponent above the order's largest term), of sum_w n_w^k Y_w."""
from fractions import Fraction

import pytest
import torch

from blocksvibe_b200 import _lib, mpf
from test_gpu_moments_mma import power_table

pytestmark = pytest.mark.gpu


def integers(x, L):
    """mantissas of limb planes (L, n) as Python integers"""
    planes = [[v & 0xFFFFFFFF for v in p] for p in x.reshape(L, -1).cpu().tolist()]
    out = []
    for limbs in zip(*planes):
        v = sum(b << (32 * i) for i, b in enumerate(limbs))
        out.append(v - (1 << (32 * L)) if v >> (32 * L - 1) else v)
    return out


def value(m, e):
    return Fraction(0) if m == 0 else Fraction(m) * Fraction(2) ** e


@pytest.mark.parametrize("L,dL,W,R1,NN,KW,m0", [
    (6, 0, 1, 1, 5, 2, 0),                  # one term, one order
    (6, 4, 5, 4, 9, 2, 0),                  # one chunk of orders exactly
    (10, 0, 7, 5, 11, 2, 2),                # one order into the second chunk
    (18, 4, 6, 9, 11, 2, 0),
    (34, 4, 8, 12, 41, 2, 30),              # the levels end inside the table
    (42, 4, 8, 28, 81, 6, 72),
    (46, 0, 3, 28, 200, 12, 190),           # the most limbs, integers of up to seven words
])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_flush_against_exact_sums(cuda, L, dL, W, R1, NN, KW, m0, accumulate):
    LO, rows, N, NB = L + dL, 7, 3, 32 * L - 2
    g = torch.Generator().manual_seed(100 * L + W)
    Y = mpf.random_mpf((W, rows, N), L, spread=40, device=cuda, generator=g)
    dead = torch.rand((W, rows, N), generator=g).to(cuda) < 0.2
    Y.m[:, dead], Y.e[dead] = 0, mpf.EZ
    Y.m[:, :, 1], Y.e[:, 1] = 0, mpf.EZ                                    # a row without terms
    w = torch.arange(W, device=cuda)[:, None]
    for row, step in ((2, 31), (3, 32 * (LO + KW) // 2 + 5), (4, 32 * (LO + 2 + KW) - NB + 32)):
        live = Y.e[:, row] != mpf.EZ                                       # word boundaries, terms cut off in part or whole
        Y.e[:, row] = torch.where(live, -step * w, Y.e[:, row])
    shift = torch.tensor([1, 2, 1, 3, 1, 0, 2], dtype=torch.int64, device=cuda)    # row 5: n = 0 at level 0 of m0 = 0
    nk, nkb = power_table(R1, NN, KW, cuda)
    start = mpf.random_mpf((rows, R1, N), LO, spread=20, device=cuda, generator=g)
    out = mpf.MPF(start.m.clone(), start.e.clone())
    p = lambda t: t.data_ptr()
    _lib.call("b3d_moments_flush", L, p(Y.m), p(Y.e), Y.m.stride(0), p(shift), m0, W, rows, N, R1, p(nk), p(nkb), NN, KW,
              accumulate, LO, p(out.m), p(out.e), out.m.stride(0), torch.cuda.current_stream(cuda).cuda_stream)
    ym, ye = integers(Y.m, L), Y.e.reshape(-1).tolist()
    om, oe = integers(out.m, LO), out.e.reshape(-1).tolist()
    sm, se = integers(start.m, LO), start.e.reshape(-1).tolist()
    for row in range(rows):
        for c in range(N):
            terms = [(m0 + v + int(shift[row]), (v * rows + row) * N + c) for v in range(W)]
            terms = [(n, ym[i], ye[i]) for n, i in terms if ye[i] != mpf.EZ and n < NN]
            for k in range(R1):
                o = (row * R1 + k) * N + c
                parts = [(n ** k, m, e) for n, m, e in terms if n ** k]
                exact = sum((value(b * m, e) for b, m, e in parts), Fraction(0))
                bound = Fraction(0)
                if parts:
                    top = max(e + NB + b.bit_length() for b, _, e in parts)
                    bound = W * Fraction(2) ** (top - 32 * (LO + 2))
                    if exact:                                              # half a unit of the sum's NB bits
                        q = abs(exact)
                        bits = q.numerator.bit_length() - q.denominator.bit_length() + 1
                        bound += Fraction(2) ** (bits - (32 * LO - 2)) / 2
                if accumulate:
                    exact += value(sm[o], se[o])
                    if parts:                                              # the addition rounds once more
                        bound += Fraction(2) ** oe[o] / 2 if om[o] else 0
                got = value(om[o], oe[o])
                assert abs(got - exact) <= bound, (row, c, k)
                assert om[o] == 0 or abs(om[o]).bit_length() == 32 * LO - 2
