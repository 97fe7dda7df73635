"""The tensor-core flush of the staged moments (b3d_moments_flush_mma) against the CUDA-core one (b3d_moments_flush) on
synthetic windows: both sum exactly above 2^-(32 Lout + 64) of the largest term and round once, so without
cancellation down to that depth they give the same bits."""
import numpy as np
import pytest
import torch

from blocksvibe_b200 import _lib, mpf

pytestmark = pytest.mark.gpu


def power_table(R1, NN, KW, device):
    limbs, bits = np.zeros((R1, NN, KW), dtype=np.uint32), np.zeros((R1, NN), dtype=np.int32)
    for k in range(R1):
        for n in range(NN):
            v = n ** k
            bits[k, n] = v.bit_length()
            for j in range(KW):
                limbs[k, n, j] = (v >> (32 * j)) & 0xFFFFFFFF
    return torch.as_tensor(limbs.view(np.int32), device=device), torch.as_tensor(bits, device=device)


@pytest.mark.parametrize("L,dL,W,R1,NN,KW,m0,N", [
    (10, 0, 10, 1, 20, 2, 0, 1),               # one order, the fewest levels, one column
    (6, 4, 32, 6, 40, 2, 3, 5),                # one K step exactly, columns 4 + 1
    (34, 4, 33, 12, 41, 2, 0, 7),              # one level into the second K step
    (34, 0, 40, 12, 41, 2, 0, 3),
    (30, 0, 64, 8, 66, 2, 1, 4),               # every digit of n^k in a K block of its own
    (26, 4, 48, 16, 49, 6, 0, 9),
    (42, 4, 72, 28, 81, 6, 0, 6),              # the largest: R = 27, order 80
    (42, 0, 80, 28, 81, 6, 2, 2),
    (46, 0, 128, 4, 200, 2, 0, 3),             # the most levels
    (10, 0, 9, 4, 20, 2, 0, 5),                # too few levels: the CUDA-core kernel
    (18, 0, 40, 32, 41, 12, 0, 2),             # integers too long for one tile: the CUDA-core kernel
])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_flush_forms_bitwise_equal(cuda, L, dL, W, R1, NN, KW, m0, N, accumulate):
    LO, rows = L + dL, 7
    g = torch.Generator().manual_seed(L * 1000 + W)
    Y = mpf.random_mpf((W, rows, N), L, spread=60, device=cuda, generator=g)
    dead = torch.rand((W, rows, N), generator=g).to(cuda) < 0.2                 # levels without a term
    Y.m[:, dead] = 0
    Y.e[dead] = mpf.EZ
    Y.m[:, :, 1], Y.e[:, 1] = 0, mpf.EZ                                         # a row without terms
    ones = mpf.from_ints([(1 << (32 * L - 2)) - 1, -(1 << (32 * L - 2)) + 1], [-3, -3], L, (2,), cuda)
    for w in range(W):                                                          # all ones, every sign
        Y.m[:, w, 2], Y.e[w, 2] = ones.m[:, w % 2:w % 2 + 1], -3
    Y.e[1:, 3] -= 32 * (LO + 8) + 13 * torch.arange(1, W, device=cuda)[:, None]  # terms far below the largest
    Y.e[:, 4] += 7 * torch.arange(W, device=cuda)[:, None]
    shift = torch.tensor([1, 2, 3, 1, 5, 0, 1], dtype=torch.int64, device=cuda)  # row 5: n = 0 at level 0
    nk, nkb = power_table(R1, NN, KW, cuda)
    p = lambda t: t.data_ptr()
    st = torch.cuda.current_stream(cuda).cuda_stream
    err = torch.zeros(1, dtype=torch.int32, device=cuda)
    start = mpf.random_mpf((rows, R1, N), LO, spread=90, device=cuda, generator=g)
    out = []
    for name, tail in (("b3d_moments_flush", ()), ("b3d_moments_flush_mma", (p(err),))):
        mom = mpf.MPF(start.m.clone(), start.e.clone())
        _lib.call(name, L, p(Y.m), p(Y.e), Y.m.stride(0), p(shift), m0, W, rows, N, R1, p(nk), p(nkb), NN, KW, accumulate, LO,
                  p(mom.m), p(mom.e), mom.m.stride(0), *tail, st)
        out.append(mom)
    assert int(err.item()) == 0
    assert torch.equal(out[0].m, out[1].m) and torch.equal(out[0].e, out[1].e)
