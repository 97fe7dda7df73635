"""Both forms of the pole step on the same tasks, every limb count: ordinary sums next to cancelling ones in the same warp (the
exact redo of a lane beside lanes that round directly), absent entries, a ragged second chunk of columns."""
import pytest
import torch

from blocksvibe_b200 import _lib, build, mpf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", build.LIMBS)
@pytest.mark.parametrize("S,B,T", [(2, 7, 40), (3, 5, 40), (5, 6, 40), (5, 9, 20), (8, 5, 12)])
def test_forms_bitwise_equal(cuda, L, S, B, T):
    g = torch.Generator().manual_seed(100 * L + S)
    NB = mpf.nbits(L)
    R, Q = mpf.random_mpf((6, S, S), L, device=cuda, generator=g), mpf.random_mpf((9, S, S), L, device=cuda, generator=g)
    for M in (R, Q):                                         # column 1 = -column 0: the two cancel where H repeats
        M.m[..., 1] = ~M.m[..., 0]                           # one unit off the negative: a remainder of a few bits
        M.e[..., 1] = M.e[..., 0]
    H = mpf.random_mpf((T, S, S, B), L, spread=6, device=cuda, generator=g)
    k = torch.arange(B, device=cuda)
    same = (k % 3 == 1)
    H.m[:, :, :, 1, same], H.e[:, :, 1, same] = H.m[:, :, :, 0, same], H.e[:, :, 0, same]
    if S > 2:                                                # nothing else in some of the cancelling columns
        H.m[:, ::2, :, 2:, 1], H.e[::2, :, 2:, 1] = 0, mpf.EZ
    H.m[:, :, 1::2] = H.m[:, :, 0:S - S % 2:2]               # rows repeat: the second stage cancels as well
    H.e[:, 1::2] = H.e[:, 0:S - S % 2:2]
    H.m[L - 1, :, :, :, 3 % B] ^= 1 << 12                    # a bit of the top limb of one column
    H.m[:, 3], H.e[3] = 0, mpf.EZ
    H = H.reshape(T, S * S * B)
    Ra, Qa = mpf.align_rows(R), mpf.align_rows(Q)
    idx = lambda n: torch.randint(0, n, (T,), generator=g).to(cuda)
    tR, tQ, ar = idx(6), idx(9), torch.arange(T, device=cuda)
    p = lambda t: t.data_ptr()
    err = torch.zeros(1, dtype=torch.int32, device=cuda)
    out = []
    for entry, tail in (("b3d_pole_level", ()), ("b3d_pole_level_mma", (p(err),))):
        Y, O = mpf.zeros((T, S * S, B), L, cuda), mpf.zeros((T, S * S, B), L, cuda)
        _lib.call(entry, L, p(H.m), p(H.e), H.m.stride(0), p(Ra[0]), p(Ra[1]), Ra[0].stride(0), p(Qa[0]), p(Qa[1]), Qa[0].stride(0),
                  p(ar), p(tR), p(tQ), p(ar), T, B, S, p(Y.m), p(Y.e), Y.m.stride(0), p(O.m), p(O.e), O.m.stride(0), *tail,
                  torch.cuda.current_stream(cuda).cuda_stream)
        out.append((Y, O))
    assert int(err.item()) == 0
    (Y0, O0), (Y1, O1) = out
    assert int((O0.e == mpf.EZ).sum()) > 0 and int((O0.e != mpf.EZ).sum()) > 0
    assert torch.equal(Y0.m, Y1.m) and torch.equal(Y0.e, Y1.e)
    assert torch.equal(O0.m, O1.m) and torch.equal(O0.e, O1.e)
