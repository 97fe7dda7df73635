"""The Cauchy step's double-precision digit form (b3d_cauchy_align_fp + b3d_cauchy_level5) against the two-terms-per-thread
integer form on synthetic levels, bit for bit."""
import pytest
import torch

from blocksvibe_b200 import mpf, recursion as RC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,dmax,N", [(6, 9, 1), (10, 247, 33), (34, 240, 150), (30, 480, 31), (42, 481, 25),
                                      (26, 1900, 70), (34, 1901, 2), (46, 65535, 5)])
def test_cauchy_double_digits_bitwise_equal(cuda, L, dmax, N):
    """the double-precision digit form (k_cauchy5) gives k_cauchy2's bits on synthetic levels: divisors at the ends of
    each digit width's range, vanishing differences, zero and all-ones operands, odd row and column counts, ragged
    groups, widely spread exponents, a level of one column"""
    import ctypes
    from blocksvibe_b200 import _lib
    g = torch.Generator().manual_seed(L * 1000 + N)
    nb, Mr, Kc, nslots, Jh, hl = 3, 7, 9, 20, 2, 3
    res = mpf.random_mpf((nslots, N), L, spread=60, device=cuda, generator=g)
    res.m[:, 3], res.e[3] = 0, mpf.EZ                                    # zero numbers
    ones = mpf.from_ints([(1 << (32 * L - 2)) - 1, -(1 << (32 * L - 2)) + 1], [0, 5], L, (2,), cuda)
    res.m[:, 4], res.e[4] = ones.m[:, :1], ones.e[0]                     # all ones, largest magnitudes
    res.m[:, 5], res.e[5] = ones.m[:, 1:], ones.e[1]
    h = mpf.random_mpf((2, hl, Jh, N), L, spread=4, device=cuda, generator=g)
    i64 = lambda v: torch.tensor(v, dtype=torch.int64, device=cuda)
    rowd = torch.randint(-dmax // 2, dmax // 2 + 1, (nb, Mr), generator=g)
    cold = torch.randint(-dmax // 2, dmax // 2 + 1, (nb, Kc), generator=g)
    rowd[0, 0], cold[0, 0], cold[0, 1] = dmax // 2, dmax // 2 - dmax, dmax // 2          # d = dmax and d = 0
    rowd[0, 1], cold[0, 2] = dmax // 2 - dmax, dmax // 2                                # d = -dmax
    col = torch.randint(0, nslots, (nb, Kc), generator=g)
    col[0, :6] = torch.arange(6)
    t = dict(gsrc=i64([0, 1, 1]), gj=i64([0, 1, 0]), rowd=rowd.to(cuda), nrow=i64([Mr, Mr - 2, 0]), cold=cold.to(cuda),
             ncol=i64([Kc, Kc - 3, 1]), col=col.to(cuda))
    p = lambda x: x.data_ptr()
    tabs = _lib.LevelTables(2, nb, Mr, Kc, N, hl, Jh, *(p(t[k]) for k in ("gsrc", "gj", "rowd", "nrow", "cold", "ncol", "col")))
    st = torch.cuda.current_stream(cuda).cuda_stream
    ref = ctypes.byref(tabs)
    out = []
    for form in (2, 5):
        H = mpf.MPF(torch.full((L, nb * Mr * N), 7, dtype=torch.int32, device=cuda), torch.full((nb * Mr * N,), 7, dtype=torch.int64, device=cuda))
        Xe = torch.empty((nb, N), dtype=torch.int64, device=cuda)
        if form == 2:
            X = torch.empty((L, nb * Kc * N), dtype=torch.int32, device=cuda)
            _lib.call("b3d_cauchy_align", L, p(res.m), p(res.e), res.m.stride(0), ref, p(X), p(Xe), X.stride(0), st)
            _lib.call("b3d_cauchy_level2", L, p(X), p(Xe), X.stride(0), p(h.m), p(h.e), h.m.stride(0), ref, p(H.m), p(H.e),
                      H.m.stride(0), st)
        else:
            X = torch.full((RC.cauchy_fp_size(L, dmax, nb, Kc, N),), float("nan"), dtype=torch.float64, device=cuda)
            _lib.call("b3d_cauchy_align_fp", L, p(res.m), p(res.e), res.m.stride(0), ref, dmax, p(X), p(Xe), st)
            _lib.call("b3d_cauchy_level5", L, p(X), p(Xe), p(h.m), p(h.e), h.m.stride(0), ref, dmax, p(H.m),
                      p(H.e), H.m.stride(0), st)
        out.append((H, Xe))
    assert torch.equal(out[0][1], out[1][1])
    assert torch.equal(out[0][0].m, out[1][0].m) and torch.equal(out[0][0].e, out[1][0].e)
