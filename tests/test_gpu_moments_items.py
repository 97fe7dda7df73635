"""The tensor-core flush with several items per CTA (coefficients kept between the items of a row and formed anew at the next, the
limb buffers and the barrier reused, rows of n = 0 and rows without terms in between, a last group of fewer columns) and with
one partly filled K step, against the CUDA-core form, bit for bit as in test_gpu_moments_mma."""
import pytest
import torch

from blocksvibe_b200 import _lib, mpf
from test_flush_rule import flush_form
from test_gpu_moments_mma import power_table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,dL,W,R1,NN,KW,m0,rows,N", [
    (10, 0, 10, 13, 20, 2, 0, 331, 9),             # ten levels of a K step, three items of a row
    (6, 4, 31, 5, 40, 2, 0, 700, 3),               # one level short of a K step; a row is one item
    (26, 4, 20, 8, 41, 2, 3, 500, 6),
    (34, 4, 40, 12, 41, 2, 0, 350, 9),             # two CTAs per SM
    (42, 4, 72, 28, 81, 6, 0, 170, 5),             # one CTA per SM, two columns an item
])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_flush_items_bitwise_equal(cuda, L, dL, W, R1, NN, KW, m0, rows, N, accumulate):
    LO = L + dL
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    assert flush_form(LO, W, R1, NN, KW, rows * N, sms) == 1 and rows * -(-N // 4) > 2 * sms * (L < 42)
    g = torch.Generator().manual_seed(L * 1000 + W)
    Y = mpf.random_mpf((W, rows, N), L, spread=60, device=cuda, generator=g)
    dead = torch.rand((W, rows, N), generator=g).to(cuda) < 0.2
    dead |= (torch.arange(rows, device=cuda) % 11 == 4)[None, :, None]                  # rows without terms
    dead[:, 17, 1:] = True                                                              # one live column of an item
    Y.m[:, dead], Y.e[dead] = 0, mpf.EZ
    shift = torch.randint(1, 5, (rows,), generator=g)
    shift[::7] = 0                                                                      # n = 0 at level 0 of m0 = 0
    shift[40:60] = 2                                                                    # the same n from row to row
    shift = shift.to(cuda)
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


@pytest.mark.parametrize("L,W,R1,NN,KW,wide", [(6, 5, 4, 9, 1, 2), (10, 6, 9, 30, 3, 6), (10, 12, 20, 60, 7, 12), (18, 40, 12, 41, 5, 6)])
@pytest.mark.parametrize("entry", ["b3d_moments_flush", "b3d_moments_flush_mma"])
def test_tables_of_any_width(cuda, L, W, R1, NN, KW, wide, entry):
    """n^k in KW words, not only the widths compiled: the same bits as from a wider table"""
    rows, N = 9, 4
    g = torch.Generator().manual_seed(L + W)
    Y = mpf.random_mpf((W, rows, N), L, spread=30, device=cuda, generator=g)
    shift = torch.arange(rows, device=cuda) % 3
    st = torch.cuda.current_stream(cuda).cuda_stream
    err = torch.zeros(1, dtype=torch.int32, device=cuda)
    tail = (err.data_ptr(),) if entry.endswith("mma") else ()
    out = []
    for kw in (KW, wide):
        nk, nkb = power_table(R1, NN, kw, cuda)
        mom = mpf.zeros((rows, R1, N), L, cuda)
        _lib.call(entry, L, Y.m.data_ptr(), Y.e.data_ptr(), Y.m.stride(0), shift.data_ptr(), 0, W, rows, N, R1, nk.data_ptr(),
                  nkb.data_ptr(), NN, kw, 0, L, mom.m.data_ptr(), mom.e.data_ptr(), mom.m.stride(0), *tail, st)
        out.append(mom)
    assert int(err.item()) == 0
    assert torch.equal(out[0].m, out[1].m) and torch.equal(out[0].e, out[1].e)
