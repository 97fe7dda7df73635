"""Alignment (b3d_align) against integers: short and long rows along either stride, row counts around the block's, batches
picked by index, both output orders."""
import pytest
import torch

from blocksvibe_b200 import _lib, mpf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 70])
@pytest.mark.parametrize("rows_first,kmajor,R", [(True, 0, 7), (True, 1, 130), (False, 1, 33), (False, 0, 129)])
def test_align_against_integers(cuda, K, rows_first, kmajor, R):
    L, nb = 6, 3
    g = torch.Generator().manual_seed(100 * K + R)
    X = mpf.random_mpf((4, R, K) if rows_first else (4, K, R), L, spread=40, device=cuda, generator=g)
    dead = torch.rand(X.e.shape, generator=g).to(cuda) < 0.3
    dead[1, :3] = True                                       # rows (or slices of k) of zeros
    X.m[:, dead], X.e[dead] = 0, mpf.EZ
    X.e[~dead] += 32 * L * torch.randint(0, 2, (int((~dead).sum()),), generator=g).to(cuda)   # some fall out whole
    bidx = torch.tensor([2, 0, 1], dtype=torch.int64, device=cuda)
    om = torch.full((L, nb * R * K), -1, dtype=torch.int32, device=cuda)
    oe = torch.full((nb, R), -1, dtype=torch.int64, device=cuda)
    sr, sk = (K, 1) if rows_first else (1, R)
    _lib.call("b3d_align", L, X.m.data_ptr(), X.e.data_ptr(), X.m.stride(0), nb, R, K, R * K, sr, sk, bidx.data_ptr(),
              om.data_ptr(), oe.data_ptr(), om.stride(0), kmajor, torch.cuda.current_stream(cuda).cuda_stream)
    vals, exps = mpf.to_ints(X), oe.reshape(-1).tolist()
    planes = [[w & 0xFFFFFFFF for w in p] for p in om.cpu().tolist()]
    got = [sum(w << (32 * i) for i, w in enumerate(ws)) for ws in zip(*planes)]
    got = [v - (1 << (32 * L)) if v >> (32 * L - 1) else v for v in got]
    for b, src in enumerate(bidx.tolist()):
        for r in range(R):
            row = [vals[src * R * K + r * sr + k * sk] for k in range(K)]
            E = max((e for m, e in row if m), default=mpf.EZ)
            assert exps[b * R + r] == E
            for k, (m, e) in enumerate(row):
                a = abs(m) >> (E - e) if m else 0
                assert got[(b * K + k) * R + r if kmajor else (b * R + r) * K + k] == (-a if m < 0 else a), (b, r, k)
