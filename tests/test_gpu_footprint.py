"""Recursion.footprint_bytes, by which the serving loop admits batches, covers what run() holds at its peak."""
import pytest
import torch

from blocksvibe_b200 import mpf
from blocksvibe_b200.plan import Plan
from blocksvibe_b200.recursion import Recursion

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cauchy", ["cuda5", "cuda4"])
@pytest.mark.parametrize("args,L,B", [((4, 4, 12, 16), 18, 4), ((0, 0, 20, 60), 26, 1), ((0, 0, 8, 122), 10, 3)])
def test_footprint_covers_the_peak(cuda, cauchy, args, L, B):
    plan = Plan(*args, ((0, 0), (1, 1)), reuse=True)
    rec = Recursion(plan, None, L, device=cuda, cauchy=cauchy)
    h = mpf.random_mpf((2, plan.order + 1, plan.Jh, plan.Smax ** 2, B), L, device=cuda)
    rec.run(h)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_stats()["requested_bytes.all.current"]
    rec.run(h)
    peak = torch.cuda.memory_stats()["requested_bytes.all.peak"] - before
    need = rec.footprint_bytes(B)
    assert peak <= need + 4096 and need < 1.35 * peak + 4096           # and a few small tensors
