"""The flags that the tensor-core kernels set when a bounded wait expires (results incomplete) are read wherever results are
handed over: a flag that the test sets by hand, as an expired wait would, makes each hand-over raise, and stays set
for the other batches of the operator."""
import threading
from types import SimpleNamespace

import pytest
import torch

from blocksvibe_b200 import _lib, dropin as DI, rns, serve


def flag(v=0, device="cpu"):
    return torch.full((1,), v, dtype=torch.int32, device=device)


@pytest.mark.parametrize("which", range(3))
def test_operator_reads_every_flag(monkeypatch, which):
    flags = [flag(), flag(), flag()]
    monkeypatch.setattr(rns, "_TABLES", {(6, "cpu"): SimpleNamespace(err=flag()), (10, "cpu"): SimpleNamespace(err=flags[2])})
    op = object.__new__(DI.Operator)
    op.rec, op.der, op.device = SimpleNamespace(err=flags[0]), SimpleNamespace(err=flags[1]), torch.device("cpu")
    op.check_errors()
    flags[which].fill_(3)
    for _ in range(2):                                   # the flag stays set for batches on other streams
        with pytest.raises(_lib.B3DError, match="did not complete"):
            op.check_errors()


def test_rns_check_clears_what_it_raises_for(monkeypatch):
    f = flag(2)
    monkeypatch.setattr(rns, "_TABLES", {(6, "cpu"): SimpleNamespace(err=flag()), (10, "cpu"): SimpleNamespace(err=f)})
    with pytest.raises(_lib.B3DError, match="code 2"):
        rns.check_errors("cpu")
    rns.check_errors(torch.device("cpu"))


def test_threads_share_one_table(monkeypatch):
    """two threads that need a limb count's tables first get the same ones: a flag set in a copy would never be read"""
    both = threading.Barrier(2)

    class Slow:
        def __init__(self, L, device):
            both.wait(10)                                # both are building
            self.err = flag()

    monkeypatch.setattr(rns, "_TABLES", {})
    monkeypatch.setattr(rns, "Tables", Slow)
    got = []
    ts = [threading.Thread(target=lambda: got.append(rns.tables(6, torch.device("cpu")))) for _ in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert got[0] is got[1] and rns.error_flags("cpu")[0] is got[0].err


@pytest.fixture(scope="module")
def group():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from test_gpu_dropin import make_group
    G, tasks, M, _, _ = make_group(nq=1, seed=31, coords=("xt",))
    return G, tasks[0], M


def operator(group, device):
    G, t, M = group
    return DI.Operator(G, t.pp, t.parity, M, t.two_js_internal, ["xt"], [t.delta_1_plus_2], device)


@pytest.mark.gpu
@pytest.mark.parametrize("device", ["cuda", "cuda:0"])
@pytest.mark.parametrize("part", ["rec", "der", "rns"])
def test_hand_over_raises(cuda, group, device, part):
    G, t, M = group
    op = operator(group, device)
    ns = t.lambda_orders(G.Lambda)
    step = DI.GraphStep(op, 1, ns, t.delta_1_plus_2)
    out = step.run([t])
    op.to_host(out)
    err = rns.tables(op.L, torch.device("cuda:0")).err if part == "rns" else getattr(op, part).err
    err.fill_(1)
    try:
        with pytest.raises(_lib.B3DError, match="did not complete"):
            op.to_host(out)
        with pytest.raises(_lib.B3DError, match="did not complete"):
            list(step.run_stream([[t]]))
        with pytest.raises(_lib.B3DError, match="did not complete"):
            step.check_errors()
        if part == "rns":                                # shared by every operator of the device
            with pytest.raises(_lib.B3DError, match="did not complete"):
                DI.run_group(G, [t], M, device=device)
        for host in (True, False):
            srv = serve.Server(device, workers=1, host_results=host)
            srv.add_operator(op, G, t)
            try:
                with pytest.raises(_lib.B3DError, match="did not complete"):
                    srv.wait(srv.submit(G, t, M), timeout=300)
                if part != "rns":                        # the next request builds the operator anew
                    assert srv.wait(srv.submit(G, t, M), timeout=300)
                    assert list(srv.ops.values()) != [op]
            finally:
                srv.close()
    finally:
        err.zero_()
    op.check_errors()
    assert len(list(step.run_stream([[t], [t]]))) == 2
