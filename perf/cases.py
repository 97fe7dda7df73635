"""The timed cases of the framework: its layers (the radial recursion, the derivative stages, the write_output maps,
the multiprecision product, the JSON writer) and whole tasks, each through the entry point that a program calls.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (the operator of the
case with its constants, built once and kept, and inputs drawn from the seed), ``run`` is one pass.  Numbers are
multiprecision: limb planes (int32) and exponents (int64), so every output is compared bit for bit and none has
a value in 64-bit floating point.

Sizes are those of the benchmark configurations (``blocksvibe_b200.workloads``): 256 to 1280 bits, spins up to
40, orders 10 to 80, Lambda 5 to 27, one to five structures a side, one to some dozens of right-hand sides."""
import math
import random

import numpy as np
import torch

from blocksvibe_b200 import dropin, jsonout, mpf, structure, workloads
from blocksvibe_b200.derivatives import Derivs
from blocksvibe_b200.output import Output, apply_per_order
from blocksvibe_b200.plan import Plan
from blocksvibe_b200.recursion import Recursion

DEVICE = "cuda"
PP = (((0, 0), (1, 1)), ((0, 1), (1, 0)), ((0, 1), (1, 1)), ((1, 0), (0, 1)))   # pseudo-parity types, by "pp"


def _op(tj12, tj43, tjmax, Lam, order, kept, precision, coord="xt", pp=0, sign=1):
    return dict(tj12=tj12, tj43=tj43, tjmax=tjmax, Lam=Lam, order=order, kept=kept, precision=precision, coord=coord,
                pp=pp, sign=sign)


def listed():
    return [
        # the smallest call: the write_output product of a 256-bit task (launch latency and host work)
        dict(name="gemm_256_map", kind="gemm", precision=256, batch=1, M=12, N=294, K=12),
        # an odd-sized batched product of the derivative stages, 1280 bits
        dict(name="gemm_1280_batched", kind="gemm", precision=1280, batch=9, M=45, N=611, K=77),
        # a small task from beginning to end: hundreds of launches, none of them large
        dict(name="task_256", kind="task", nq=1, graph=False, **_op(0, 0, 12, 5, 10, 6, 256)),
        # one lambda order of a stress-tensor task: the plain schedule's recursion
        dict(name="recursion_1024_one_order", kind="recursion", B=1, **_op(8, 8, 44, 11, 40, 20, 1024)),
        # all lambda orders of a stress-tensor task in one recursion: the batched schedule
        dict(name="recursion_1024", kind="recursion", B=6, **_op(8, 8, 44, 11, 40, 20, 1024)),
        # seven tasks of the 644-task set together: three structures, 768 bits, mixed parity
        dict(name="recursion_768_seven_tasks", kind="recursion", B=42, **_op(2, 4, 16, 11, 40, 20, 768, pp=1)),
        # moments and numerators of a stress-tensor task, with pole shifting
        dict(name="derivatives_1024", kind="derivatives", B=6, R=11, **_op(8, 8, 44, 11, 40, 20, 1024)),
        # the same without pole shifting at half-integer spins: an odd lambda order, three structures of two sides
        dict(name="derivatives_896_odd", kind="derivatives", B=5, R=6, **_op(1, 1, 33, 7, 32, 32, 896, pp=1, sign=-1)),
        # write_output maps of two tasks at Lambda 15
        dict(name="output_896_xt", kind="output", nq=2, Jo=13, S=3, D=57, **_op(2, 2, 24, 15, 48, 24, 896)),
        # the JSON files of a 768-bit task, assembled on the device into the program's buffer
        dict(name="json_768", kind="json", **_op(2, 2, 22, 7, 32, 16, 768)),
        # the benchmark's task: recursion, derivatives, numerators and maps as one replayed graph
        dict(name="task_1024_graph", kind="task", nq=1, graph=True, **_op(8, 8, 44, 11, 40, 20, 1024)),
        # the largest task: spins 0-40, Lambda 27, order 80, 1280 bits, xt_radial with pole shifting
        dict(name="task_1280", kind="task", nq=1, graph=False, **_op(8, 8, 80, 27, 80, 40, 1280, coord="xt_radial")),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_operator(rng):
    tj12, tj43 = rng.choice(((0, 0), (1, 1), (2, 0), (2, 2), (2, 4), (4, 4), (6, 4), (8, 8)))
    Lam = rng.choice((5, 7, 11, 15))
    order = 10 if Lam == 5 else 2 * Lam + 18
    kept = rng.choice((Lam + 1 if Lam == 5 else Lam + 9, order))
    top = rng.randint(4, 8 if Lam == 5 else 30)
    return _op(tj12, tj43, 2 * top + tj12 % 2, Lam, order, kept, rng.choice((256, 512, 768, 896, 1024, 1280)),
               rng.choice(("xt", "xt_radial")), rng.randrange(4) if tj12 and tj43 else 0, rng.choice((1, -1)))


MAX_FLOPS = 4e13                # under a third of the largest listed case's


def draw(rng):
    while True:
        kind = rng.choice(("gemm", "recursion", "derivatives", "output", "json", "task"))
        if kind == "gemm":
            c = dict(kind=kind, precision=rng.choice((256, 512, 768, 896, 1024, 1280)), batch=_log_int(rng, 1, 40),
                     M=_log_int(rng, 1, 160), N=_log_int(rng, 1, 4000), K=_log_int(rng, 1, 250))
        else:
            c = dict(kind=kind, **_draw_operator(rng))
            if kind == "recursion":
                c["B"] = _log_int(rng, 1, 60)
            elif kind == "derivatives":
                c.update(B=_log_int(rng, 1, 24), R=rng.randint(1, c["Lam"]))
            elif kind == "output":
                c.update(nq=_log_int(rng, 1, 9), Jo=rng.randint(1, 31), S=rng.randint(1, 5), D=rng.randint(20, 90))
            elif kind == "json":
                c["precision"] = rng.choice((256, 512, 768))
                c["Lam"] = rng.choice((5, 7))
            else:
                c.update(nq=_log_int(rng, 1, 7), graph=rng.random() < 0.3)
        if work(c)["flops"] < MAX_FLOPS:
            return c


# ---------------------------------------------------------------- what a program keeps
_KEPT = {}                      # operators and graphs of the cases met so far


def _kept(key, build):
    if key not in _KEPT:
        while len(_KEPT) >= 24:
            _KEPT.pop(next(iter(_KEPT)))
        _KEPT[key] = build()
    return _KEPT[key]


def _orders(c):
    parity = (1 - c["sign"]) // 2
    return [parity] if c["coord"].endswith("_radial") else list(range(parity, c["Lam"] + 1, 2))


def _spins(c):
    return list(range(c["tj12"] % 2, c["tjmax"] + 1, 2))


def _group(c):
    return dropin.Group((0, 0, 0, 0), c["tj12"], c["tj43"], c["order"], c["Lam"], c["tjmax"], c["precision"], c["kept"])


def _plan(c):
    return _kept(("plan",) + tuple(c[k] for k in ("tj12", "tj43", "tjmax", "order", "pp")),
                 lambda: Plan(c["tj12"], c["tj43"], c["tjmax"], c["order"], PP[c["pp"]], reuse=True))


def _case_key(c, *more):
    return tuple(sorted((k, v) for k, v in c.items() if k not in ("name", "nq", "B", "graph"))) + more


def _operator(c):
    return _kept(_case_key(c, "operator"), lambda: dropin.Operator(
        _group(c), PP[c["pp"]], (1 - c["sign"]) // 2, None, _spins(c), (c["coord"],), ("0.5",), DEVICE))


# ---------------------------------------------------------------- inputs
def _numbers(shape, L, gen, spread=2):
    """random normalised numbers of both signs, |x| in about [2^-spread, 2^spread]"""
    n = math.prod(shape)
    m = torch.randint(-2 ** 31, 2 ** 31, (L, n), dtype=torch.int32, device=DEVICE, generator=gen)
    # the top limb of a number of NB = 32 L - 2 bits: [2^29, 2^30), or [-2^30, -2^29) for a negative one
    top = torch.randint(0, 2 ** 29, (n,), dtype=torch.int32, device=DEVICE, generator=gen)
    neg = torch.randint(0, 2, (n,), dtype=torch.int32, device=DEVICE, generator=gen)
    m[L - 1] = torch.where(neg == 1, top - 2 ** 30, top + 2 ** 29)
    e = torch.randint(-spread, spread + 1, (n,), device=DEVICE, generator=gen) - mpf.nbits(L)
    return mpf.MPF(m.reshape((L,) + tuple(shape)), e.reshape(shape))


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def prepare(case, seed):
    c, gen = case, _generator(seed)
    L = mpf.limbs_for_precision(c["precision"])
    kind = c["kind"]
    if kind == "gemm":
        return dict(kind=kind, A=_numbers((c["batch"], c["M"], c["K"]), L, gen, 8),
                    B=_numbers((c["batch"], c["K"], c["N"]), L, gen, 8))
    if kind == "recursion":
        plan = _plan(c)
        rec = _kept(_case_key(c, "recursion"), lambda: Recursion(plan, None, L, device=DEVICE))
        return dict(kind=kind, rec=rec, h=_numbers((2, c["order"] + 1, plan.Jh, plan.Smax ** 2, c["B"]), L, gen))
    if kind == "derivatives":
        plan = _plan(c)
        der = _kept(_case_key(c, "derivatives"),
                    lambda: Derivs(plan, c["R"], L, kept_pole_order=c["kept"], device=DEVICE))
        # residues fall off with the level in earnest; slots are recycled, so every slot gets the whole range
        return dict(kind=kind, der=der, B=c["B"], levels=len(plan.levels),
                    res=_numbers((plan.nphys + 1, plan.Smax ** 2, c["B"]), L, gen, 20),
                    h=_numbers((2, c["order"] + 1, plan.Jh, plan.Smax ** 2, c["B"]), L, gen))
    if kind == "output":
        out = _kept(_case_key(c, "output"),
                    lambda: Output(c["coord"], c["Lam"], (1 - c["sign"]) // 2, "0.5", L, DEVICE))
        ns = _orders(c)
        nums = []
        for n in ns:
            R1, D = c["Lam"] - n + 1, c["D"] - n                # a lambda order less is a coefficient less
            nums.append(_numbers((c["Jo"], D, R1, 2, c["S"] ** 2, c["nq"]), L, gen, 30))
        return dict(kind=kind, out=out, nums=nums)
    if kind == "json":
        return _prepare_json(c, L, gen)
    op = _operator(c)
    ns, nq = _orders(c), c["nq"]
    plan = op.plan
    if c["graph"]:
        step = _kept(_case_key(c, "graph", nq), lambda: dropin.GraphStep(op, nq, ns, "0.5"))
        tasks = []
        for q in range(nq):
            t = dropin.Task((q, 0, 0, 0), c["sign"], PP[c["pp"]], _spins(c), (c["coord"],), "0.5")
            for n in ns:
                t.h_inf[n] = _numbers((2, c["order"] + 1, plan.Jh, plan.Smax ** 2), L, gen)
            tasks.append(t)
        return dict(kind="graph", step=step, tasks=tasks)
    return dict(kind=kind, op=op, ns=ns, nq=nq,
                h=_numbers((2, c["order"] + 1, plan.Jh, plan.Smax ** 2, nq * len(ns)), L, gen))


def _output_rows(c):
    """(derivative, derivative) pairs of the write_output rows"""
    O, p = c["Lam"], (1 - c["sign"]) // 2
    if c["coord"] == "xt_radial":
        return [(i, 0) for i in range(O - p + 1)]
    return [(n, b) for n in range(O - p + 1) for b in range((O - n - p) // 2 + 1)]


def _json_shape(c):
    S = min(c["tj12"], c["tj43"], 4) // 2 + 1
    return len(_spins(c)), S, _output_rows(c), 2 * c["Lam"] + 16


def _prepare_json(c, L, gen):
    Jo, S, rows, D = _json_shape(c)
    group = _group(c)
    task = dropin.Task((0, 0, 0, 0), c["sign"], PP[c["pp"]], _spins(c), (c["coord"],), "0.5")
    Smax = max(len(structure.so3_structures(p, t, tj)) for pp in PP[c["pp"]] for p, t in zip(pp, (c["tj12"], c["tj43"]))
               for tj in _spins(c))
    S = max(S, Smax)
    x = _numbers((Jo, 2, S * S, 1, len(rows), D), L, gen, 10)
    # coefficients of a numerator fall with their degree; some twenty decades over the polynomial
    x.e.sub_(torch.arange(D, device=DEVICE) * 66 // D)
    w = jsonout.SpinWriter(jsonout.task_options(group, task), _spins(c), PP[c["pp"]], {c["coord"]: rows}, S, 1, D, DEVICE)
    # the program's buffer for the text: every number at its longest, brackets and headers
    p, n, polys = w.p, x.numel(), Jo * 2 * S * S * len(rows)
    text = torch.zeros(n * (p + 16) + polys * 800 + Jo * 16384, dtype=torch.uint8, device=DEVICE)
    return dict(kind="json", writer=w, outs={c["coord"]: x}, text=text)


# ---------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "gemm":
        C = mpf.gemm(state["A"], state["B"])
        return C.m, C.e
    if kind == "recursion":
        res = state["rec"].run(state["h"])
        return res.m, res.e
    if kind == "derivatives":
        der = state["der"]
        der.start(state["B"])
        for m in range(state["levels"]):
            der.accumulate(m, state["res"])
        num = der.finish(state["h"])
        return num.m, num.e
    if kind == "output":
        out = apply_per_order(state["out"], state["nums"])
        return out.m, out.e
    if kind == "json":
        text, ends, _ = state["writer"].render_device(state["outs"])
        state["text"][:text.numel()].copy_(text)
        return state["text"], np.asarray(ends)
    if kind == "graph":
        outs = state["step"].run(state["tasks"])
    else:
        op = state["op"]
        outs = op.apply_outputs(op.run_batched_h(state["h"], state["nq"], state["ns"]), "0.5")
    return {coord: (x.m, x.e) for coord, x in outs.items()}


def exact(case, seed):
    """Every output is a limb plane, an exponent or a byte: whole numbers, none with a 64-bit floating value."""
    return None


# ---------------------------------------------------------------- what a pass cannot do without
def _recursion_work(c, L, B):
    """bytes of h_inf, the matrices and the residues; multiply-adds of two L-limb numbers (pole step) and of an
    L-limb number with a rational of one limb (Cauchy step)"""
    plan = _plan_host(c)
    S, N = plan["S"], plan["S"] ** 2 * B
    numbers = 2 * (c["order"] + 1) * plan["Jh"] * N + (plan["nM"] + plan["nLQ"]) * S * S + plan["T"] * N
    return numbers, 2 * S * N * plan["T"], plan["terms"] * N


_HOST = {}


def _plan_host(c):
    key = tuple(c[k] for k in ("tj12", "tj43", "tjmax", "order", "pp"))
    if key not in _HOST:
        p = _plan(c)
        levels = [lev for lev in p.levels if lev]
        _HOST[key] = dict(S=p.Smax, Jh=p.Jh, nM=len(p.Mkeys), nLQ=len(p.LQpairs), T=sum(len(v["t_slot"]) for v in levels),
                          terms=sum(int((v["nrow"] * v["ncol"]).sum()) for v in levels))
    return _HOST[key]


def _derivatives_macs(c, R, B):
    """(numbers read and written, multiply-adds) of the moments and the numerators"""
    plan = _plan_host(c)
    Jo, R1, S2 = len(_spins(c)), R + 1, plan["S"] ** 2
    poles = [structure.block_poles(tj, c["tj12"], c["tj43"], c["order"]) for tj in _spins(c)]
    NP = sum(len(p) for p in poles)
    kept = NP if c["kept"] >= c["order"] else sum(len(structure.block_poles(tj, c["tj12"], c["tj43"], c["kept"]))
                                                  for tj in _spins(c))
    D = kept + Jo * R1
    cols = 2 * S2 * B
    terms = NP * cols * c["order"]                                    # a residue per pole, level and column
    macs = terms * 1 + R1 * (c["order"] + 1) * Jo * cols              # r_c^n, and c from h_inf
    macs += NP * R1 * R1 * cols + NP * R * R1 * cols                  # a_i[e], G
    macs += sum((len(p) + R1) for p in poles) * (D // Jo) * R1 * cols  # numerators
    return terms + (c["order"] + 1) * Jo * cols + D * R1 * cols, macs


def work(case):
    """flops: byte products of the multiprecision multiply-adds (the tensor cores' unit), two a product"""
    c = case
    L = mpf.limbs_for_precision(c["precision"])
    nb, mac = 4 * L + 8, 2 * (4 * L) ** 2
    kind = c["kind"]
    if kind == "gemm":
        b, M, N, K = c["batch"], c["M"], c["N"], c["K"]
        return dict(bytes=b * (M * K + K * N + M * N) * nb, flops=b * M * N * K * mac)
    if kind == "recursion":
        n, macs, divs = _recursion_work(c, L, c["B"])
        return dict(bytes=n * nb, flops=macs * mac + divs * 2 * 4 * L)
    if kind == "derivatives":
        n, macs = _derivatives_macs(c, c["R"], c["B"])
        return dict(bytes=n * nb, flops=macs * mac)
    if kind == "output":
        rows, cols = len(_output_rows(c)), c["Jo"] * 2 * c["S"] ** 2 * c["nq"] * c["D"]
        inputs = sum(c["Lam"] - n + 1 for n in _orders(c))
        return dict(bytes=(inputs + rows) * cols * nb, flops=rows * inputs * cols * mac)
    if kind == "json":
        Jo, S, rows, D = _json_shape(c)
        n, digits = Jo * 2 * S * S * len(rows) * D, jsonout.digits10(c["precision"])
        return dict(bytes=n * (nb + digits + 5), flops=n * 4 * L * digits)
    ns = _orders(c)
    n, macs, divs = _recursion_work(c, L, c["nq"] * len(ns))
    Jo, S2 = len(_spins(c)), _plan_host(c)["S"] ** 2
    for o in ns:
        macs += _derivatives_macs(c, c["Lam"] - o, c["nq"])[1]
    rows, inputs = len(_output_rows(c)), sum(c["Lam"] - o + 1 for o in ns)
    kept = max(len(structure.block_poles(tj, c["tj12"], c["tj43"], min(c["kept"], c["order"]))) for tj in _spins(c))
    cols = Jo * 2 * S2 * c["nq"] * (kept + c["Lam"] - ns[0] + 1)
    return dict(bytes=(2 * (c["order"] + 1) * _plan_host(c)["Jh"] * S2 * c["nq"] * len(ns) + rows * cols) * nb,
                flops=(macs + rows * inputs * cols) * mac + divs * 2 * 4 * L)


if __name__ == "__main__":
    for k in listed() + [draw(random.Random(s)) for s in range(12)]:
        w = work(k)
        print(f"{k.get('name', k['kind']):28s} {w['bytes'] / 1e6:10.2f} MB {w['flops'] / 1e9:12.2f} Gflop")
