"""The carry chains of csrc/mp.cuh on the device (inline PTX, which the host check does not compile) against Python integers:
sums, differences and products of 1 to 20 limbs, results over either operand, and a loop that carries the limbs of each result
into other limbs' variables."""
import ctypes
import os
import random
import subprocess

import pytest
import torch

from blocksvibe_b200 import build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
RESULTS, CASES, TURNS = 13, 192, 7


@pytest.fixture(scope="module")
def check(cuda, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("chains") / "mp_device_check.so")
    subprocess.run([build._nvcc(), *build.ARCH, *build.FLAGS, "-shared", "-o", so, os.path.join(HERE, "mp_device_check.cu")],
                   check=True)
    fn = ctypes.CDLL(so).mp_device_check
    fn.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int]
    return fn


def words(v, n):
    return [(v >> (32 * k)) & 0xFFFFFFFF for k in range(n)]


def number(ws):
    return sum(w << (32 * k) for k, w in enumerate(ws))


@pytest.mark.parametrize("n", range(1, 21))
def test_chains(cuda, check, n):
    rng, mod = random.Random(n), 1 << (32 * n)
    edge = lambda: number([rng.choice((0, 1, 0xFFFFFFFF, 0x80000000, rng.getrandbits(32))) for _ in range(n)])
    pairs = [(edge(), edge()) for _ in range(CASES)]
    pairs[:4] = [(0, 0), (mod - 1, mod - 1), (mod - 1, 0), (0, mod - 1)]       # runs of carries and borrows
    flat = [w for a, b in pairs for v in (a, b) for w in words(v, n)]
    x = torch.tensor(flat, dtype=torch.int64).to(torch.int32).to(cuda)
    y = torch.zeros(CASES * RESULTS * n, dtype=torch.int32, device=cuda)
    assert check(n, x.data_ptr(), y.data_ptr(), CASES, TURNS) == 0
    torch.cuda.synchronize()
    got = [v & 0xFFFFFFFF for v in y.tolist()]
    for t, (a, b) in enumerate(pairs):
        c, m = t & 1, (a & 0xFFFFFFFF) | 1
        s, d = a + b + c, a - b - c
        want = [s, s, s, d, d, d, a + b, b * m, b * m, b * m, -a]
        u, v = words(a, n), words(b, n)
        for _ in range(TURNS):
            r = words((number(u) + number(v) + c) % mod, n)
            q = words((number(r) - number(u) - c) % mod, n)
            u, v = [r[(k + 1) % n] for k in range(n)], [q[(k + n - 1) % n] for k in range(n)]
        want += [number(u), (s >> (32 * n)) | (d < 0) << 1]
        o = t * RESULTS * n
        have = [number(got[o + i * n:o + (i + 1) * n]) for i in range(RESULTS)]
        assert have == [w % mod for w in want], (t, a, b)
