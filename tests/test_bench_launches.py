"""The bench's launch count: entry points that launch nothing (sizes and choices computed on the host) count nothing."""
import ctypes

from blocksvibe_b200 import _lib


def test_host_only_entries_are_not_counted(monkeypatch):
    import bench
    monkeypatch.setattr(_lib, "call", _lib.call)              # restored after the probe has wrapped it
    probe = bench.Probe()
    n, v = ctypes.c_int64(), ctypes.c_int()
    _lib.call("b3d_cauchy_fp_size", 34, 200, 3, 7, 150, ctypes.addressof(n))
    _lib.call("b3d_moments_flush_form", 38, 40, 12, 41, 2, 12500, 148, ctypes.addressof(v))
    assert n.value > 0 and probe.launches == 0
