"""Kernel attributes belong to a device: what sets them (csrc/once.h, compiled
here on its own) runs once for each device of the process and again after a
failure."""
import ctypes as C
import os
import subprocess

CSRC = os.path.join(os.path.dirname(__file__), "..", "gpu-intensities_gb300", "csrc")
HARNESS = r"""
#include "once.h"
static gi::OncePerDevice once;
static int calls;
extern "C" int run(int device, int result) { return once.run(device, [&] { ++calls; return result; }); }
extern "C" int count() { return calls; }
"""


def test_each_device_is_set_up(tmp_path):
    (tmp_path / "h.cpp").write_text(HARNESS)
    so = str(tmp_path / "h.so")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}",
                           str(tmp_path / "h.cpp"), "-o", so])
    L = C.CDLL(so)
    assert [L.run(0, 0), L.run(0, 9), L.count()] == [0, 0, 1]
    assert [L.run(1, 2), L.count()] == [2, 2]           # another device; it fails
    assert [L.run(1, 0), L.run(1, 5), L.count()] == [0, 0, 3]
    assert [L.run(0, 7), L.count()] == [0, 3]
    for device in (-1, 64, 1 << 20):                    # not remembered: set up on every call
        n = L.count()
        assert [L.run(device, 0), L.run(device, 3), L.count()] == [0, 3, n + 2]
