"""The rule that picks the members' slices (csrc/hw_slices.hpp) on both sides of its
lines: CTAs of 512 points up to one an SM, of 1024 up to five on four SMs, else 2048; the
SM count is the device's; a cluster of sixteen CTAs only where one can be resident."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include "hw_slices.hpp"
extern "C" void slices(const int* nx, const int* named, int n, int sms, int sixteen, int* out) {
  const std::vector<int> m = hw::choose_slices(std::vector<int>(nx, nx + n), std::vector<int>(named, named + n), sms,
                                               [&](int) { return sixteen != 0; });
  for (int i = 0; i < n; ++i) out[i] = m[size_t(i)];
}
"""


@pytest.fixture(scope="module")
def choose(tmp_path_factory):
    d = tmp_path_factory.mktemp("slices")
    (d / "s.cpp").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "hawassi_c_b200", "csrc"),
                    "-o", str(d / "s.so"), str(d / "s.cpp")], check=True)
    lib = ctypes.CDLL(str(d / "s.so"))

    def call(nx, sms=148, sixteen=True, named=None):
        a = (ctypes.c_int * len(nx))
        out = a()
        lib.slices(a(*nx), a(*(named or [0] * len(nx))), len(nx), sms, int(sixteen), out)
        return list(out)
    return call


@pytest.mark.parametrize("nx,count,sms,want", [
    (256, 1, 148, 256), (1024, 148, 148, 1024), (2048, 1, 148, 512), (4096, 1, 148, 512), (8192, 1, 148, 1024),
    (16384, 1, 148, 1024), (32768, 1, 148, 2048), (2048, 37, 148, 512), (2048, 38, 148, 1024), (2048, 92, 148, 1024),
    (2048, 93, 148, 2048), (4096, 18, 148, 512), (4096, 19, 148, 1024), (4096, 46, 148, 1024), (4096, 47, 148, 2048),
    (16384, 9, 148, 1024), (16384, 11, 148, 1024), (16384, 12, 148, 2048),
    (2048, 33, 132, 512), (2048, 34, 132, 1024), (2048, 82, 132, 1024), (2048, 83, 132, 2048)])
def test_sides_of_the_lines(choose, nx, count, sms, want):
    assert choose([nx] * count, sms) == [want] * count


def test_grids_and_names_together(choose):
    assert choose([1024, 4096] * 8) == [1024, 512] * 8                       # 72 CTAs
    assert choose([512, 2048, 8192] * 16) == [512, 1024, 1024] * 16           # 208 of 512, 176 of 1024 points
    assert choose([512, 2048, 8192] * 17) == [512, 2048, 2048] * 17           # 187 of 1024
    assert choose([4096, 4096], named=[2048, 0]) == [2048, 512]


def test_sixteen_ctas_only_where_resident(choose):
    assert choose([16384, 4096], sixteen=False) == [2048, 512]
    assert choose([16384], sixteen=False, named=[1024]) == [1024]             # named: the launch says so
    assert choose([32768], sixteen=False) == [2048]                           # no smaller cluster holds it
