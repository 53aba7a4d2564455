"""third() of the field kernels (x / 3 by a product and its remainder), compiled for the
host from its source, against the division: the same bits for any x, subnormal,
infinite, NaN and negative zero among them."""
import os
import re
import subprocess

import solids4foam_gb300 as sg

HEADER = os.path.join(os.path.dirname(sg.__file__), "csrc", "device_common.cuh")

MAIN = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
using std::isfinite;
static double __dmul_rn(double a, double b) { return a * b; }
static uint64_t bits(double x) { uint64_t b; std::memcpy(&b, &x, 8); return b; }
static int __double2hiint(double x) { return (int)(bits(x) >> 32); }
static int __double2loint(double x) { return (int)bits(x); }
static double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
%s
int main() {
  uint64_t s = 88172645463325252ull;
  long bad = 0;
  for (int i = 0; i < 3000000; ++i) {
    s ^= s << 13; s ^= s >> 7; s ^= s << 17;
    uint64_t b = s;  // any bits, and every third one a small exponent
    if (i %% 3 == 0) b = (b & 0x800fffffffffffffull) | ((s >> 20) %% 120) << 52;
    if (i < 4) b = (uint64_t)(i & 1) << 63 | (i < 2 ? 0ull : 0x7ffull << 52);
    double x, a, c;
    std::memcpy(&x, &b, 8);
    a = third(x);
    c = x / 3.0;
    if (std::memcmp(&a, &c, 8) && !(a != a && c != c)) ++bad;
  }
  std::printf("%%ld\n", bad);
}
"""


def test_third_is_the_division(tmp_path):
    with open(HEADER) as f:
        src = re.search(r"__device__ __forceinline__ (double third\(double x\) \{.*?\n\})", f.read(), re.S)
    cpp, exe = tmp_path / "third.cpp", tmp_path / "third"
    cpp.write_text(MAIN % src.group(1))
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", str(cpp), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "0\n"
