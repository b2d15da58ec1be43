"""The integer-pipe FP64 quotient and square root (csrc/xc_fp64.cuh), compiled
for the host, against the processor's own: the same bits for every pair of
operands, with the seeds moved by the error the device's approximations may
have (and the wider one of their emulation here)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = r"""
#include <cstdint>
static int g_ulps = 0;
#define XC_SEED_ULPS (g_ulps)
#include "xc_fp64.cuh"
#include <cstdio>
#include <random>
static const uint64_t M = (1ull << 52) - 1;
// significands at the edges of the algorithms: all ones, few bits, long runs
static uint64_t significand(uint64_t v, int kind) {
  uint64_t run = (1ull << ((v >> 58) % 52)) - 1;
  switch (kind) {
    case 0: return v & M;
    case 1: return v & M & ~run;
    case 2: return (v & M) | run;
    case 3: return v & 0xff;
    default: return (v & M) | (M ^ 0xff);
  }
}
int main() {
  std::mt19937_64 g(20);
  long bad = 0;
  const double special[] = {0.0, -0.0, 1.0, 3.0, 5e-324, 2.2250738585072014e-308, 1.7976931348623157e308,
                            1.0 / 0.0, 0.0 / 0.0, 4.0, 2.0, 1.0000000000000002, 0.9999999999999999};
  auto check = [&](double x, double y) {
    const double q = xc_div(x, y), r = x / y, s = xc_sqrt(x), t = std::sqrt(x);
    if (xc_bits(q) != xc_bits(r) && !(q != q && r != r)) { if (bad++ < 5) std::printf("div %a %a: %a not %a\n", x, y, q, r); }
    if (xc_bits(s) != xc_bits(t) && !(s != s && t != t)) { if (bad++ < 5) std::printf("sqrt %a: %a not %a\n", x, s, t); }
  };
  for (g_ulps = -2; g_ulps <= 2; ++g_ulps) {
    for (double x : special) for (double y : special) { check(x, y); check(y, -x); }
    for (long i = 0; i < 3000000; ++i) {
      const uint64_t a = g(), b = g();
      const bool mid = i & 1;     // exponents of ordinary fields, or all of them
      auto make = [&](uint64_t v, int kind) {
        const uint64_t e = mid ? 963 + (v >> 52) % 120 : (v >> 52) & 0x7ff;
        return xc_from_bits((v & (1ull << 63)) | (e << 52) | significand(v, kind));
      };
      const double x = make(a, (i >> 1) % 5), y = make(b, (i / 10) % 5);
      check(std::fabs(x), y);
      check(x, 0.1 + (double)(i % 97));
    }
  }
  std::printf("bad %ld\n", bad);
  return bad != 0;
}
"""


def test_quotient_and_root_have_the_processors_bits(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    src = tmp_path / "probe.cpp"
    src.write_text(PROBE)
    exe = tmp_path / "probe"
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "xcore.jl_gb300", "csrc"), str(src), "-o",
                    str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
