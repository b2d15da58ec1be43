"""The integer-pipe FP64 functions (csrc/xc_fp64.cuh), compiled for the host.

The quotient, the square root, the scalings and the comparisons against the
processor's own: the same bits for every operand, with the seeds moved by the
error the device's approximations may have (and the wider one of their
emulation here).  The exponential and the logarithm against long double."""
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
  auto same = [&](double a, double b) { if (xc_bits(a) != xc_bits(b) && !(a != a && b != b)) ++bad; };
  for (long i = 0; i < 1000000; ++i) {
    double x = xc_from_bits(g());
    if (i % 2) x = xc_from_bits((g() % (6ull << 52)) | (g() & (1ull << 63)));      // subnormals and their neighbours
    if (i < 13) x = special[i];
    same(xc_half(x), x * 0.5); same(xc_scale2<-2>(x), x * 0.25); same(xc_scale2<1>(x), x * 2.0);
    const double lo = 1e-16, hi = 1.0 - 1e-16;
    same(xc_clamp_pos(x, lo, hi), x > hi ? hi : (x < lo ? lo : x));
    same(xc_max_pos(x, lo), x != x ? x : (x > lo ? x : lo));
    same(xc_max0(x), x != x ? x : (x > 0 ? x : 0.0));
    if (xc_ge_pos(x, 1e-8) != (x >= 1e-8) || xc_isnan(x) != (x != x)) ++bad;
  }
  // exp: half an ulp plus the fixed point's error, which grows with |x| as the
  // 64-bit log2(e) does (2^-64 of x log2(e), 2^-53 being half an ulp at worst)
  std::uniform_real_distribution<double> U(-1.0, 1.0);
  const double scale[] = {1e-9, 5e-5, 7e-5, 0.02, 1.0, 64.0, 707.0};
  for (long i = 0; i < 3000000; ++i) {
    const double sc = scale[i % 7], x = U(g) * sc, e = xc_exp(x);
    const long double t = expl((long double)x);
    int k;
    std::frexp((double)t, &k);
    const double err = (double)(fabsl((long double)e - t) / ldexpl(1.0L, k - 53));
    if (!(err <= 0.504 + std::fabs(x) * 1.45 * 0.0005)) { if (bad++ < 9) std::printf("exp %a: %g ulp\n", x, err); }
  }
  for (double x : {0.0, -0.0, 5e-324, -1e-300, 1e-17, -5e-17, 709.0, 710.0, -746.0, 1.0 / 0.0, -1.0 / 0.0, 0.0 / 0.0})
    same(xc_exp(x), std::exp(x));
  // log2 to 2^-54 of one, the powers built on it to 2e-15 (c times twice that, half an ulp)
  for (long i = 0; i < 3000000; ++i) {
    double x = std::exp(U(g) * 36.5);
    if (i & 1) x = 1.0 - std::fabs(U(g)) * 1e-9;
    if (!xc_log2_ok(x) || fabsl((long double)xc_log2_fixed(x) - log2l((long double)x) * 0x1p57L) > 8) ++bad;
    const double c = i % 3 ? 1 / 2.09 : 1 / 0.37, B = 0.63;
    const long double t = powl((long double)x / B, (long double)c);
    const double r = xc_exp2_product((uint64_t)(c * 0x1p58), xc_log2_fixed(x) - xc_log2_fixed(B));
    if (!(fabsl(r - t) <= 2e-15L * t)) ++bad;
  }
  std::printf("bad %ld\n", bad);
  return bad != 0;
}
"""


def test_integer_functions_against_the_processor(tmp_path):
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


SQUARES = PROBE[:PROBE.index("int main() {")] + r"""
int main() {
  std::mt19937_64 g(22);
  long bad = 0;
  const double edge[] = {0.0, -0.0, 1.0, -1.5, 5e-324, 0x1p-1022, 0x1.fffffffffffffp1023, INFINITY, -INFINITY, NAN,
                         0x1p-511, 0x1p-507, 0x1.fffffffffffffp-508, 0x1p515, 0x1.fffffffffffffp515, 0x1p516};
  auto check = [&](double a) {
    const double q = xc_sqr<8>(a), r = (a * 0.0625) * (a * 0.0625);
    if (xc_bits(q) != xc_bits(r) && !(q != q && r != r)) { if (bad++ < 5) std::printf("%a: %a not %a\n", a, q, r); }
  };
  for (double a : edge) check(a);
  for (long i = 0; i < 4000000; ++i) {       // all exponents whose quotient by 16 is normal
    const uint64_t e = i % 2 ? 983 + g() % 80 : 5 + g() % 2042;
    check(xc_from_bits((g() & (1ull << 63)) | (e << 52) | significand(g(), g() % 5)));
  }
  std::printf("bad %ld\n", bad);
  return bad != 0;
}
"""


def test_scaled_squares_against_the_processor(tmp_path):
    """xc_sqr<K>: the bits of the square of a 2^(-K/2), through both ends of the range, zeros, infinities and NaN."""
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    src = tmp_path / "squares.cpp"
    src.write_text(SQUARES)
    exe = tmp_path / "squares"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "xcore.jl_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


PRODUCTS = PROBE[:PROBE.index("int main() {")] + r"""
static bool same(double a, double b) { return xc_bits(a) == xc_bits(b) || (a != a && b != b); }
static long check(double a, double b) {
  long bad = !same(xc_mul(a, b), a * b) + !same(xc_sqr(a), a * a);
  const float f = (float)a, r = xc_to_float(a);
  bad += std::memcmp(&f, &r, 4) != 0 && f == f;
  return bad + !same(xc_mul_small<3>(a), 3 * a) + !same(xc_mul_small<5>(a), 5 * a) + !same(xc_mul_small<6>(a), 6 * a) +
         !same(xc_mul_small<7>(a), 7 * a) + !same(xc_mul_small<11>(a), 11 * a);
}
int main() {
  std::mt19937_64 g(21);
  long bad = 0;
  const double edge[] = {0.0, -0.0, 1.0, -1.5, 5e-324, 0x1p-1022, 0x1.fffffffffffffp-1023, 0x1.fffffffffffffp1023, INFINITY,
                         -INFINITY, NAN, 0x1p-511, 0x1.fffffffffffffp-512, 0x1p512, 0x1.fffffffffffffp511};
  for (double a : edge)
    for (double b : edge) bad += check(a, b);
  for (long i = 0; i < 8000000; ++i) {
    const int wide = i % 4 == 0 ? 2048 : (i % 4 == 1 ? 80 : 1100), low = i % 4 == 3 ? 948 : (i % 4 == 1 ? 983 : 0);
    auto draw = [&] {
      return xc_from_bits((g() & (1ull << 63)) | ((uint64_t)(low + g() % wide) << 52) | significand(g(), g() % 5));
    };
    const double a = draw(), b = draw();
    bad += check(a, b);
  }
  std::printf("bad %ld\n", bad);
  return bad != 0;
}
"""


def test_integer_products_against_the_processor(tmp_path):
    """xc_mul, xc_sqr, xc_mul_small and the conversion to float: the processor's bits for all kinds of significands and all exponents, through
    both ends of the range, and for zeros, infinities and NaN."""
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    src = tmp_path / "products.cpp"
    src.write_text(PRODUCTS)
    exe = tmp_path / "products"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "xcore.jl_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("call", ["xc_exp(0.5)", "(double)xc_log2_fixed(0.5)", "xc_exp2_product(1ull << 58, 5)"])
def test_table_functions_do_not_compile_for_the_host_under_nvcc(tmp_path, call):
    """Their tables are in device memory: a host call in a .cu file is an error, not a wrong number."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    for body, ok in ((f"__global__ void k(double* y) {{ *y = {call}; }}", True), (f"double h() {{ return {call}; }}", False)):
        src = tmp_path / "call.cu"
        src.write_text('#include "xc_fp64.cuh"\n' + body + "\n")
        r = subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_103a,code=sm_103a",
                            "-I", os.path.join(ROOT, "xcore.jl_gb300", "csrc"), "-c", str(src), "-o",
                            str(tmp_path / "call.o")], capture_output=True, text=True)
        assert (r.returncode == 0) == ok, r.stderr
